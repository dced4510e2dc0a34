// gg_surrogate.cu -- the surrogate ΔASPL ranker (gg_surrogate_* in gg.h).
//
// Every product rounds its operands to bf16 (round to nearest even) in shared memory and
// multiplies with mma.sync m16n8k16 (bf16 in, fp32 accumulate).  The forward pass (graph
// embedding and swap readout) is one cooperative launch with a bounded grid barrier per
// message-passing layer; a training step (readout of its swaps, backward pass, Adam) is
// another.  A block of eight warps owns 32-row tiles: at n = 4096 that is 128 blocks, and
// what bounds every step is the latency of its gathers (nothing here is large enough to
// fill the chip), so a thread's loads are 16 bytes wide and all in flight together, the
// weights of a step are staged before the barrier it waits at, and steps that need no
// barrier between them run as one.  n = 4096, d = 8: 4096 predictions 142 -> 36 us, a
// training step on 64 swaps 44 + 246 -> 57 us (tiles of 64 rows, four warps, 4-byte
// loads, a separate readout launch and a pass of its own for each neighbour mean).
#include "gg.h"
#include "gg_kernels.cuh"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <string>
#include <vector>

namespace gg {
void set_last_error(const char *msg);  // gg_engine.cu
}

namespace {

constexpr int kH = 64;           // hidden width
constexpr int kZ = 3 * kH;       // swap readout width
constexpr int kLayers = 3;       // message-passing layers
__host__ __device__ constexpr int cmax3(int a, int b, int c) { return a > b ? (a > c ? a : c) : (b > c ? b : c); }

__device__ __forceinline__ uint16_t bf16_bits(float x) {
    __nv_bfloat16 h = __float2bfloat16_rn(x);
    return *reinterpret_cast<uint16_t *>(&h);
}

__device__ __forceinline__ void mma_bf16(float c[4], const uint32_t a[4], const uint32_t b[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// ---------------------------------------------------------------------------
// swap readout helpers
// ---------------------------------------------------------------------------

__device__ __forceinline__ void partners(const gg_swap &s, int &p, int &q) {
    p = s.mode ? s.d : s.c;  // new edges (a,p), (b,q)
    q = s.mode ? s.c : s.d;
}

// Per-call scalars, written by the host before each replay: [0] 1/count of
// unmasked swaps, [1] learning rate, [2] 1 - beta1^t, [3] 1 - beta2^t.
enum { kHypInvCnt = 0, kHypLr = 1, kHypC1 = 2, kHypC2 = 3, kHypN = 4 };

// ---------------------------------------------------------------------------
// Tiles: 32 rows, eight warps.  Shared-memory operands are bf16, row-major with a stride
// of 8 elements more than a multiple of 16 (fragment loads spread over the banks).
// ---------------------------------------------------------------------------
constexpr int kTile = 32;                  // rows (vertices or swaps) of a tile
constexpr int kBlock = 256;
constexpr int kFmax = 256;                 // in_features
constexpr int kLdH = kH + 8;               // K = 64 operands
constexpr int kLd2H = 2 * kH + 8;          // K = 128
constexpr int kLdZ = kZ + 8;               // K = 192
constexpr int kLdT = kTile + 8;            // K = 32 (the weight gradients)
constexpr int kLdO = kH + 1;               // fp32 rows of the readout's hidden layer

__device__ __forceinline__ uint32_t bf16_pair(const float lo, const float hi) {
    return (uint32_t)bf16_bits(lo) | ((uint32_t)bf16_bits(hi) << 16);
}

// acc[2][4]: the warp's 16 rows (from row0) x 16 columns (from col0) of A (rows x K,
// stride lda) times B^T (columns x K, stride ldb), K % 16 == 0.
__device__ __forceinline__ void tile_mma(const uint16_t *A, const int lda, const uint16_t *B, const int ldb, const int K,
                                         const int row0, const int col0, float (&acc)[2][4]) {
    const int lane = threadIdx.x & 31, gid = lane >> 2, tg = lane & 3;
#pragma unroll
    for (int j = 0; j < 2; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    const uint16_t *a0 = A + (row0 + gid) * lda + 2 * tg, *a1 = a0 + 8 * lda;
    const uint16_t *b0 = B + (col0 + gid) * ldb + 2 * tg, *b1 = b0 + 8 * ldb;
#pragma unroll 4
    for (int k0 = 0; k0 < K; k0 += 16) {
        uint32_t a[4], b[2];
        a[0] = *reinterpret_cast<const uint32_t *>(a0 + k0);
        a[1] = *reinterpret_cast<const uint32_t *>(a1 + k0);
        a[2] = *reinterpret_cast<const uint32_t *>(a0 + k0 + 8);
        a[3] = *reinterpret_cast<const uint32_t *>(a1 + k0 + 8);
        b[0] = *reinterpret_cast<const uint32_t *>(b0 + k0);
        b[1] = *reinterpret_cast<const uint32_t *>(b0 + k0 + 8);
        mma_bf16(acc[0], a, b);
        b[0] = *reinterpret_cast<const uint32_t *>(b1 + k0);
        b[1] = *reinterpret_cast<const uint32_t *>(b1 + k0 + 8);
        mma_bf16(acc[1], a, b);
    }
}

// f(row, column, x, y) for the lane's pairs of neighbouring columns of acc.
template <class F>
__device__ __forceinline__ void tile_pairs(const float (&acc)[2][4], const int row0, const int col0, F f) {
    const int lane = threadIdx.x & 31, gid = lane >> 2, tg = lane & 3;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int c = col0 + 8 * j + 2 * tg;
        f(row0 + gid, c, acc[j][0], acc[j][1]);
        f(row0 + gid + 8, c, acc[j][2], acc[j][3]);
    }
}

// B[c][k0 + k] = bf16(W[k][c]), k < K (even), c < 64: a weight block, transposed.  Rows
// k >= rows are 0.
__device__ __forceinline__ void stage_t(uint16_t *B, const int ldb, const int k0, const float *W, const int K,
                                        const int rows) {
#pragma unroll 8
    for (int e = threadIdx.x; e < K / 2 * kH; e += kBlock) {
        const int k = e / kH * 2, c = e % kH;
        const float lo = k < rows ? __ldcg(W + k * kH + c) : 0.f, hi = k + 1 < rows ? __ldcg(W + (k + 1) * kH + c) : 0.f;
        *reinterpret_cast<uint32_t *>(B + c * ldb + k0 + k) = bf16_pair(lo, hi);
    }
}

// B[k][c] = bf16(W[k][c]), k < K, c < 64: a weight block as it lies (4-byte loads: the
// parameter blocks start at odd multiples of 4 bytes).
__device__ __forceinline__ void stage_n(uint16_t *B, const int ldb, const float *W, const int K) {
#pragma unroll 8
    for (int e = threadIdx.x; e < K * kH / 2; e += kBlock) {
        const int k = e / (kH / 2), c = e % (kH / 2) * 2;
        *reinterpret_cast<uint32_t *>(B + k * ldb + c) = bf16_pair(__ldcg(W + k * kH + c), __ldcg(W + k * kH + c + 1));
    }
}

// B[c][r] = bf16(S[(v0 + r) * ld + c]), r < 32 (0 past `rows`), c < cols (0 up to cpad): the
// transposed tile of a matrix of row stride ld.
__device__ __forceinline__ void stage_rows_t(uint16_t *B, const float *S, const int ld, const int v0, const int rows,
                                             const int cols, const int cpad) {
#pragma unroll 4
    for (int e = threadIdx.x; e < kTile / 2 * cpad; e += kBlock) {
        const int r = e / cpad * 2, c = e % cpad, v = v0 + r;
        const float lo = v < rows && c < cols ? __ldcg(S + (size_t)v * ld + c) : 0.f;
        const float hi = v + 1 < rows && c < cols ? __ldcg(S + (size_t)(v + 1) * ld + c) : 0.f;
        *reinterpret_cast<uint32_t *>(B + c * kLdT + r) = bf16_pair(lo, hi);
    }
}

__device__ __forceinline__ float4 ldcg4(const float *p) { return __ldcg(reinterpret_cast<const float4 *>(p)); }

// Mean of the neighbours' rows of S at columns [c, c + 4): added in slot order, the loads
// of eight neighbours in flight together.
__device__ __forceinline__ float4 neighbour_sum(const float *S, const int32_t *adj, const int d, const int v, const int c) {
    float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
    const int32_t *row = adj + (size_t)v * d;
    for (int i0 = 0; i0 < d; i0 += 8) {
        float4 x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i0 + i < d) x[i] = ldcg4(S + (size_t)__ldg(row + i0 + i) * kH + c);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i0 + i < d) { m.x += x[i].x; m.y += x[i].y; m.z += x[i].z; m.w += x[i].w; }
    }
    return m;
}

// Layout of the parameters (floats from the start of the vector).
struct ParamAt {
    int win, bin, ws[kLayers], wn[kLayers], b[kLayers], wr1, br1, wr2, br2;
};

// The rows of a swap: its ends and the new partners of a and b.
struct SwapIds {
    int a, b, c, d, p, q;
    __device__ __forceinline__ explicit SwapIds(const gg_swap &s) : a(s.a), b(s.b), c(s.c), d(s.d) { partners(s, p, q); }
};

// The swaps of a tile into shared memory (a block's first tile while it waits for the layers).
__device__ __forceinline__ void load_swaps(gg_swap *s_sw, const gg_swap *sw, const int p0, const int n_sw) {
    constexpr int kWords = (int)(sizeof(gg_swap) / 4);
    for (int e = threadIdx.x; e < kTile * kWords; e += kBlock)
        if (p0 + e / kWords < n_sw)
            reinterpret_cast<int *>(s_sw)[e] = __ldg(reinterpret_cast<const int *>(sw + p0) + e);
}

// Z of a tile of swaps into As (bf16 rows of 192) and, with ZT, also transposed:
// z = [Ha + Hb + Hc + Hd, Ha Hb + Hc Hd, Ha Hp + Hb Hq]; rows past n_sw are 0.
__device__ __forceinline__ void stage_z(uint16_t *As, uint16_t *ZT, const float *H3, const gg_swap *s_sw, const int p0,
                                        const int n_sw) {
    for (int e = threadIdx.x; e < kTile * (kH / 4); e += kBlock) {
        const int r = e / (kH / 4), c = e % (kH / 4) * 4, p = p0 + r;
        float z[3][4] = {};
        if (p < n_sw) {
            const SwapIds s(s_sw[r]);
            const float4 a = ldcg4(H3 + (size_t)s.a * kH + c), b = ldcg4(H3 + (size_t)s.b * kH + c);
            const float4 cc = ldcg4(H3 + (size_t)s.c * kH + c), d = ldcg4(H3 + (size_t)s.d * kH + c);
            const float4 pp = ldcg4(H3 + (size_t)s.p * kH + c), q = ldcg4(H3 + (size_t)s.q * kH + c);
            const float ha[4] = {a.x, a.y, a.z, a.w}, hb[4] = {b.x, b.y, b.z, b.w}, hc[4] = {cc.x, cc.y, cc.z, cc.w};
            const float hd[4] = {d.x, d.y, d.z, d.w}, hp[4] = {pp.x, pp.y, pp.z, pp.w}, hq[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                z[0][k] = ha[k] + hb[k] + hc[k] + hd[k];
                z[1][k] = ha[k] * hb[k] + hc[k] * hd[k];
                z[2][k] = ha[k] * hp[k] + hb[k] * hq[k];
            }
        }
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            *reinterpret_cast<uint2 *>(As + r * kLdZ + t * kH + c) = make_uint2(bf16_pair(z[t][0], z[t][1]), bf16_pair(z[t][2], z[t][3]));
            if (ZT)
#pragma unroll
                for (int k = 0; k < 4; ++k) ZT[(t * kH + c + k) * kLdT + r] = bf16_bits(z[t][k]);
        }
    }
}

// s_o = relu(Z Wr1 + br1) of the tile (fp32), and y = s_o . wr2 + br2 (one thread a row)
// through f(row, y).
template <class F>
__device__ __forceinline__ void readout(const uint16_t *As, const uint16_t *BR, float *s_o, const float *P, const ParamAt &at,
                                        F f) {
    const int warp = threadIdx.x >> 5, row0 = (warp & 1) * 16, col0 = (warp >> 1) * 16;
    float acc[2][4];
    tile_mma(As, kLdZ, BR, kLdZ, kZ, row0, col0, acc);
    tile_pairs(acc, row0, col0, [&](const int r, const int c, const float x, const float y) {
        const float u = x + P[at.br1 + c], w = y + P[at.br1 + c + 1];
        s_o[r * kLdO + c] = u > 0.f ? u : 0.f;
        s_o[r * kLdO + c + 1] = w > 0.f ? w : 0.f;
    });
    __syncthreads();
    if (threadIdx.x < kTile) {
        float sum = 0.f;
#pragma unroll 16
        for (int j = 0; j < kH; ++j) sum += s_o[threadIdx.x * kLdO + j] * P[at.wr2 + j];
        f((int)threadIdx.x, sum + P[at.br2]);
    }
}

// ---------------------------------------------------------------------------
// Forward: the graph embedding (H0 .. H3, with the neighbour means M0 .. M2 kept for the
// backward pass) when n > 0, then the readout of n_sw swaps (y), with a bounded grid
// barrier after each layer (every block needs the whole previous layer for its neighbour
// means).  A layer's two products H Ws + M Wn run as one K = 128 product over [H | M] and
// [Ws ; Wn].
// ---------------------------------------------------------------------------
struct FwdArgs {
    const float *X;
    int F;
    const int32_t *adj;
    int n, d;
    const float *P;
    ParamAt at;
    float *H[kLayers + 1];
    float *M[kLayers];
    const gg_swap *sw;
    int n_sw;
    float *y;
    gg::Ctl *ctl;
    unsigned expected;
    long long wait_ns;
};

__host__ __device__ constexpr int pad16(int x) { return (x + 15) / 16 * 16; }
// bf16 elements of the forward's shared operands: the tile, and every step's weights
__host__ __device__ constexpr int fwd_tile_elems(int F) { return kTile * (cmax3(pad16(F), 2 * kH, kZ) + 8); }
__host__ __device__ constexpr size_t fwd_smem(int F) {
    return sizeof(uint16_t) * (size_t)(fwd_tile_elems(F) + kH * (pad16(F) + 8) + kLayers * kH * kLd2H + kH * kLdZ) +
           sizeof(float) * kTile * kLdO;
}

__global__ void __launch_bounds__(kBlock) surrogate_forward_kernel(const FwdArgs a) {
    extern __shared__ __align__(16) uint16_t fsm[];
    const int K0 = pad16(a.F), ld0 = K0 + 8;
    uint16_t *As = fsm;
    uint16_t *B0 = As + fwd_tile_elems(a.F), *BL = B0 + kH * ld0, *BR = BL + kLayers * kH * kLd2H;
    float *s_o = reinterpret_cast<float *>(BR + kH * kLdZ);
    __shared__ gg_swap s_sw[kTile];
    load_swaps(s_sw, a.sw, (int)blockIdx.x * kTile, a.n_sw);
    const int tid = threadIdx.x, warp = tid >> 5, row0 = (warp & 1) * 16, col0 = (warp >> 1) * 16;
    unsigned epoch = 0;
    float acc[2][4];
    auto store_relu = [&](const float *bias, float *out, const int v0) {
        tile_pairs(acc, row0, col0, [&](const int r, const int c, const float x, const float y) {
            const float u = x + bias[c], w = y + bias[c + 1];
            if (v0 + r < a.n)
                *reinterpret_cast<float2 *>(out + (size_t)(v0 + r) * kH + c) = make_float2(u > 0.f ? u : 0.f, w > 0.f ? w : 0.f);
        });
    };
    if (a.n > 0) {
        const int ntile = (a.n + kTile - 1) / kTile;
        // every layer's weights, once
        stage_t(B0, ld0, 0, a.P + a.at.win, K0, a.F);
        for (int l = 0; l < kLayers; ++l) {
            stage_t(BL + l * kH * kLd2H, kLd2H, 0, a.P + a.at.ws[l], kH, kH);
            stage_t(BL + l * kH * kLd2H, kLd2H, kH, a.P + a.at.wn[l], kH, kH);
        }
        if (a.n_sw > 0) stage_t(BR, kLdZ, 0, a.P + a.at.wr1, kZ, kZ);
        // H0 = relu(X W_in + b_in); K = in_features padded to 16
        for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
            for (int e = tid; e < kTile * K0 / 2; e += kBlock) {
                const int r = e / (K0 / 2), k = e % (K0 / 2) * 2, v = t * kTile + r;
                const float lo = v < a.n && k < a.F ? a.X[(size_t)v * a.F + k] : 0.f;
                const float hi = v < a.n && k + 1 < a.F ? a.X[(size_t)v * a.F + k + 1] : 0.f;
                *reinterpret_cast<uint32_t *>(As + r * ld0 + k) = bf16_pair(lo, hi);
            }
            __syncthreads();
            tile_mma(As, ld0, B0, ld0, K0, row0, col0, acc);
            store_relu(a.P + a.at.bin, a.H[0], t * kTile);
            __syncthreads();
        }
        const float inv = 1.f / (float)a.d;
        for (int l = 0; l < kLayers; ++l) {
            if (!gg::grid_sync(a.ctl, a.expected, a.wait_ns, l, epoch)) return;
            for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
                // A = [H_l | mean of the neighbours' H_l rows]; the means are kept in M_l
#pragma unroll
                for (int e = tid; e < kTile * (kH / 4); e += kBlock) {
                    const int r = e / (kH / 4), c = e % (kH / 4) * 4, v = t * kTile + r;
                    float4 h = make_float4(0.f, 0.f, 0.f, 0.f), m = h;
                    if (v < a.n) {
                        h = ldcg4(a.H[l] + (size_t)v * kH + c);
                        m = neighbour_sum(a.H[l], a.adj, a.d, v, c);
                        m.x *= inv; m.y *= inv; m.z *= inv; m.w *= inv;
                        *reinterpret_cast<float4 *>(a.M[l] + (size_t)v * kH + c) = m;
                    }
                    *reinterpret_cast<uint2 *>(As + r * kLd2H + c) = make_uint2(bf16_pair(h.x, h.y), bf16_pair(h.z, h.w));
                    *reinterpret_cast<uint2 *>(As + r * kLd2H + kH + c) = make_uint2(bf16_pair(m.x, m.y), bf16_pair(m.z, m.w));
                }
                __syncthreads();
                tile_mma(As, kLd2H, BL + l * kH * kLd2H, kLd2H, 2 * kH, row0, col0, acc);
                store_relu(a.P + a.at.b[l], a.H[l + 1], t * kTile);
                __syncthreads();
            }
        }
        if (!gg::grid_sync(a.ctl, a.expected, a.wait_ns, kLayers, epoch)) return;
    } else if (a.n_sw > 0) {
        stage_t(BR, kLdZ, 0, a.P + a.at.wr1, kZ, kZ);
    }
    for (int t = blockIdx.x; t * kTile < a.n_sw; t += gridDim.x) {
        if (t != (int)blockIdx.x) load_swaps(s_sw, a.sw, t * kTile, a.n_sw);
        __syncthreads();
        stage_z(As, nullptr, a.H[kLayers], s_sw, t * kTile, a.n_sw);
        __syncthreads();
        readout(As, BR, s_o, a.P, a.at, [&](const int r, const float y) {
            if (t * kTile + r < a.n_sw) a.y[t * kTile + r] = y;
        });
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Training step: the readout of n_sw swaps, the gradient of their masked mean squared
// error with respect to every parameter and, with `train`, the Adam step, in one
// cooperative launch with a bounded grid barrier between dependent stages:
//   1. swap tiles: Z, O, y as in the forward; dy, dO = dy w_r2 (O > 0), dZ = dO Wr1^T,
//      dWr1 += Z^T dO, the output biases and weights, and dZ scattered into dH3 (fp32
//      atomics);
//   2. per layer l = 2, 1, 0, vertex tiles: dPre = dH (H_{l+1} > 0), with dH the upstream
//      rows plus the neighbour mean of the layer above's G (symmetric adjacency); db_l,
//      dWs_l += H_l^T dPre, dWn_l += M_l^T dPre; the rows dPre Ws_l^T and G = dPre Wn_l^T;
//   3. the input layer: dPre0 the same way, db_in, dWin += X^T dPre0;
//   4. Adam on every parameter.
// Weight gradients add each tile's partial product with fp32 atomics; elementwise steps
// stay in fp32.  Data other blocks wrote earlier in the launch is read through the L2.
// ---------------------------------------------------------------------------
struct BwdArgs {
    const float *X;
    int F;
    const int32_t *adj;
    int n, d;
    const float *P;
    float *Gd;
    ParamAt at;
    const float *H[kLayers + 1];
    const float *M[kLayers];
    const gg_swap *sw;
    int n_sw;
    const float *t;
    const int32_t *mask;
    const float *hyper;
    float *dH[2], *G[2];          // dH[0] zero before; layers alternate
    float *loss;
    float *adam_m, *adam_v;
    float *params;
    int n_params, train;
    gg::Ctl *ctl;
    unsigned expected;
    long long wait_ns;
};

// p[0], p[1] += x, y (8-byte aligned when `wide`)
__device__ __forceinline__ void red2(float *p, const float x, const float y, const bool wide) {
    if (wide) {
        asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(x), "f"(y) : "memory");
    } else {
        atomicAdd(p, x);
        atomicAdd(p + 1, y);
    }
}
__device__ __forceinline__ void red4(float *p, const float x, const float y, const float z, const float w) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

// bf16 elements of the training step's shared operands (stage 1; the later stages use less,
// but for many input features)
__host__ __device__ constexpr int bwd_swap_elems() {
    return kTile * kLdZ + kH * kLdZ + kZ * kLdH + kZ * kLdT + kTile * kLdH + kH * kLdT;
}
__host__ __device__ constexpr int bwd_layer_elems(int F) {
    return 2 * kH * kLdH + kTile * kLdH + kH * kLdT + cmax3(2 * kH, pad16(F), 0) * kLdT;
}
__host__ __device__ constexpr size_t bwd_smem(int F) {
    return sizeof(float) * kTile * (kLdO + kZ + 4) + sizeof(uint16_t) * (size_t)cmax3(bwd_swap_elems(), bwd_layer_elems(F), 0);
}

__global__ void __launch_bounds__(kBlock) surrogate_backward_kernel(const BwdArgs a) {
    extern __shared__ __align__(16) float bsmf[];
    float *s_o = bsmf, *s_dz = s_o + kTile * kLdO;     // fp32: O, dZ (rows of kZ + 4)
    uint16_t *sm = reinterpret_cast<uint16_t *>(s_dz + kTile * (kZ + 4));
    __shared__ float s_dy[kTile], s_hyper[kHypN];
    __shared__ gg_swap s_sw[kTile];
    load_swaps(s_sw, a.sw, (int)blockIdx.x * kTile, a.n_sw);
    if (threadIdx.x < kHypN) s_hyper[threadIdx.x] = __ldg(a.hyper + threadIdx.x);
    const int tid = threadIdx.x, warp = tid >> 5;
    unsigned epoch = 0;
    float acc[2][4];
    const float *Pm = a.P;
    float *Gd = a.Gd;
    // a weight gradient's rows start at parameter `o`
    auto add_grad = [&](const int o, const int row0, const int col0, const int rows) {
        tile_pairs(acc, row0, col0, [&](const int r, const int c, const float x, const float y) {
            if (r < rows) red2(Gd + o + r * kH + c, x, y, (o & 1) == 0);
        });
    };
    // 1. swap tiles
    if ((int)blockIdx.x * kTile < a.n_sw) {
        uint16_t *As = sm, *BR = As + kTile * kLdZ, *BZ = BR + kH * kLdZ, *ZT = BZ + kZ * kLdH, *Do = ZT + kZ * kLdT,
                 *DoT = Do + kTile * kLdH;
        stage_t(BR, kLdZ, 0, Pm + a.at.wr1, kZ, kZ);
        stage_n(BZ, kLdH, Pm + a.at.wr1, kZ);
        __syncthreads();
        const float inv_cnt = s_hyper[kHypInvCnt];
        const float *H3 = a.H[kLayers];
        for (int t = blockIdx.x; t * kTile < a.n_sw; t += gridDim.x) {
            const int p0 = t * kTile;
            if (t != (int)blockIdx.x) {
                load_swaps(s_sw, a.sw, p0, a.n_sw);
                __syncthreads();
            }
            stage_z(As, ZT, H3, s_sw, p0, a.n_sw);
            __syncthreads();
            readout(As, BR, s_o, Pm, a.at, [&](const int r, const float y) {
                float dy = 0.f;
                if (p0 + r < a.n_sw) {
                    const float m = a.mask[p0 + r] ? 1.f : 0.f;
                    const float err = (y - a.t[p0 + r]) * m;
                    dy = 2.f * err * inv_cnt;
                    atomicAdd(a.loss, err * err * inv_cnt);
                }
                s_dy[r] = dy;
            });
            __syncthreads();
            // dO = dy w_r2 where O > 0, both ways round
            for (int e = tid; e < kTile / 2 * kH; e += kBlock) {
                const int r = e / kH * 2, j = e % kH;
                const float w = Pm[a.at.wr2 + j];
                const float u = s_o[r * kLdO + j] > 0.f ? s_dy[r] * w : 0.f, v = s_o[(r + 1) * kLdO + j] > 0.f ? s_dy[r + 1] * w : 0.f;
                Do[r * kLdH + j] = bf16_bits(u);
                Do[(r + 1) * kLdH + j] = bf16_bits(v);
                *reinterpret_cast<uint32_t *>(DoT + j * kLdT + r) = bf16_pair(u, v);
            }
            if (tid < kH) {
                float g_wr2 = 0.f, g_br1 = 0.f, g_br2 = 0.f;
                const float w = Pm[a.at.wr2 + tid];
                for (int r = 0; r < kTile; ++r) {
                    const float o = s_o[r * kLdO + tid], dy = s_dy[r];
                    g_wr2 += dy * o;
                    g_br1 += o > 0.f ? dy * w : 0.f;
                    g_br2 += dy;
                }
                atomicAdd(Gd + a.at.wr2 + tid, g_wr2);
                atomicAdd(Gd + a.at.br1 + tid, g_br1);
                if (tid == 0) atomicAdd(Gd + a.at.br2, g_br2);
            }
            __syncthreads();
            // dZ = dO Wr1^T (32 x 192), dWr1 += Z^T dO (192 x 64)
            for (int q = warp; q < 2 * (kZ / 16); q += kBlock / 32) {
                const int row0 = (q & 1) * 16, col0 = (q >> 1) * 16;
                tile_mma(Do, kLdH, BZ, kLdH, kH, row0, col0, acc);
                tile_pairs(acc, row0, col0, [&](const int r, const int c, const float x, const float y) {
                    s_dz[r * (kZ + 4) + c] = x;
                    s_dz[r * (kZ + 4) + c + 1] = y;
                });
            }
            for (int q = warp; q < (kZ / 16) * (kH / 16); q += kBlock / 32) {
                tile_mma(ZT, kLdT, DoT, kLdT, kTile, q / (kH / 16) * 16, q % (kH / 16) * 16, acc);
                add_grad(a.at.wr1, q / (kH / 16) * 16, q % (kH / 16) * 16, kZ);
            }
            __syncthreads();
            // dZ of the tile's swaps into dH3
            for (int e = tid; e < kTile * (kH / 4); e += kBlock) {
                const int r = e / (kH / 4), c = e % (kH / 4) * 4;
                if (p0 + r >= a.n_sw) continue;
                const SwapIds w(s_sw[r]);
                const float *z = s_dz + r * (kZ + 4) + c;
                const float4 g0 = *reinterpret_cast<const float4 *>(z), g1 = *reinterpret_cast<const float4 *>(z + kH),
                             g2 = *reinterpret_cast<const float4 *>(z + 2 * kH);
                const float4 ha = ldcg4(H3 + (size_t)w.a * kH + c), hb = ldcg4(H3 + (size_t)w.b * kH + c);
                const float4 hc = ldcg4(H3 + (size_t)w.c * kH + c), hd = ldcg4(H3 + (size_t)w.d * kH + c);
                const float4 hp = ldcg4(H3 + (size_t)w.p * kH + c), hq = ldcg4(H3 + (size_t)w.q * kH + c);
                float *D = a.dH[0] + c;
                red4(D + (size_t)w.a * kH, g0.x + g1.x * hb.x + g2.x * hp.x, g0.y + g1.y * hb.y + g2.y * hp.y,
                     g0.z + g1.z * hb.z + g2.z * hp.z, g0.w + g1.w * hb.w + g2.w * hp.w);
                red4(D + (size_t)w.b * kH, g0.x + g1.x * ha.x + g2.x * hq.x, g0.y + g1.y * ha.y + g2.y * hq.y,
                     g0.z + g1.z * ha.z + g2.z * hq.z, g0.w + g1.w * ha.w + g2.w * hq.w);
                red4(D + (size_t)w.c * kH, g0.x + g1.x * hd.x, g0.y + g1.y * hd.y, g0.z + g1.z * hd.z, g0.w + g1.w * hd.w);
                red4(D + (size_t)w.d * kH, g0.x + g1.x * hc.x, g0.y + g1.y * hc.y, g0.z + g1.z * hc.z, g0.w + g1.w * hc.w);
                red4(D + (size_t)w.p * kH, g2.x * ha.x, g2.y * ha.y, g2.z * ha.z, g2.w * ha.w);
                red4(D + (size_t)w.q * kH, g2.x * hb.x, g2.y * hb.y, g2.z * hb.z, g2.w * hb.w);
            }
            __syncthreads();
        }
    }
    // 2. layers 2, 1, 0, then 3. the input layer (l = -1)
    uint16_t *BW = sm, *Dp = BW + 2 * kH * kLdH, *DpT = Dp + kTile * kLdH, *TT = DpT + kH * kLdT;
    const int ntile = (a.n + kTile - 1) / kTile;
    const float inv = 1.f / (float)a.d;
    for (int l = kLayers - 1; l >= -1; --l) {
        if (l >= 0) {   // (the weights do not wait for the other blocks)
            __syncthreads();
            stage_n(BW, kLdH, Pm + a.at.ws[l], kH);
            stage_n(BW + kH * kLdH, kLdH, Pm + a.at.wn[l], kH);
        }
        if (!gg::grid_sync(a.ctl, a.expected, a.wait_ns, kLayers - l, epoch)) return;
        const int from = (kLayers - 1 - l) & 1;
        const float *up = a.dH[from], *Gup = l == kLayers - 1 ? nullptr : a.G[from];
        float *dn = a.dH[from ^ 1], *Gn = a.G[from ^ 1];
        for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
            const int v0 = t * kTile;
            // dPre = (upstream + neighbour mean of G) where H_{l+1} > 0, both ways round
            float *q32 = s_dz;   // fp32 rows of the tile (stride kH + 4)
            for (int e = tid; e < kTile * (kH / 4); e += kBlock) {
                const int r = e / (kH / 4), c = e % (kH / 4) * 4, v = v0 + r;
                float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                if (v < a.n) {
                    const float4 h = ldcg4(a.H[l + 1] + (size_t)v * kH + c);
                    q = ldcg4(up + (size_t)v * kH + c);
                    if (Gup) {
                        const float4 m = neighbour_sum(Gup, a.adj, a.d, v, c);
                        q.x += m.x * inv; q.y += m.y * inv; q.z += m.z * inv; q.w += m.w * inv;
                    }
                    q.x = h.x > 0.f ? q.x : 0.f; q.y = h.y > 0.f ? q.y : 0.f;
                    q.z = h.z > 0.f ? q.z : 0.f; q.w = h.w > 0.f ? q.w : 0.f;
                }
                *reinterpret_cast<float4 *>(q32 + r * (kH + 4) + c) = q;
                *reinterpret_cast<uint2 *>(Dp + r * kLdH + c) = make_uint2(bf16_pair(q.x, q.y), bf16_pair(q.z, q.w));
                DpT[c * kLdT + r] = bf16_bits(q.x);
                DpT[(c + 1) * kLdT + r] = bf16_bits(q.y);
                DpT[(c + 2) * kLdT + r] = bf16_bits(q.z);
                DpT[(c + 3) * kLdT + r] = bf16_bits(q.w);
            }
            // the rows the weight gradients multiply, transposed
            if (l >= 0) {
                stage_rows_t(TT, a.H[l], kH, v0, a.n, kH, kH);
                stage_rows_t(TT + kH * kLdT, a.M[l], kH, v0, a.n, kH, kH);
            } else {
                stage_rows_t(TT, a.X, a.F, v0, a.n, a.F, pad16(a.F));
            }
            __syncthreads();
            if (tid < kH) {
                float g = 0.f;
                for (int r = 0; r < kTile; ++r) g += q32[r * (kH + 4) + tid];
                atomicAdd(Gd + (l >= 0 ? a.at.b[l] : a.at.bin) + tid, g);
            }
            if (l >= 0) {
                // dH_l rows = dPre Ws^T, G = dPre Wn^T
                for (int q = warp; q < 2 * (2 * kH / 16); q += kBlock / 32) {
                    const int row0 = (q & 1) * 16, col0 = (q >> 1) * 16;
                    tile_mma(Dp, kLdH, BW, kLdH, kH, row0, col0, acc);
                    tile_pairs(acc, row0, col0, [&](const int r, const int c, const float x, const float y) {
                        if (v0 + r < a.n)
                            *reinterpret_cast<float2 *>((c < kH ? dn : Gn) + (size_t)(v0 + r) * kH + (c & (kH - 1))) = make_float2(x, y);
                    });
                }
                // dWs_l += H_l^T dPre, dWn_l += M_l^T dPre
                for (int q = warp; q < (2 * kH / 16) * (kH / 16); q += kBlock / 32) {
                    const int row0 = q / (kH / 16) * 16, col0 = q % (kH / 16) * 16;
                    tile_mma(TT, kLdT, DpT, kLdT, kTile, row0, col0, acc);
                    tile_pairs(acc, row0, col0, [&](const int r, const int c, const float x, const float y) {
                        const int o = r < kH ? a.at.ws[l] + r * kH : a.at.wn[l] + (r - kH) * kH;
                        red2(Gd + o + c, x, y, (o & 1) == 0);
                    });
                }
            } else {
                // dWin += X^T dPre0
                for (int q = warp; q < (pad16(a.F) / 16) * (kH / 16); q += kBlock / 32) {
                    const int row0 = q / (kH / 16) * 16, col0 = q % (kH / 16) * 16;
                    tile_mma(TT, kLdT, DpT, kLdT, kTile, row0, col0, acc);
                    add_grad(a.at.win, row0, col0, a.F);
                }
            }
            __syncthreads();
        }
    }
    // 4. Adam on every parameter
    if (a.train) {
        if (!gg::grid_sync(a.ctl, a.expected, a.wait_ns, kLayers + 2, epoch)) return;
        const float lr = s_hyper[kHypLr], c1 = s_hyper[kHypC1], c2 = s_hyper[kHypC2];
        for (int i = (int)blockIdx.x * kBlock + tid; i < a.n_params; i += (int)gridDim.x * kBlock) {
            const float gi = __ldcg(Gd + i);
            const float b1 = 0.9f, b2 = 0.999f;
            const float mi = b1 * a.adam_m[i] + (1.f - b1) * gi;
            const float vi = b2 * a.adam_v[i] + (1.f - b2) * gi * gi;
            a.adam_m[i] = mi;
            a.adam_v[i] = vi;
            a.params[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
        }
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// host object
// ---------------------------------------------------------------------------
struct gg_surrogate {
    int device = 0, n = 0, d = 0, F = 0;
    cudaStream_t st = nullptr;
    ParamAt at{};
    int n_params = 0;
    float *params = nullptr, *adam_m = nullptr, *adam_v = nullptr;
    int32_t *adj = nullptr;
    float *X = nullptr;
    float *Hs[kLayers + 1] = {};
    float *Ms[kLayers] = {};
    float *dH1 = nullptr, *G0 = nullptr, *G1 = nullptr;
    // What a training step zeroes, in one allocation: control block of the grid barrier,
    // loss, gradient, dL/dH3
    unsigned char *step = nullptr;
    size_t step_bytes = 0;
    float *loss = nullptr, *grad = nullptr, *dH0 = nullptr;
    // A call's swaps, then (training) targets, mask and scalars, packed for its swap count;
    // and a prediction's control block, then its results (capacity `cap` swaps): one copy
    // in, one out
    int cap = 0;
    unsigned char *in = nullptr, *h_in = nullptr, *out = nullptr, *h_out = nullptr;
    unsigned char *h_stat = nullptr;       // a training step's control block and loss
    int fwd_per_sm = 0, bwd_per_sm = 0, sms = 0;
    bool fwd_valid = false, graph_set = false;
    long long adam_step = 0;
    // captured launch sequences, per swap count: predict (with the graph
    // forward), gradient, training step
    struct Cached { int P; int kind; cudaGraphExec_t exec; };
    std::vector<Cached> graphs;
};

namespace {

gg_status sfail(gg_status s, const std::string &m) {
    (void)cudaGetLastError();
    gg::set_last_error(m.c_str());
    return s;
}

#define GS_CK(call)                                                                          \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess)                                                               \
            return sfail(e_ == cudaErrorMemoryAllocation ? GG_OUT_OF_MEMORY : GG_CUDA_ERROR, \
                         std::string(#call) + ": " + cudaGetErrorString(e_));                \
    } while (0)


void drop_graphs(gg_surrogate *s) {
    for (auto &c : s->graphs) cudaGraphExecDestroy(c.exec);
    s->graphs.clear();
}

constexpr size_t kCtlBytes = 256;                  // sizeof(gg::Ctl)
constexpr size_t kStepHead = kCtlBytes + 256;      // control block and loss
static_assert(sizeof(gg::Ctl) == kCtlBytes, "control block size");

// Bytes of a call's packed input for P swaps, and where its parts start.
size_t in_t(int P) { return (size_t)P * sizeof(gg_swap); }
size_t in_mask(int P) { return in_t(P) + (size_t)P * 4; }
size_t in_hyper(int P) { return in_mask(P) + (size_t)P * 4; }
size_t in_bytes(int P) { return in_hyper(P) + kHypN * 4; }

gg_status ensure_swaps(gg_surrogate *s, int P) {
    if (P <= s->cap) return GG_OK;
    const int cap = std::max(P, 2 * s->cap);
    drop_graphs(s);
    cudaFree(s->in); cudaFree(s->out);
    cudaFreeHost(s->h_in); cudaFreeHost(s->h_out);
    s->in = s->out = s->h_in = s->h_out = nullptr;
    s->cap = 0;
    GS_CK(cudaMalloc(&s->in, in_bytes(cap)));
    GS_CK(cudaMallocHost(&s->h_in, in_bytes(cap)));
    GS_CK(cudaMalloc(&s->out, kCtlBytes + (size_t)cap * 4));
    GS_CK(cudaMallocHost(&s->h_out, kCtlBytes + (size_t)cap * 4));
    s->cap = cap;
    return GG_OK;
}

int barrier_err(const unsigned char *ctl) { return reinterpret_cast<const gg::Ctl *>(ctl)->err; }

// One launch (surrogate_forward_kernel): the embeddings of the current graph, then the
// readout of P swaps when P > 0; control block and results in s->out.
void forward(gg_surrogate *s, int P) {
    FwdArgs a{};
    a.X = s->X; a.F = s->F; a.adj = s->adj; a.n = s->n; a.d = s->d;
    a.P = s->params; a.at = s->at;
    for (int l = 0; l <= kLayers; ++l) a.H[l] = s->Hs[l];
    for (int l = 0; l < kLayers; ++l) a.M[l] = s->Ms[l];
    a.sw = reinterpret_cast<const gg_swap *>(s->in); a.n_sw = P;
    a.y = reinterpret_cast<float *>(s->out + kCtlBytes);
    const int tiles = std::max((s->n + kTile - 1) / kTile, (P + kTile - 1) / kTile);
    const int grid = std::max(1, std::min(s->fwd_per_sm * s->sms, tiles));
    a.ctl = reinterpret_cast<gg::Ctl *>(s->out);
    a.expected = (unsigned)grid;
    a.wait_ns = 10ll * 1000 * 1000 * 1000;
    cudaMemsetAsync(s->out, 0, kCtlBytes, s->st);
    void *args[] = {&a};
    cudaLaunchCooperativeKernel((void *)surrogate_forward_kernel, dim3(grid), dim3(kBlock), args, fwd_smem(s->F), s->st);
    cudaMemcpyAsync(s->h_out, s->out, kCtlBytes + (size_t)P * 4, cudaMemcpyDeviceToHost, s->st);
}

// Loss and full gradient into s->grad for the packed input of P swaps on the device, and
// with `train` the Adam step: one launch (surrogate_backward_kernel) after one memset.
void backward(gg_surrogate *s, int P, bool train) {
    cudaMemsetAsync(s->step, 0, s->step_bytes, s->st);
    BwdArgs a{};
    a.X = s->X; a.F = s->F; a.adj = s->adj; a.n = s->n; a.d = s->d;
    a.P = s->params; a.Gd = s->grad; a.at = s->at;
    for (int l = 0; l <= kLayers; ++l) a.H[l] = s->Hs[l];
    for (int l = 0; l < kLayers; ++l) a.M[l] = s->Ms[l];
    a.sw = reinterpret_cast<const gg_swap *>(s->in); a.n_sw = P;
    a.t = reinterpret_cast<const float *>(s->in + in_t(P));
    a.mask = reinterpret_cast<const int32_t *>(s->in + in_mask(P));
    a.hyper = reinterpret_cast<const float *>(s->in + in_hyper(P));
    a.dH[0] = s->dH0; a.dH[1] = s->dH1; a.G[0] = s->G0; a.G[1] = s->G1; a.loss = s->loss;
    a.adam_m = s->adam_m; a.adam_v = s->adam_v; a.params = s->params;
    a.n_params = s->n_params; a.train = train ? 1 : 0;
    // a block a tile, and no more than can be resident
    const int tiles = std::max((s->n + kTile - 1) / kTile, (P + kTile - 1) / kTile);
    const int grid = std::max(1, std::min(s->bwd_per_sm * s->sms, tiles));
    a.ctl = reinterpret_cast<gg::Ctl *>(s->step);
    a.expected = (unsigned)grid;
    a.wait_ns = 10ll * 1000 * 1000 * 1000;
    void *args[] = {&a};
    cudaLaunchCooperativeKernel((void *)surrogate_backward_kernel, dim3(grid), dim3(kBlock), args, bwd_smem(s->F), s->st);
}

enum { kPredict = 0, kGrad = 1, kTrain = 2 };

// The launch sequence of one call kind for P swaps, staged from/to pinned memory.
void enqueue_kind(gg_surrogate *s, int kind, int P) {
    cudaMemcpyAsync(s->in, s->h_in, kind == kPredict ? in_t(P) : in_bytes(P), cudaMemcpyHostToDevice, s->st);
    if (kind == kPredict) {
        forward(s, P);
        return;
    }
    backward(s, P, kind == kTrain);
    cudaMemcpyAsync(s->h_stat, s->step, kStepHead, cudaMemcpyDeviceToHost, s->st);
}

// Replay (capturing on first use) the sequence `kind` for P swaps, then wait.
gg_status run_kind(gg_surrogate *s, int kind, int P) {
    cudaGraphExec_t exec = nullptr;
    for (auto &c : s->graphs)
        if (c.P == P && c.kind == kind) exec = c.exec;
    if (!exec) {
        GS_CK(cudaStreamBeginCapture(s->st, cudaStreamCaptureModeThreadLocal));
        enqueue_kind(s, kind, P);
        cudaGraph_t g = nullptr;
        GS_CK(cudaStreamEndCapture(s->st, &g));
        const cudaError_t e = cudaGraphInstantiate(&exec, g, 0);
        cudaGraphDestroy(g);
        GS_CK(e);
        s->graphs.push_back({P, kind, exec});
    }
    GS_CK(cudaGraphLaunch(exec, s->st));
    GS_CK(cudaStreamSynchronize(s->st));
    if (barrier_err(kind == kPredict ? s->h_out : s->h_stat))
        return sfail(GG_TIMEOUT, kind == kPredict ? "grid barrier wait of the fused forward exceeded its limit"
                                                  : "grid barrier wait of the fused backward exceeded its limit");
    return GG_OK;
}

gg_status stage_swaps(gg_surrogate *s, int P, const gg_swap *swaps) {
    for (int i = 0; i < P; ++i) {
        const gg_swap &w = swaps[i];
        if (w.a < 0 || w.a >= s->n || w.b < 0 || w.b >= s->n || w.c < 0 || w.c >= s->n || w.d < 0 ||
            w.d >= s->n || (w.mode != 0 && w.mode != 1))
            return sfail(GG_BAD_ARG, "swap " + std::to_string(i) + " out of range");
    }
    gg_status r = ensure_swaps(s, P);
    if (r != GG_OK) return r;
    std::memcpy(s->h_in, swaps, (size_t)P * sizeof(gg_swap));
    return GG_OK;
}

gg_status grad_common(gg_surrogate *s, int kind, int P, const gg_swap *swaps, const float *target,
                      const int32_t *mask, float lr, float *loss) {
    if (!s || P < 1 || !swaps || !target) return sfail(GG_BAD_ARG, "bad arguments");
    if (!s->graph_set) return sfail(GG_BAD_ARG, "no graph set");
    GS_CK(cudaSetDevice(s->device));
    gg_status r = stage_swaps(s, P, swaps);
    if (r != GG_OK) return r;
    int cnt = 0;
    int32_t *h_mask = reinterpret_cast<int32_t *>(s->h_in + in_mask(P));
    float *h_hyper = reinterpret_cast<float *>(s->h_in + in_hyper(P));
    for (int i = 0; i < P; ++i) {
        h_mask[i] = mask ? (mask[i] != 0) : 1;
        cnt += h_mask[i];
    }
    std::memcpy(s->h_in + in_t(P), target, (size_t)P * 4);
    h_hyper[kHypInvCnt] = cnt ? 1.f / (float)cnt : 0.f;
    h_hyper[kHypLr] = lr;
    h_hyper[kHypC1] = h_hyper[kHypC2] = 0.f;
    if (kind == kTrain) {
        const long long t = s->adam_step + 1;
        h_hyper[kHypC1] = 1.f - std::pow(0.9f, (float)t);
        h_hyper[kHypC2] = 1.f - std::pow(0.999f, (float)t);
    }
    if (!s->fwd_valid) {  // embeddings of the current graph and parameters
        forward(s, 0);
        GS_CK(cudaGetLastError());
        GS_CK(cudaStreamSynchronize(s->st));
        if (barrier_err(s->h_out)) return sfail(GG_TIMEOUT, "grid barrier wait of the fused forward exceeded its limit");
        s->fwd_valid = true;
    }
    r = run_kind(s, kind, P);
    if (r != GG_OK) return r;
    if (kind == kTrain) {
        s->adam_step += 1;
        s->fwd_valid = false;
    }
    if (loss) *loss = *reinterpret_cast<const float *>(s->h_stat + kCtlBytes);
    return GG_OK;
}

}  // namespace

extern "C" {

gg_status gg_surrogate_create(int device, int n, int degree, int in_features, uint64_t seed,
                              gg_surrogate **out) {
    if (!out || n < 2 || degree < 1 || in_features < 1 || in_features > 256)
        return sfail(GG_BAD_ARG, "need n >= 2, degree >= 1, 1 <= in_features <= 256");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return sfail(GG_NO_DEVICE, "no CUDA device");
    if (device < 0 || device >= ndev) return sfail(GG_NO_DEVICE, "device index out of range");
    gg_surrogate *s = new gg_surrogate();
    s->device = device; s->n = n; s->d = degree; s->F = in_features;
    int o = 0;
    s->at.win = o; o += in_features * kH;
    s->at.bin = o; o += kH;
    for (int l = 0; l < kLayers; ++l) {
        s->at.ws[l] = o; o += kH * kH;
        s->at.wn[l] = o; o += kH * kH;
        s->at.b[l] = o; o += kH;
    }
    s->at.wr1 = o; o += kZ * kH;
    s->at.br1 = o; o += kH;
    s->at.wr2 = o; o += kH;
    s->at.br2 = o; o += 1;
    s->n_params = o;
    // Glorot-uniform weights, zero biases, from a seeded host generator
    std::vector<float> p(o, 0.f);
    uint64_t x = seed * 0x9e3779b97f4a7c15ull + 1;
    auto unif = [&]() {
        x ^= x << 13; x ^= x >> 7; x ^= x << 17;  // xorshift64
        return (double)(x >> 11) * (1.0 / 9007199254740992.0);
    };
    auto fill = [&](int off, int fin, int fout) {
        const double a = std::sqrt(6.0 / (fin + fout));
        for (int i = 0; i < fin * fout; ++i) p[off + i] = (float)((2 * unif() - 1) * a);
    };
    fill(s->at.win, in_features, kH);
    for (int l = 0; l < kLayers; ++l) { fill(s->at.ws[l], kH, kH); fill(s->at.wn[l], kH, kH); }
    fill(s->at.wr1, kZ, kH);
    fill(s->at.wr2, kH, 1);
    auto bad = [&](gg_status st) { gg_surrogate_destroy(s); return st; };
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&s->st, cudaStreamNonBlocking) != cudaSuccess)
        return bad(sfail(GG_CUDA_ERROR, "stream creation failed"));
    const size_t pb = (size_t)o * 4, gb = (pb + 255) / 256 * 256;
    s->step_bytes = kStepHead + gb + (size_t)n * kH * 4;
    bool ok = cudaMalloc(&s->params, pb) == cudaSuccess && cudaMalloc(&s->adam_m, pb) == cudaSuccess &&
              cudaMalloc(&s->adam_v, pb) == cudaSuccess &&
              cudaMalloc(&s->adj, (size_t)n * degree * 4) == cudaSuccess &&
              cudaMalloc(&s->X, (size_t)n * in_features * 4) == cudaSuccess &&
              cudaMalloc(&s->dH1, (size_t)n * kH * 4) == cudaSuccess &&
              cudaMalloc(&s->G0, (size_t)n * kH * 4) == cudaSuccess && cudaMalloc(&s->G1, (size_t)n * kH * 4) == cudaSuccess &&
              cudaMalloc(&s->step, s->step_bytes) == cudaSuccess && cudaMallocHost(&s->h_stat, kStepHead) == cudaSuccess;
    for (int l = 0; l <= kLayers && ok; ++l) ok = cudaMalloc(&s->Hs[l], (size_t)n * kH * 4) == cudaSuccess;
    for (int l = 0; l < kLayers && ok; ++l) ok = cudaMalloc(&s->Ms[l], (size_t)n * kH * 4) == cudaSuccess;
    if (!ok) return bad(sfail(GG_OUT_OF_MEMORY, "surrogate allocation failed"));
    s->loss = reinterpret_cast<float *>(s->step + kCtlBytes);
    s->grad = reinterpret_cast<float *>(s->step + kStepHead);
    s->dH0 = reinterpret_cast<float *>(s->step + kStepHead + gb);
    if (cudaFuncSetAttribute(surrogate_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem(kFmax)) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&s->fwd_per_sm, surrogate_forward_kernel, kBlock, fwd_smem(in_features)) !=
            cudaSuccess ||
        cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || s->fwd_per_sm < 1)
        return bad(sfail(GG_CUDA_ERROR, "fused forward cannot be resident"));
    if (cudaFuncSetAttribute(surrogate_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bwd_smem(kFmax)) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&s->bwd_per_sm, surrogate_backward_kernel, kBlock, bwd_smem(in_features)) !=
            cudaSuccess ||
        s->bwd_per_sm < 1)
        return bad(sfail(GG_CUDA_ERROR, "fused backward cannot be resident"));
    if (cudaMemcpyAsync(s->params, p.data(), pb, cudaMemcpyHostToDevice, s->st) != cudaSuccess ||
        cudaMemsetAsync(s->adam_m, 0, pb, s->st) != cudaSuccess || cudaMemsetAsync(s->adam_v, 0, pb, s->st) != cudaSuccess ||
        cudaStreamSynchronize(s->st) != cudaSuccess)
        return bad(sfail(GG_CUDA_ERROR, "surrogate initialisation failed"));
    *out = s;
    return GG_OK;
}

gg_status gg_surrogate_set_graph(gg_surrogate *s, const int32_t *adj, const float *features) {
    if (!s || !adj || !features) return sfail(GG_BAD_ARG, "null argument");
    for (long long k = 0; k < (long long)s->n * s->d; ++k)
        if (adj[k] < 0 || adj[k] >= s->n) return sfail(GG_BAD_ARG, "adjacency entry outside [0, n)");
    GS_CK(cudaSetDevice(s->device));
    GS_CK(cudaMemcpyAsync(s->adj, adj, (size_t)s->n * s->d * 4, cudaMemcpyHostToDevice, s->st));
    GS_CK(cudaMemcpyAsync(s->X, features, (size_t)s->n * s->F * 4, cudaMemcpyHostToDevice, s->st));
    s->graph_set = true;
    s->fwd_valid = false;
    GS_CK(cudaStreamSynchronize(s->st));
    return GG_OK;
}

gg_status gg_surrogate_predict(gg_surrogate *s, int P, const gg_swap *swaps, float *pred) {
    if (!s || P < 0 || (P && (!swaps || !pred))) return sfail(GG_BAD_ARG, "bad arguments");
    if (!s->graph_set) return sfail(GG_BAD_ARG, "no graph set");
    if (P == 0) return GG_OK;
    GS_CK(cudaSetDevice(s->device));
    gg_status r = stage_swaps(s, P, swaps);
    if (r != GG_OK) return r;
    r = run_kind(s, kPredict, P);  // recomputes the embeddings: they are valid afterwards
    if (r != GG_OK) return r;
    s->fwd_valid = true;
    std::memcpy(pred, s->h_out + kCtlBytes, (size_t)P * 4);
    return GG_OK;
}

gg_status gg_surrogate_grad(gg_surrogate *s, int P, const gg_swap *swaps, const float *target,
                            const int32_t *mask, float *grad, float *loss) {
    if (!grad) return sfail(GG_BAD_ARG, "null grad");
    gg_status r = grad_common(s, kGrad, P, swaps, target, mask, 0.f, loss);
    if (r != GG_OK) return r;
    GS_CK(cudaMemcpy(grad, s->grad, (size_t)s->n_params * 4, cudaMemcpyDeviceToHost));
    return GG_OK;
}

gg_status gg_surrogate_train(gg_surrogate *s, int P, const gg_swap *swaps, const float *target,
                             const int32_t *mask, float lr, float *loss) {
    return grad_common(s, kTrain, P, swaps, target, mask, lr, loss);
}

gg_status gg_surrogate_param_count(gg_surrogate *s, int *count) {
    if (!s || !count) return sfail(GG_BAD_ARG, "null argument");
    *count = s->n_params;
    return GG_OK;
}

gg_status gg_surrogate_get_params(gg_surrogate *s, float *params) {
    if (!s || !params) return sfail(GG_BAD_ARG, "null argument");
    GS_CK(cudaSetDevice(s->device));
    GS_CK(cudaMemcpy(params, s->params, (size_t)s->n_params * 4, cudaMemcpyDeviceToHost));
    return GG_OK;
}

gg_status gg_surrogate_set_params(gg_surrogate *s, const float *params) {
    if (!s || !params) return sfail(GG_BAD_ARG, "null argument");
    GS_CK(cudaSetDevice(s->device));
    GS_CK(cudaMemcpyAsync(s->params, params, (size_t)s->n_params * 4, cudaMemcpyHostToDevice, s->st));
    s->fwd_valid = false;
    GS_CK(cudaStreamSynchronize(s->st));
    return GG_OK;
}

gg_status gg_surrogate_destroy(gg_surrogate *s) {
    if (!s) return GG_OK;
    cudaSetDevice(s->device);
    if (s->st) cudaStreamSynchronize(s->st);
    drop_graphs(s);
    cudaFree(s->params); cudaFree(s->adam_m); cudaFree(s->adam_v); cudaFree(s->step); cudaFreeHost(s->h_stat);
    cudaFree(s->adj); cudaFree(s->X); cudaFree(s->dH1); cudaFree(s->G0); cudaFree(s->G1);
    for (auto p : s->Hs) cudaFree(p);
    for (auto p : s->Ms) cudaFree(p);
    cudaFree(s->in); cudaFree(s->out); cudaFreeHost(s->h_in); cudaFreeHost(s->h_out);
    if (s->st) cudaStreamDestroy(s->st);
    delete s;
    return GG_OK;
}

}  // extern "C"
