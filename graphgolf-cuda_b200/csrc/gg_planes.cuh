// gg_planes.cuh -- per-source statistics of a distance matrix kept as bit-planes,
// and the symmetry test that makes them cheap.
//
// Plane layout (BfsArgs::planes in gg_kernels.cuh): bit s % 128 of
// planes[k * stride + v * cols + s / 128] is bit k of dist(source s, vertex v);
// bits of columns past the last source and of unreached pairs are 0.
//
// On a symmetric adjacency (u in adj[v] <=> v in adj[u]) the distance matrix is
// symmetric, so source s's distance sum and eccentricity are reductions along
// ROW v = s: a popcount of each plane weighted by 2^k, and a most-significant-
// plane-first search for the largest value.  One warp per row, coalesced 16-byte
// loads along it: one read of the planes, no transposition.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

// ---- bit-sliced distances: four plane words hold 32 sources' distances ------------
struct Dist4 {
    uint32_t p[4];
};
__device__ __forceinline__ Dist4 dist4_load(const uint32_t *planes, const size_t stride, const size_t at) {
    Dist4 d;
#pragma unroll
    for (int k = 0; k < 4; ++k) d.p[k] = __ldg(planes + (size_t)k * stride + at);
    return d;
}
__device__ __forceinline__ Dist4 dist4_const(const unsigned v) {
    Dist4 d;
#pragma unroll
    for (int k = 0; k < 4; ++k) d.p[k] = (v >> k) & 1u ? 0xffffffffu : 0u;
    return d;
}
__device__ __forceinline__ Dist4 dist4_inc(const Dist4 a) {
    Dist4 r;
    uint32_t c = 0xffffffffu;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        r.p[k] = a.p[k] ^ c;
        c &= a.p[k];
    }
    return r;
}
// a == b, a < b, per source
__device__ __forceinline__ uint32_t dist4_eq(const Dist4 a, const Dist4 b) {
    uint32_t x = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) x |= a.p[k] ^ b.p[k];
    return ~x;
}
__device__ __forceinline__ uint32_t dist4_lt(const Dist4 a, const Dist4 b) {
    uint32_t lt = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) lt = (~a.p[k] & b.p[k]) | (~(a.p[k] ^ b.p[k]) & lt);
    return lt;
}
// the sum of the distances of the sources in `mask`
__device__ __forceinline__ unsigned dist4_sum(const Dist4 a, const uint32_t mask) {
    return __popc(a.p[0] & mask) + 2u * __popc(a.p[1] & mask) + 4u * __popc(a.p[2] & mask) + 8u * __popc(a.p[3] & mask);
}

// What one replaced pull entry of a 2-opt (row r lists t in place of f) does to 32 sources
// (word w of the planes): `aff` -- the row loses its last parent, or the added edge
// shortens it; `near` -- the source lies within `radius` of r.  The rows' plane words are
// coalesced over the lanes' words, four neighbours' loads in flight together.
__device__ __forceinline__ void edit_masks(const uint32_t *pw, const size_t ps, const size_t cw, const int32_t *adj,
                                           const int d, const int r, const int f, const int t, const unsigned w,
                                           const unsigned radius, uint32_t &aff, uint32_t &near) {
    const Dist4 er = dist4_load(pw, ps, (size_t)r * cw + w);
    const Dist4 ef = dist4_load(pw, ps, (size_t)f * cw + w);
    const Dist4 et = dist4_load(pw, ps, (size_t)t * cw + w);
    uint32_t lost = dist4_eq(dist4_inc(ef), er);
    bool skipped = false;   // the first slot that lists f is the one that goes
    for (int j = 0; j < d; j += 4) {
        int u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            u[k] = __ldg(adj + (size_t)r * d + min(j + k, d - 1));
            if (j + k < d && !skipped && u[k] == f) { u[k] = r; skipped = true; }   // (r itself is no parent)
            if (j + k >= d) u[k] = r;
        }
        Dist4 x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = dist4_load(pw, ps, (size_t)u[k] * cw + w);
#pragma unroll
        for (int k = 0; k < 4; ++k) lost &= ~dist4_eq(x[k], ef);
    }
    aff = lost | dist4_lt(dist4_inc(et), er);
    near = ~dist4_lt(dist4_const(radius), er);
}

// Distance sum and eccentricity of every source; with `top`, also the number of its
// vertices at distance `diam`.
template <int NP>
static __global__ void plane_row_stats(const uint4 *planes, unsigned long long stride, unsigned cols, int n,
                                       unsigned *rowsum, unsigned *ecc, unsigned *top = nullptr, unsigned diam = 0u) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
    for (unsigned long long v = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < (unsigned)n;
         v += nwarps) {
        const uint4 *row = planes + v * cols;
        unsigned sum = 0, mx = 0, tops = 0;
#pragma unroll 2
        for (unsigned c = lane; c < cols; c += 32) {
            uint4 w[NP];
#pragma unroll
            for (int p = 0; p < NP; ++p) w[p] = __ldg(row + (size_t)p * stride + c);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                unsigned cand = 0xffffffffu, val = 0;
#pragma unroll
                for (int p = NP - 1; p >= 0; --p) {
                    const unsigned x = k == 0 ? w[p].x : k == 1 ? w[p].y : k == 2 ? w[p].z : w[p].w;
                    sum += (unsigned)__popc(x) << p;
                    const unsigned hit = cand & x;
                    if (hit) {
                        cand = hit;
                        val |= 1u << p;
                    }
                }
                mx = max(mx, val);
                if (top) {
                    unsigned at = 0xffffffffu;   // (planes past the last source are 0: diam >= 1)
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
                        const unsigned x = k == 0 ? w[p].x : k == 1 ? w[p].y : k == 2 ? w[p].z : w[p].w;
                        at &= (diam >> p) & 1u ? x : ~x;
                    }
                    tops += (unsigned)__popc(at);
                }
            }
        }
        sum = __reduce_add_sync(0xffffffffu, sum);
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (top) tops = __reduce_add_sync(0xffffffffu, tops);
        if (lane == 0) {
            if (top) top[v] = tops;
            rowsum[v] = sum;
            ecc[v] = mx;
        }
    }
}

// 1 into *asym when some entry u of row v has no entry v in row u (one thread
// per entry; entries outside [0, n) are the caller's to reject first).
static __global__ void table_symmetry(const int32_t *adj, int n, int d, int *asym) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= (long long)n * d) return;
    const int v = (int)(k / d), u = adj[k];
    bool back = false;
    for (int j = 0; j < d && !back; ++j) back = adj[(size_t)u * d + j] == v;
    if (!back) *asym = 1;
}

// Launch shape of plane_row_stats: one warp per row, at most 8 blocks of 8
// warps per SM in flight.
static inline int plane_row_stats_grid(int n, int sms) {
    const long long blocks = ((long long)n + 7) / 8;
    return (int)(blocks < (long long)sms * 8 ? blocks : (long long)sms * 8);
}
