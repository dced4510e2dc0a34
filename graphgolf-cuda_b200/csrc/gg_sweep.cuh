// Balls of a few steps and the dense levels after them, when every vertex is a source (or,
// for a lift, one vertex of each orbit) and the table has no one-way entries: ball_kernel
// or source_ball_kernel, then sweep_kernel<D>.  bfs_batch_kernel does the same job in general;
// this one takes the plain case, where each level is a whole dense pull, and ends each
// batch with last_rows.
//
// last_rows (one pass in place of the last two levels).  Distances are symmetric, so
// with every vertex a source, of the pairs the levels before L left over it looks only at those whose vertex is
// in the source's batch or a later one, and counts the later ones twice: half of the
// rows on average.  A row's chunk that level L does not fill is finished on the spot
// from two steps away, V_{L+1}[v] = OR of V_{L-1}[w] over the walks v-u-w (the rows of
// level L - 1 are all there and nothing overwrites them), so neither level writes rows
// and no barrier lies between them.  All batches take it at the same level, the one
// batch 0 finds (else pairs would be counted twice or not at all), and the counts add
// up over the batches only: a batch's own may be off, or "negative", mod 2^64.
//
// Measured, whole calls: n = 65536, d = 8: 1925 us with bfs_batch_kernel, 1225 here; n =
// 30011, d = 6, irregular: 766 / 390; n = 40000, d = 10: 1857 / 617; n = 16384, d = 6:
// 302 / 187.  Of the 1225: ball_kernel 265, per 8192-source batch two levels of 45 (rows
// from HBM) and 39 us and last_rows 27 falling to 7, the table's way to the device 100.
// A level is bound by the gathers' way from L2: 537 MB in 39 us (ncu on 4096-source
// batches: L2 at 46 %, warps waiting for loads), 148 blocks finishing within 2 us.
//
// When something does not fit -- a one-way entry, a thin level (flag words would be
// better), the level cap, a pair further than L + 1 -- *redo is set and the host runs
// bfs_batch_kernel instead.
#pragma once
#include "gg_kernels.cuh"

namespace gg {

// ---------------------------------------------------------------------------
// ball_kernel<D, K>: the rows V_K of every batch, one warp per row.  Row v is a bit string
// over all vertices in shared memory (8 KB at 65536); the ends of v's walks of up to K
// steps set their bits -- neighbours, the level-2 list of v, those of its neighbours
// (level 3) and, K = 4, those of its level-2 ends other than v -- and the row goes out
// once, each 4096-source part to its batch.  An end is new at its level when atomicOr
// returns its bit clear; the last level's count is the row's popcount less the others'.
//
// Bound by the shared-memory atomics (d^K ends a row, random banks).
// ---------------------------------------------------------------------------
constexpr int kBallBlock = 256;
constexpr int kBallCounts = 256;   // batches * K

struct BallArgs {
    const int32_t *adj, *h2;  // [rows][D], [rows][D * D]
    const int *bad, *oneway;
    uint4 *vall;              // [nb][rows][nC]
    unsigned long long *counts;   // [nb][stride]: levels 1..K added
    int stride;
    int rows, nC, nb;
};

__host__ __device__ constexpr int ball_warp_bytes(int D, int K, int parts) {
    return parts * 512 + (K == 4 ? D * D * 4 + 15 : D * 4 + 15) / 16 * 16;
}

template <int D, int K>
__global__ void __launch_bounds__(kBallBlock, 3) ball_kernel(const __grid_constant__ BallArgs a) {
    extern __shared__ __align__(16) unsigned char s_ball[];
    __shared__ unsigned long long s_cnt[kBallCounts];
    if ((a.bad && *a.bad) || ld_acquire_i(a.oneway) != 0) return;   // (one-way: sweep_kernel says so)
    constexpr int Q = D * D, V = Q % 4 == 0 ? 4 : 1, SL = Q / V;    // a list: SL slots of V ends
    constexpr int UN = V == 4 ? 4 : 8;                              // slots a lane has in flight
    const unsigned lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const int sub = a.nC / 32, parts = a.nb * sub;
    for (int k = (int)threadIdx.x; k < a.nb * K; k += (int)blockDim.x) s_cnt[k] = 0ull;
    uint4 *row4 = reinterpret_cast<uint4 *>(s_ball + (size_t)wib * ball_warp_bytes(D, K, parts));
    unsigned *row = reinterpret_cast<unsigned *>(row4);
    int *list = reinterpret_cast<int *>(row4 + parts * 32);
    for (int p = 0; p < parts; ++p) row4[p * 32 + lane] = u4zero();
    __syncthreads();
    auto add = [&](const unsigned w) -> unsigned {   // 1 when w's bit was clear
        const unsigned bit = 1u << (w & 31u);
        return (atomicOr(row + (w >> 5), bit) & bit) == 0u;
    };
    auto put = [&](const unsigned w) { atomicOr(row + (w >> 5), 1u << (w & 31u)); };
    // The ends in the level-2 lists of list[0 .. n): f on each.
    auto lists = [&](const int n, auto &&f) {
        const int slots = n * SL;
        for (int i0 = (int)lane; i0 < slots; i0 += 32 * UN) {
            if constexpr (V == 4) {
                uint4 q[UN];
#pragma unroll
                for (int k = 0; k < UN; ++k) {
                    const int i = i0 + 32 * k;
                    if (i < slots) {
                        const int j = i / SL;
                        q[k] = __ldg(reinterpret_cast<const uint4 *>(a.h2 + (size_t)list[j] * Q) + (i - j * SL));
                    }
                }
#pragma unroll
                for (int k = 0; k < UN; ++k)
                    if (i0 + 32 * k < slots) { f(q[k].x); f(q[k].y); f(q[k].z); f(q[k].w); }
            } else {
                unsigned q[UN];
#pragma unroll
                for (int k = 0; k < UN; ++k) {
                    const int i = i0 + 32 * k;
                    if (i < slots) {
                        const int j = i / SL;
                        q[k] = (unsigned)__ldg(a.h2 + (size_t)list[j] * Q + (i - j * SL));
                    }
                }
#pragma unroll
                for (int k = 0; k < UN; ++k)
                    if (i0 + 32 * k < slots) f(q[k]);
            }
        }
    };
    const size_t items = (size_t)a.rows * (size_t)a.nC;
    for (int v = (int)(blockIdx.x * (kBallBlock / 32) + wib); v < a.rows; v += (int)(gridDim.x * (kBallBlock / 32))) {
        unsigned n1 = 0u, n2 = 0u, n3 = 0u, all = 0u;
        int mine[(Q + 31) / 32];   // this lane's share of v's level-2 list
#pragma unroll
        for (int k = 0; k < (Q + 31) / 32; ++k) {
            const int i = (int)lane + 32 * k;
            mine[k] = i < Q ? __ldg(a.h2 + (size_t)v * Q + i) : v;
        }
        if (lane == 0) put((unsigned)v);
        int u = v;
        if (lane < (unsigned)D) {
            u = __ldg(a.adj + (size_t)v * D + lane);
            list[lane] = u;
        }
        __syncwarp();
        if (lane < (unsigned)D) n1 = add((unsigned)u);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < (Q + 31) / 32; ++k)
            if (mine[k] != v) n2 += add((unsigned)mine[k]);
        __syncwarp();
        if constexpr (K == 4) {
            lists(D, [&](const unsigned w) { n3 += add(w); });
            __syncwarp();
            // the level-2 ends other than v itself (its list is set)
            int n = 0;
#pragma unroll
            for (int k = 0; k < (Q + 31) / 32; ++k) {
                const unsigned m = __ballot_sync(0xffffffffu, mine[k] != v);
                if (mine[k] != v) list[n + __popc(m & ((1u << lane) - 1u))] = mine[k];
                n += __popc(m);
            }
            __syncwarp();
            lists(n, put);
        } else {
            lists(D, put);
        }
        __syncwarp();
        uint4 *out = a.vall + (size_t)v * a.nC + lane;
        for (int p = 0, c = 0; p < parts; ++p) {
            uint4 q = row4[p * 32 + lane];
            row4[p * 32 + lane] = u4zero();
            if (a.rows < (p + 1) * 4096) q = u4or(q, pad_mask((int)lane, a.rows - p * 4096));
            all += u4popc(q);
            __stcs(out + c * 32, q);
            if (++c == sub) {
                c = 0;
                out += items;
            }
        }
        n1 = __reduce_add_sync(0xffffffffu, n1);
        n2 = __reduce_add_sync(0xffffffffu, n2);
        if (K == 4) n3 = __reduce_add_sync(0xffffffffu, n3);
        all = __reduce_add_sync(0xffffffffu, all) - (unsigned)(parts * 4096 - a.rows) - 1u - n1 - n2 - n3;
        if (lane == 0) {
            unsigned long long *c = s_cnt + v / (128 * a.nC) * K;
            atomicAdd(c, (unsigned long long)n1);
            atomicAdd(c + 1, (unsigned long long)n2);
            if (K == 4) atomicAdd(c + 2, (unsigned long long)n3);
            atomicAdd(c + K - 1, (unsigned long long)all);
        }
        __syncwarp();
    }
    __syncthreads();
    for (int k = (int)threadIdx.x; k < a.nb * K; k += (int)blockDim.x)
        if (s_cnt[k]) atomicAdd(a.counts + (size_t)(k / K) * a.stride + k % K + 1, s_cnt[k]);
}

// ---------------------------------------------------------------------------
// source_ball_kernel<D>: the same rows for a list of sources (the orbits of a lift), from
// the sources' side: one warp walks out from a source, level by level over the new
// vertices, with a bit per vertex in shared memory, and sets its own bit in each vertex's
// row by a reduction in L2.  The rows hold the padding beforehand (expand_kernel).  The
// blocks after ball_blocks do the table's one-way check meanwhile (the lists are as long
// as the levels need, so that those find room: 16 -> 11 us at 32768 rows of 8).
// A lift's sources are few: from the rows' side all of them would walk.
// Bound by the reductions (41 a ns) and, at two levels, by its round trips.  Whole calls,
// bfs_batch_kernel first: cyclic lift of 1024 x 32, d = 12: 118 -> 104 us; 2-D lift of
// 32768 vertices, 1024 orbits, d = 8: 120 -> 97; 60000 vertices, 2000 orbits, d = 4: 240 ->
// 136; 60000, 4000, d = 12: 362 -> 209; 50000, 10000, d = 8: 422 -> 393.
// ---------------------------------------------------------------------------
constexpr int kSrcBallBlock = 128;
constexpr int kSrcBallList = 1024;   // most new vertices of a level that a warp walks on from
constexpr int kSrcBallLevels = 16;

struct SourceBallArgs {
    const int32_t *adj;       // [rows][D]
    const int32_t *src;       // sources, or nullptr: src_first, src_first + 1, ...
    int src_first, ns_total;
    unsigned *vall;           // [nb][rows][nC] uint4
    unsigned long long *counts;
    int stride;
    int *oneway;
    int rows, nC, K;
    int list;                 // most new vertices of a level below K: D^(K-1), one-way entries included
    int ball_blocks;
};

__host__ __device__ constexpr int source_ball_warp_bytes(int rows, int list) {
    return (rows + 127) / 128 * 16 + 2 * ((list + 3) / 4 * 4) * 4;
}

template <int D>
__global__ void __launch_bounds__(kSrcBallBlock) source_ball_kernel(const __grid_constant__ SourceBallArgs a) {
    extern __shared__ __align__(16) unsigned char s_ball[];
    __shared__ unsigned s_cnt[kSrcBallLevels];
    if ((int)blockIdx.x >= a.ball_blocks) {
        const long long n = (long long)a.rows * D;
        for (long long k = (long long)(blockIdx.x - a.ball_blocks) * blockDim.x + threadIdx.x; k < n;
             k += (long long)(gridDim.x - a.ball_blocks) * blockDim.x) {
            const int v = (int)(k / D);
            const int32_t *ur = a.adj + (size_t)__ldg(a.adj + k) * D;
            bool f = false;
#pragma unroll
            for (int j = 0; j < D; ++j) f |= __ldg(ur + j) == v;
            if (!f) *a.oneway = 1;
        }
        return;
    }
    const unsigned lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const int words4 = (a.rows + 127) / 128;
    uint4 *set4 = reinterpret_cast<uint4 *>(s_ball + (size_t)wib * source_ball_warp_bytes(a.rows, a.list));
    unsigned *set = reinterpret_cast<unsigned *>(set4);
    int *lists = reinterpret_cast<int *>(set4 + words4);
    const int S = 128 * a.nC, half = (a.list + 3) / 4 * 4;
    const int j = (int)(blockIdx.x * (kSrcBallBlock / 32) + wib);   // (a batch's sources are whole blocks)
    if (threadIdx.x < kSrcBallLevels) s_cnt[threadIdx.x] = 0u;
    __syncthreads();
    if (j < a.ns_total) {
        for (int i = (int)lane; i < words4; i += 32) set4[i] = u4zero();
        const int s = a.src ? __ldg(a.src + j) : a.src_first + j;
        const int b = j / S, jj = j - b * S;
        unsigned *col = a.vall + (size_t)b * a.rows * a.nC * 4 + (jj >> 5);
        const unsigned mine = 1u << (jj & 31);
        const size_t pitch = (size_t)a.nC * 4;
        if (lane == 0) {
            lists[0] = s;
            atomicOr(col + (size_t)s * pitch, mine);
        }
        __syncwarp();
        if (lane == 0) set[s >> 5] = 1u << (s & 31);
        __syncwarp();
        int n = 1;
        for (int L = 1; L <= a.K && n > 0; ++L) {
            const int *list = lists + ((L - 1) & 1) * half;
            int *next = lists + (L & 1) * half;
            const int total = n * D;
            int nn = 0;
            for (int i0 = 0; i0 < total; i0 += 32 * 8) {
                unsigned w[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int i = i0 + 32 * k + (int)lane;
                    w[k] = i < total ? (unsigned)__ldg(a.adj + (size_t)list[i / D] * D + i % D) : 0u;
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (i0 + 32 * k >= total) break;
                    const unsigned bit = 1u << (w[k] & 31u);
                    const bool fresh = i0 + 32 * k + (int)lane < total && (atomicOr(set + (w[k] >> 5), bit) & bit) == 0u;
                    if (fresh) atomicOr(col + w[k] * pitch, mine);
                    const unsigned m = __ballot_sync(0xffffffffu, fresh);
                    const int at = nn + __popc(m & ((1u << lane) - 1u));
                    if (fresh && L < a.K && at < half) next[at] = (int)w[k];   // (never more: D^L at most)
                    nn += __popc(m);
                }
            }
            if (lane == 0) atomicAdd(s_cnt + L, (unsigned)nn);
            n = min(nn, half);
            __syncwarp();
        }
    }
    __syncthreads();
    if (threadIdx.x >= 1u && (int)threadIdx.x <= a.K && s_cnt[threadIdx.x])
        atomicAdd(a.counts + (size_t)((int)(blockIdx.x * (kSrcBallBlock / 32)) / S) * a.stride + threadIdx.x,
                  (unsigned long long)s_cnt[threadIdx.x]);
}

constexpr int kSweepBlock = 1024;   // one block per SM: a grid barrier takes 148 arrivals, not 592

struct SweepArgs {
    const int32_t *adj;
    const int *bad, *oneway;
    const uint4 *vall;        // [nb][rows * nC]: level-K rows (ball_kernel)
    uint4 *A, *B;             // [rows * nC] each: the levels after it in turn
    Ctl *ctl;
    unsigned expected;
    long long wait_ns;
    unsigned long long *counts;   // [nb][stride], levels 1..K from the walk, zeros above
    unsigned long long *vtot;     // [nb][3], zeros
    int stride;
    int *levels_run;              // [nb], zeros
    unsigned long long *batch_ns;
    int *redo;
    int rows, nC, nb, K, max_levels;
    int ns_total, all;        // sources; 1: every vertex, in order (last_rows takes half of the rows)
    int sh;                   // log2 of nC, when that is below 32
    int thin_ppm;             // below this share of the pairs a feeding frontier is thin
    int last_ppm;             // last_rows once fewer of the pairs than this are left
    int adj_smem_rows;
};

// A block's state in shared memory (thread 0 writes it between block barriers), so that
// the functions below keep the kernel's registers to their loops: with these as kernel
// variables a value of sweep_rows' loop was spilled, and its levels took 46 us, not 39.
struct SweepState {
    unsigned long long reached, c_prev, pairs;
    int last;                 // level at which every batch takes last_rows (0: none yet)
    int half;                 // last_rows' H
    const uint4 *X;           // rows the next level reads
    uint4 *Y;                 // and writes
    const int32_t *adj;       // the table, or the block's slice of it in shared memory,
    unsigned v_base;          // which starts at this row
    unsigned t_lo, t_hi;      // the block's tiles of a level
    unsigned next;            // its next tile
    unsigned long long sum;   // its level total
    unsigned epoch;           // grid barriers passed
    int act;                  // next step: 0 level, 1 last_rows, 2 batch done, 3 give up
};

// Row and chunk of a lane in tile t (32 chunks in a row).  Batches of whole 4096-source
// parts (kOnePart: one): a part of one row; narrower ones (kNarrow): 32 / nC rows.  False:
// past the last row.
enum { kOnePart = 0, kParts = 1, kNarrow = 2 };
template <int MODE>
__device__ __forceinline__ bool tile_place(const SweepArgs &a, const unsigned t, const unsigned lane, unsigned &v, unsigned &at) {
    if constexpr (MODE == kOnePart) {
        v = t;
        at = lane;
    } else if constexpr (MODE == kParts) {
        const unsigned parts = (unsigned)a.nC / 32u;
        v = t / parts;
        at = (t - v * parts) * 32u + lane;
    } else {
        const unsigned item = t * 32u + lane;
        v = item >> a.sh;
        at = item & ((1u << a.sh) - 1u);
        if (v >= (unsigned)a.rows) {
            v = (unsigned)a.rows - 1u;
            return false;
        }
    }
    return true;
}

// The block's share [lo, hi) of the tiles of the rows from v0 on, and the rows they lie in.
template <bool WIDE>
__device__ __forceinline__ void tile_share(const SweepArgs &a, const unsigned v0, unsigned &t_lo, unsigned &t_hi, unsigned &r_lo,
                                           unsigned &r_hi) {
    const unsigned step = WIDE ? (unsigned)a.nC / 32u : 1u;                     // tiles that stay together
    const unsigned first = WIDE ? v0 : 0u;
    const unsigned n = WIDE ? (unsigned)a.rows - v0 : ((unsigned)a.rows * (unsigned)a.nC + 31u) / 32u;
    const unsigned lo = first + (unsigned)((unsigned long long)n * blockIdx.x / gridDim.x);
    const unsigned hi = first + (unsigned)((unsigned long long)n * (blockIdx.x + 1) / gridDim.x);
    t_lo = lo * step;
    t_hi = hi * step;
    r_lo = WIDE ? lo : lo * (32u >> a.sh);
    r_hi = WIDE ? hi : min((unsigned)a.rows, hi * (32u >> a.sh));
}

// Adjacency row v of the table, the same in every lane.
template <int D>
__device__ __forceinline__ void sweep_row(const int32_t *adj, const unsigned v, unsigned (&u)[D]) {
    if constexpr (D % 4 == 0) {
        const int4 *p = reinterpret_cast<const int4 *>(adj + (size_t)v * D);
#pragma unroll
        for (int i = 0; i < D / 4; ++i) {
            const int4 x = __ldg(p + i);
            u[4 * i] = (unsigned)x.x; u[4 * i + 1] = (unsigned)x.y;
            u[4 * i + 2] = (unsigned)x.z; u[4 * i + 3] = (unsigned)x.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < D; ++i) u[i] = (unsigned)__ldg(adj + (size_t)v * D + i);
    }
}

// Up to 32 chunks (item = v * nC + place, one a lane) that some of their row's neighbours
// left open: the other neighbours, and for the pairs that level L misses (counted twice
// when the vertex is in a later batch) two steps from V_{L-1}.
template <int D>
static __device__ __noinline__ unsigned finish_chunks(const SweepArgs &a, const SweepState &S, const int b, const int L,
                                                      const unsigned *list, const unsigned n) {
    const uint4 *X = S.X;
    const unsigned lane = threadIdx.x & 31u, nC = (unsigned)a.nC;
    if (lane >= n) return 0u;
    const unsigned item = list[lane], v = item / nC, at = item - v * nC;
    unsigned u[D];
    sweep_row<D>(a.adj, v, u);
    uint4 q = __ldcg(X + (u[0] * nC + at));
#pragma unroll
    for (int i = 1; i < D; ++i) or_into(q, __ldcg(X + (u[i] * nC + at)));
    if (u4full(q)) return 0u;
    const unsigned miss = 128u - u4popc(q);
    for (int i = 0; i < D && !u4full(q); ++i) {
        unsigned w[D];
        sweep_row<D>(a.adj, (unsigned)__ldg(a.adj + (size_t)v * D + i), w);
        uint4 x[D];
#pragma unroll
        for (int j = 0; j < D; ++j) x[j] = __ldcg(X + (w[j] * nC + at));
#pragma unroll
        for (int j = 0; j < D; ++j) or_into(q, x[j]);
    }
    if (!u4full(q)) *a.redo = 1;
    atomicMax(a.levels_run + b, L + 1);
    if (!a.all) return miss;
    const int bv = (int)(v / (128u * nC));
    // (level L + 1 is not empty for either batch of these pairs)
    atomicMax(a.levels_run + bv, L + 1);
    return bv == b ? miss : 2u * miss;
}

// The block's share of the rows from batch b on (its slice of the table to s_row first).
// A tile takes the first H neighbours of its row, such that a chunk is then rarely open;
// those go on a list of the warp's and are finished 32 at a time.  (At
// once, a warp in three waited for a second round of gathers; and in line with the kernel,
// as sweep_rows: as a call the loop's gathers were held back by the registers kept for the
// caller.  All rows of n = 65536, d = 8 on an 8192-source batch: 31 -> 27 us.)
template <int D, int H, bool WIDE>
__device__ __forceinline__ unsigned last_rows(const SweepArgs &a, SweepState &S, const int b, const int L,
                                              int32_t *s_row, unsigned *list) {
    constexpr int U = H <= 4 ? 8 / H : 1;   // tiles a round: up to 8 gathers in flight
    const uint4 *X = S.X;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned nC = (unsigned)a.nC;
    unsigned t_lo, t_end, r_lo, r_hi;
    tile_share<WIDE>(a, a.all ? (unsigned)b * 128u * nC : 0u, t_lo, t_end, r_lo, r_hi);
    const bool keep = r_hi <= r_lo + (unsigned)a.adj_smem_rows;
    if (keep)
        for (unsigned k = threadIdx.x; r_lo < r_hi && k < (r_hi - r_lo) * D; k += blockDim.x) s_row[k] = __ldg(a.adj + (size_t)r_lo * D + k);
    const int32_t *adj = keep ? s_row : a.adj;
    const unsigned v_base = keep ? r_lo : 0u;
    if (threadIdx.x == 0) S.next = t_lo;
    __syncthreads();
    unsigned cnt = 0u, open = 0u;
    for (;;) {
        unsigned t0 = 0u;
        if (lane == 0) t0 = atomicAdd(&S.next, (unsigned)U);
        t0 = __shfl_sync(0xffffffffu, t0, 0);
        if (t0 >= t_end) break;
        uint4 x[U][H];
        bool in[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            unsigned v, at;
            in[k] = tile_place<WIDE ? kParts : kNarrow>(a, min(t0 + (unsigned)k, t_end - 1u), lane, v, at);
            const int32_t *row = adj + (size_t)(v - v_base) * D;
#pragma unroll
            for (int i = 0; i < H; ++i) x[k][i] = __ldcg(X + ((unsigned)row[i] * nC + at));
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            uint4 q = x[k][0];
#pragma unroll
            for (int i = 1; i < H; ++i) or_into(q, x[k][i]);
            const bool o = t0 + (unsigned)k < t_end && in[k] && !u4full(q);
            const unsigned m = __ballot_sync(0xffffffffu, o);
            if (m == 0u) continue;
            if (o) list[open + __popc(m & ((1u << lane) - 1u))] = (t0 + (unsigned)k) * 32u + lane;
            open += __popc(m);
            __syncwarp();
            if (open >= 32u) {
                open -= 32u;
                cnt += finish_chunks<D>(a, S, b, L, list + open, 32u);
                __syncwarp();
            }
        }
    }
    cnt += finish_chunks<D>(a, S, b, L, list, open);
    return cnt;
}

// Neighbours a tile of last_rows takes, with a share u of the pairs left: a chunk of 128
// stays open with 128 u^H, and costs D gathers of a 32-byte sector each when it does.
__device__ __forceinline__ int last_half(const int D, const float u) {
    const int hs[5] = {2, 3, 4, 6, 8};
    float p = u;
    int k = 1;
    for (int i = 0; i < 5; ++i) {
        if (hs[i] >= D) break;
        for (; k < hs[i]; ++k) p *= u;
        if (128.f * p < 0.03f) return hs[i];
    }
    return D <= 8 ? D : 8;
}

template <int D, bool WIDE>
__device__ __forceinline__ unsigned last_rows_of(const SweepArgs &a, SweepState &S, const int b, const int L,
                                                 int32_t *s_row, unsigned *list) {
    const int H = S.half;
    if (H == 2) return last_rows<D, 2, WIDE>(a, S, b, L, s_row, list);
    if constexpr (D >= 3) if (H == 3) return last_rows<D, 3, WIDE>(a, S, b, L, s_row, list);
    if constexpr (D >= 4) if (H == 4) return last_rows<D, 4, WIDE>(a, S, b, L, s_row, list);
    if constexpr (D >= 6) if (H == 6) return last_rows<D, 6, WIDE>(a, S, b, L, s_row, list);
    return last_rows<D, (D < 8 ? D : 8), WIDE>(a, S, b, L, s_row, list);
}

// One dense level on the block's tiles [next, t_hi): Y[v] = OR of the neighbours' X
// rows (without one-way entries V_{L-1}[v] lies within them for L >= 2), and this
// thread's popcount of what it wrote.
template <int D, int MODE>
__device__ __forceinline__ unsigned sweep_rows(const SweepArgs &a, SweepState &S) {
    const unsigned lane = threadIdx.x & 31u;
    const uint4 *X = S.X;
    uint4 *Y = S.Y;
    const int32_t *adj = S.adj;
    const unsigned v_base = S.v_base, t_hi = S.t_hi;
    unsigned cnt = 0u;
    for (;;) {
        unsigned t = 0u;
        if (lane == 0) t = atomicAdd(&S.next, 1u);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= t_hi) break;
        unsigned v, at;
        const bool in = tile_place<MODE>(a, t, lane, v, at);
        const unsigned w = MODE == kOnePart ? 32u : (unsigned)a.nC;
        const int32_t *row = adj + (size_t)(v - v_base) * D;
        unsigned tu[D];
#pragma unroll
        for (int i = 0; i < D; ++i) tu[i] = (unsigned)row[i] * w + at;
        uint4 x[D];
#pragma unroll
        for (int i = 0; i < D; ++i) x[i] = __ldcg(X + tu[i]);
        uint4 q = x[0];
#pragma unroll
        for (int i = 1; i < D; ++i) or_into(q, x[i]);
        if (in) {
            Y[(size_t)t * 32 + lane] = q;
            cnt += u4popc(q);
        }
    }
    return cnt;
}

// What comes next in batch b, whose levels below L are done (thread 0).
template <int D>
__device__ __forceinline__ void sweep_next(const SweepArgs &a, SweepState &S, const int b, const int L) {
    const unsigned long long left = S.pairs - S.reached;
    if (left == 0ull) {
        if (blockIdx.x == 0) atomicMax(a.levels_run + b, L - 1);
        S.act = 2;
        return;
    }
    if ((b == 0 || !a.all) && S.last == 0 && L >= 2 && left * 1000000ull < S.pairs * (unsigned long long)a.last_ppm) S.last = L;
    if (L == S.last) {
        S.act = L + 1 <= a.max_levels ? 1 : 3;
        S.half = last_half(D, (float)left / (float)S.pairs);
    } else {
        const bool thin = S.c_prev == 0ull || S.c_prev * 1000000ull < S.pairs * (unsigned long long)a.thin_ppm;
        S.act = thin || L > a.max_levels ? 3 : 0;
    }
}

template <int D, bool WIDE>
__global__ void __launch_bounds__(kSweepBlock, 1) sweep_kernel(const __grid_constant__ SweepArgs a) {
    extern __shared__ int32_t s_adj[];
    __shared__ unsigned s_open[kSweepBlock / 32][64];   // last_rows' lists (one array for all its instances)
    __shared__ SweepState S;
    if (a.bad && *a.bad) return;   // uniform across the grid, as is the next
    if (ld_acquire_i(a.oneway) != 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *a.redo = 1;
        return;
    }
    {
        unsigned t_lo, t_hi, v_lo, v_hi;
        tile_share<WIDE>(a, 0u, t_lo, t_hi, v_lo, v_hi);
        const bool keep = v_hi <= v_lo + (unsigned)a.adj_smem_rows;   // the block's slice of the table
        if (keep)
            for (unsigned k = threadIdx.x; v_lo < v_hi && k < (v_hi - v_lo) * D; k += blockDim.x) s_adj[k] = __ldg(a.adj + (size_t)v_lo * D + k);
        if (threadIdx.x == 0) {
            S.adj = keep ? s_adj : a.adj;
            S.v_base = keep ? v_lo : 0u;
            S.t_lo = t_lo;
            S.t_hi = t_hi;
            S.last = 0;
            S.epoch = 0u;
            S.Y = a.A;
        }
    }
    for (int b = 0; b < a.nb; ++b) {
        int L = a.K + 1;
        if (threadIdx.x == 0) {
            const int ns = min(128 * a.nC, a.ns_total - b * 128 * a.nC);
            unsigned long long *counts = a.counts + (size_t)b * (size_t)a.stride;
            if (blockIdx.x == 0) {
                a.batch_ns[2 * b] = gtimer();
                counts[0] = (unsigned long long)ns;
            }
            S.pairs = (unsigned long long)ns * (unsigned long long)a.rows;
            S.reached = (unsigned long long)ns;
            S.c_prev = 0ull;
            if (!a.all) S.last = 0;
            S.X = a.vall + (size_t)b * ((size_t)a.rows * (size_t)a.nC);
            int k = 1;
            for (; k <= a.K && S.reached < S.pairs; ++k) {
                S.c_prev = ld_relaxed_u64(counts + k);
                S.reached += S.c_prev;
            }
            sweep_next<D>(a, S, b, S.reached == S.pairs ? k : L);
            S.next = S.t_lo;
            S.sum = 0ull;
        }
        __syncthreads();
        for (; S.act == 0; ++L) {
            const unsigned cnt = !WIDE ? sweep_rows<D, kNarrow>(a, S) : a.nC == 32 ? sweep_rows<D, kOnePart>(a, S) : sweep_rows<D, kParts>(a, S);
            const unsigned wsum = __reduce_add_sync(0xffffffffu, cnt);
            if ((threadIdx.x & 31u) == 0u) atomicAdd(&S.sum, (unsigned long long)wsum);
            __syncthreads();
            unsigned long long *vt = a.vtot + 3 * (size_t)b;
            if (threadIdx.x == 0) {
                atomicAdd(vt + L % 3, S.sum);
                if (blockIdx.x == 0) vt[(L + 1) % 3] = 0ull;   // read last after level L - 2
            }
            unsigned long long total = 0ull;
            unsigned epoch = S.epoch;
            if (!grid_sync_value(a.ctl, a.expected, a.wait_ns, L, epoch, vt + L % 3, total)) return;
            if (threadIdx.x == 0) {
                // total bits of V_L less the padding and the pairs reached before
                const int ns = min(128 * a.nC, a.ns_total - b * 128 * a.nC);
                const unsigned long long pad = (unsigned long long)a.rows * (unsigned long long)(128 * a.nC - ns);
                const unsigned long long cL = total - pad - S.reached;
                if (blockIdx.x == 0) a.counts[(size_t)b * (size_t)a.stride + L] = cL;
                S.reached += cL;
                S.c_prev = cL;
                S.epoch = epoch;
                S.X = S.Y;
                S.Y = S.Y == a.A ? a.B : a.A;
                S.next = S.t_lo;
                S.sum = 0ull;
                sweep_next<D>(a, S, b, L + 1);
            }
            __syncthreads();
        }
        if (S.act == 3) {
            if (blockIdx.x == 0 && threadIdx.x == 0) *a.redo = 1;
            return;
        }
        if (S.act == 1) {
            // No barrier before the next batch: its first level writes the other buffer,
            // and the second one only after the barrier between them.
            unsigned long long *counts = a.counts + (size_t)b * (size_t)a.stride + L;
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                atomicMax(a.levels_run + b, L);
                atomicAdd(counts, S.pairs - S.reached);
            }
            const unsigned cnt = last_rows_of<D, WIDE>(a, S, b, L, s_adj + (size_t)a.adj_smem_rows * D, s_open[threadIdx.x >> 5]);
            const unsigned m = __reduce_add_sync(0xffffffffu, cnt);
            if ((threadIdx.x & 31u) == 0u && m) {
                atomicAdd(counts, 0ull - (unsigned long long)m);
                atomicAdd(counts + 1, (unsigned long long)m);
            }
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) a.batch_ns[2 * b + 1] = gtimer();
        __syncthreads();   // S is rewritten for the next batch
    }
}

}  // namespace gg
