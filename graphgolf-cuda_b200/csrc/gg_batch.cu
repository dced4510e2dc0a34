// gg_batch.cu -- batched exact evaluation of 2-opt candidates (gg_batch_* in gg.h).
//
// One persistent launch scores every candidate of a batch.  Work unit ("task") =
// one candidate x one chunk of its sources.  A CTA takes a task, builds the
// candidate's adjacency in shared memory (the base rows as uint16, then the four
// rows the 2-opt edit touches), and runs the whole BFS of the chunk's sources
// with both visited bitsets resident in shared memory:
//     next[v][c] = cur[v][c] | (OR_{u in adj[v]} cur[u][c])        (all rows, one level)
// i.e. the level step of cudaASPLconv.cu:35-56 with the reduction of :59-99
// folded into per-thread popcounts, a shared sum and one block barrier per level.  The grid
// barrier of the single-graph path is not needed: a task never leaves its CTA.
//
// Near sources (default): per base, one pass of the single-graph engine also writes the
// base's distance matrix as 4 bit-planes, from which every source's distance sum and
// eccentricity follow.  A candidate then searches only from the set T of sources that
//   * its 2-opt can affect (the test of gg_inc.cu: a removed edge between consecutive
//     BFS levels whose deeper end has no other parent, or an added edge between vertices
//     whose distances differ by 2 or more), and that
//   * lie within floor((diameter - 1) / 2) of one of its four endpoints.
// A pair whose distance changes has a shortest path, old or new, no longer than the old
// diameter through a changed edge, so one of the two lies that near to an endpoint of it
// (in the base graph) -- and both are affected.  The distance matrices are symmetric, so
// with w = 1 for v in T and 2 for the others
//   new total = old total + sum over s in T, every v, of w(v) (new - old distance),
// and every changed pair is seen.  T is 116 of 1024 sources (d = 6), 442 of 3000 (d = 4),
// 221 of 4096 (d = 8) on average, against 406, 1859 and 1116 affected ones.
// The diameter is the larger of the largest new distance from T and the largest old
// distance between vertices outside T.  Bases that are not symmetric, not connected or of
// diameter above 15, small bases and populations (kIncMinN, worth_near), candidates whose
// removed edges the base does not hold (or not equally often at both ends) and the histogram
// pass search every source.  GG_BATCH_FULL=1 makes every candidate do so, 0 none of the
// small ones.
//
// batch_select finds each candidate's sources and cuts them into work units; the units
// come off one counter, and the candidate and base counts are read from device memory, so
// one captured CUDA graph serves every batch size up to the capacity it was captured for.
#include "gg.h"
#include "gg_internal.h"
#include "gg_planes.cuh"

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_runtime.h>


namespace {

constexpr int kBatchBlock = 1024;
constexpr size_t kSmemBudget = 220 * 1024;
constexpr size_t kSmemMost = kSmemBudget + 4 * 1024;   // with T's bits

constexpr int kPlanes = 4;   // distance bit-planes: distances up to 15

struct BatchBase {
    const int32_t *adj;   // [n][d] in global memory
    const uint16_t *adj16;   // the same rows as uint16, padded to adj16_bytes (a multiple of 16)
    unsigned adj16_bytes;
    int n, d;
    int log_nc;           // chunks (of 128 sources) per task row = 1 << log_nc
    int chunks;           // tasks per candidate = ceil(n / (128 << log_nc))
    // near-source mode (valid != 0)
    const uint4 *planes;  // [kPlanes][n][cols]: bit k of dist(source, vertex)
    unsigned cols;        // plane columns of 128 sources
    const unsigned *rowsum;  // [n]: distance sum of each source
    const unsigned *ecc;     // [n]: eccentricity of each source
    const unsigned *top;     // [n]: vertices at distance `levels` from each source
    unsigned long long total, reached;  // the base's own counts
    unsigned long long at_top;          // ordered pairs at distance `levels`
    int levels;
    int radius;           // floor((levels - 1) / 2)
    int valid;            // symmetric, connected, diameter <= 15
    int few_near;         // near sources even where a population's full searches fill no wave of blocks
};

// How a candidate is scored.
enum { kNear = 0, kFull = 1, kBase = 2 };

// A candidate's state between the launches of one evaluation.
struct CandState {
    unsigned long long old_sum;   // base distance sums of T
    unsigned long long tt_sum;    // base distances within T
    unsigned count;               // |T|
    unsigned tops;                // pairs (T, any) at distance `levels` of the base
    unsigned groups_done;         // blocks of batch_select that finished the candidate
    int mode;
};

// A work unit: `ns` sources of a candidate from `first` on (entries of its list, or
// vertices for a full search), rows of 1 << log_nc chunks.
struct Unit {
    int cand;
    int first;
    int ns;
    int log_nc;
};

struct BatchCtl {
    unsigned unit_ctr;    // work units taken
    int n_cand;
    int n_units;          // work units
    int bad;              // set by batch_reset when a candidate is outside the domain
    int n_bases;          // registered bases
    int bad_index;        // lowest index of such a candidate (INT_MAX: none)
    int timeout;          // a CTA's wait for its adjacency copy ran past its limit
    int pad;
};

struct BatchArgs {
    const BatchBase *bases;
    const gg_swap *cands;
    gg_cand_result *out;
    BatchCtl *ctl;
    unsigned *hist;       // nullptr, or [n][hist_k]: per-vertex new pairs at levels 1..hist_k
    int hist_k;           // (only meaningful for a launch of one candidate)
    CandState *cs;        // [cand]
    uint16_t *lists;      // [cand][list_stride]: the sources of T
    int list_stride;
    uint32_t *tbits;      // [cand][tbits_stride]: bit v: v in T
    int tbits_stride;
    Unit *units;
    int force_full;       // every candidate searches every source
    int wave;             // blocks of batch_kernel that run at once
};

__device__ __forceinline__ uint4 z4() { return make_uint4(0u, 0u, 0u, 0u); }
__device__ __forceinline__ unsigned padw(int lo, int ns) {
    if (ns <= lo) return 0xffffffffu;
    if (ns >= lo + 32) return 0u;
    return ~((1u << (ns - lo)) - 1u);
}

// Bulk copy (the TMA unit's untiled cp.async.bulk, no multicast, this GPU's
// memory) of `bytes` (a multiple of 16, both addresses 16-byte aligned) from global
// memory into this CTA's shared memory, completing on the mbarrier `bar`.
__device__ __forceinline__ unsigned smem_addr(const void *p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void bulk_to_smem(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 :: "r"(smem_addr(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned phase) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 " selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(smem_addr(bar)), "r"(phase) : "memory");
    return ok != 0;
}

constexpr long long kCopyWaitNs = 2000000000ll;   // 2 s: a copy of at most 128 KB never takes that

// The four pull entries a 2-opt replaces: row r[i] lists t[i] in place of f[i].
struct SwapRows {
    int r[4], f[4], t[4];
    __device__ __forceinline__ explicit SwapRows(const gg_swap &s) {
        r[0] = s.a; r[1] = s.b; r[2] = s.c; r[3] = s.d;
        f[0] = s.b; f[1] = s.a; f[2] = s.d; f[3] = s.c;
        t[0] = s.mode ? s.d : s.c; t[1] = s.mode ? s.c : s.d;
        t[2] = s.mode ? s.b : s.a; t[3] = s.mode ? s.a : s.b;
    }
};

// The d neighbour ids of a row in shared memory, in the widest loads its alignment
// allows (rows start at multiples of 2 d bytes).
template <int D>
__device__ __forceinline__ void row_ids(const uint16_t *ar, unsigned (&id)[D]) {
    if constexpr (D % 8 == 0) {
#pragma unroll
        for (int k = 0; k < D / 8; ++k) {
            const uint4 q = reinterpret_cast<const uint4 *>(ar)[k];
            id[8 * k] = q.x & 0xffffu; id[8 * k + 1] = q.x >> 16;
            id[8 * k + 2] = q.y & 0xffffu; id[8 * k + 3] = q.y >> 16;
            id[8 * k + 4] = q.z & 0xffffu; id[8 * k + 5] = q.z >> 16;
            id[8 * k + 6] = q.w & 0xffffu; id[8 * k + 7] = q.w >> 16;
        }
    } else if constexpr (D % 4 == 0) {
#pragma unroll
        for (int k = 0; k < D / 4; ++k) {
            const uint2 q = reinterpret_cast<const uint2 *>(ar)[k];
            id[4 * k] = q.x & 0xffffu; id[4 * k + 1] = q.x >> 16;
            id[4 * k + 2] = q.y & 0xffffu; id[4 * k + 3] = q.y >> 16;
        }
    } else if constexpr (D % 2 == 0) {
#pragma unroll
        for (int k = 0; k < D / 2; ++k) {
            const unsigned q = reinterpret_cast<const unsigned *>(ar)[k];
            id[2 * k] = q & 0xffffu; id[2 * k + 1] = q >> 16;
        }
    } else {
#pragma unroll
        for (int k = 0; k < D; ++k) id[k] = ar[k];
    }
}

// One level of a unit: nxt = cur | OR of the neighbours' cur, every row.  Bound by the
// shared-memory gathers: random 16-byte rows put 8 lanes on 2.6 of 8 bank groups.  cnt: new pairs
// of the thread, wcnt: the same weighted (1 where bit v of tb is set, else 2).
// D > 0: the degree at compile time, a row's gathers all in flight together.
template <int D>
static __device__ __forceinline__ void level_pass(const uint4 *cur, uint4 *nxt, const uint16_t *adj, const int d,
                                               const int items, const int lnc, const uint32_t *tb, unsigned *hist,
                                               const int hist_k, const int L, unsigned &cnt_out, unsigned &wcnt_out) {
    const int nC = 1 << lnc;
    unsigned cnt = 0u, wcnt = 0u;
    for (int t = threadIdx.x; t < items; t += kBatchBlock) {
        const int v = t >> lnc, c = t & (nC - 1);
        const uint4 own = cur[t];
        uint4 out = own;
        if ((own.x & own.y & own.z & own.w) != 0xffffffffu) {
            uint4 acc = z4();
            const uint16_t *ar = adj + v * d;
            if constexpr (D > 0) {
                unsigned id[D];
                row_ids<D>(ar, id);
#pragma unroll
                for (int i = 0; i < D; ++i) {
                    const uint4 x = cur[(id[i] << lnc) + c];
                    acc.x |= x.x; acc.y |= x.y; acc.z |= x.z; acc.w |= x.w;
                }
            } else {
                for (int i = 0; i < d; ++i) {
                    const uint4 x = cur[((int)ar[i] << lnc) + c];
                    acc.x |= x.x; acc.y |= x.y; acc.z |= x.z; acc.w |= x.w;
                }
            }
            out = make_uint4(own.x | acc.x, own.y | acc.y, own.z | acc.z, own.w | acc.w);
            const unsigned pc = __popc(acc.x & ~own.x) + __popc(acc.y & ~own.y) + __popc(acc.z & ~own.z) +
                                __popc(acc.w & ~own.w);
            cnt += pc;
            wcnt += pc << (((tb[v >> 5] >> (v & 31)) & 1u) ^ 1u);
            if (hist && L <= hist_k && pc) atomicAdd(hist + (size_t)v * hist_k + (L - 1), pc);
        }
        nxt[t] = out;
    }
    cnt_out = cnt;
    wcnt_out = wcnt;
}

// The first levels of a unit of few sources from the other side: source j's walk ends of
// length L (d^L of them) get bit j, the ones not set before are its new pairs.  A pass
// reads d + 2 rows of 16 bytes per vertex whatever is new; a walk end costs one atomic and
// L dependent id loads, so the walk takes the levels with at most kWalkItems ends a row.
// Walks leave a source along the table's rows, so their ends are the vertices that reach it
// only in a graph without one-way entries: a near-source candidate is one (batch_select), a
// full search need not be.
//
// batch_kernel and its three small launches, 2048 x (n=1024, d=6) + 512 x (n=3000, d=4)
// candidates: 2243 us a call with every affected source searched (2020 us of it here), 720
// (632) with T; 32 x (n=4096, d=8): 215 (162) and 90 us (45).
constexpr int kWalkItems = 2;   // walk ends of all sources, at most this many times the rows

__global__ void __launch_bounds__(kBatchBlock, 1) batch_kernel(const BatchArgs a) {
    extern __shared__ uint4 sm[];
    __shared__ unsigned s_unit;
    __shared__ unsigned long long s_tot[kBatchBlock / 32], s_reach[kBatchBlock / 32];
    __shared__ unsigned s_cnt[3];
    __shared__ __align__(8) uint64_t s_bar;   // completion of the adjacency copy
    __shared__ int s_late;
    if (a.ctl->bad) return;   // batch_reset rejected a candidate: index nothing
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned n_units = (unsigned)a.ctl->n_units;
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(&s_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    unsigned phase = 0;

    for (;;) {
        if (tid == 0) s_unit = atomicAdd(&a.ctl->unit_ctr, 1u);
        __syncthreads();
        const unsigned u = s_unit;
        if (u >= n_units) return;
        const Unit un = a.units[u];
        const int cand = un.cand, lnc = un.log_nc, ns = un.ns;
        const gg_swap sw = a.cands[cand];
        const BatchBase &B = a.bases[sw.base];
        const int n = B.n, d = B.d, nC = 1 << lnc;
        const bool full = a.cs[cand].mode != kNear;
        const int items = n << lnc, twords = (n + 31) / 32;
        const uint16_t *lst = a.lists + (size_t)cand * a.list_stride + un.first;   // (not full)

        // shared memory: adjacency (uint16, padded to 16 bytes), T's bits (padded too),
        // then two bitsets.  The base's packed rows arrive by one bulk copy; every thread
        // waits on the mbarrier (bounded: past kCopyWaitNs the CTA flags a timeout and stops).
        uint16_t *adj = reinterpret_cast<uint16_t *>(sm);
        uint32_t *tb = reinterpret_cast<uint32_t *>(sm + ((size_t)n * d * 2 + 15) / 16);
        uint4 *cur = reinterpret_cast<uint4 *>(tb) + (twords + 3) / 4;
        uint4 *nxt = cur + items;
        if (tid == 0) {
            // the previous unit's generic-proxy accesses to this memory come first
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            bulk_to_smem(adj, B.adj16, B.adj16_bytes, &s_bar);
            s_late = 0;
        }
        if (tid < 3) s_cnt[tid] = 0u;
        for (int k = tid; k < twords; k += kBatchBlock)
            tb[k] = full ? 0xffffffffu : __ldcg(a.tbits + (size_t)cand * a.tbits_stride + k);
        // visited after level 0: the padding sources and (below) the diagonal
        for (int t = tid; t < items; t += kBatchBlock) {
            const int b = (t & (nC - 1)) * 128;
            cur[t] = make_uint4(padw(b, ns), padw(b + 32, ns), padw(b + 64, ns), padw(b + 96, ns));
        }
        if (!full) {
            // base distances within T, from these sources' plane rows (their loads and the
            // adjacency copy are in flight together)
            const uint32_t *pw = reinterpret_cast<const uint32_t *>(B.planes);
            const size_t ps = (size_t)n * B.cols * 4, cw = (size_t)B.cols * 4;
            const uint32_t *tg = a.tbits + (size_t)cand * a.tbits_stride;
            unsigned sum = 0u;
            for (int j = warp; j < ns; j += kBatchBlock / 32) {
                const size_t row = (size_t)__ldcg(lst + j) * cw;
#pragma unroll 4
                for (int k = lane; k < twords; k += 32)
                    sum += dist4_sum(dist4_load(pw, ps, row + k), __ldcg(tg + k));
            }
            sum = __reduce_add_sync(0xffffffffu, sum);
            if (lane == 0 && sum) atomicAdd(&a.cs[cand].tt_sum, (unsigned long long)sum);
        }
        {
            bool done = mbar_try_wait(&s_bar, phase);
            if (!done) {
                unsigned long long t0;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
                for (unsigned it = 1; !done; ++it) {
                    done = mbar_try_wait(&s_bar, phase);
                    if (!done && (it & 63u) == 0u) {
                        unsigned long long t;
                        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                        if ((long long)(t - t0) > kCopyWaitNs) break;
                    }
                }
            }
            if (!done) s_late = 1;
        }
        phase ^= 1u;
        __syncthreads();
        if (s_late) {
            // the copy did not complete: report it and leave (the host sees
            // GG_TIMEOUT); only this CTA's tail of units is left unscored
            if (tid == 0) atomicExch(&a.ctl->timeout, 1);
            return;
        }
        if (sw.a >= 0 && tid < 4) {
            // 2-opt: (a,b),(c,d) -> (a,c),(b,d) [mode 0] or (a,d),(b,c) [mode 1]
            const SwapRows sr(sw);
            const int row = tid == 0 ? sr.r[0] : tid == 1 ? sr.r[1] : tid == 2 ? sr.r[2] : sr.r[3];
            const int f = tid == 0 ? sr.f[0] : tid == 1 ? sr.f[1] : tid == 2 ? sr.f[2] : sr.f[3];
            const int t = tid == 0 ? sr.t[0] : tid == 1 ? sr.t[1] : tid == 2 ? sr.t[2] : sr.t[3];
            for (int j = 0; j < d; ++j)
                if (adj[row * d + j] == (uint16_t)f) { adj[row * d + j] = (uint16_t)t; break; }
        }
        // source j of the unit: vertex un.first + j, or entry j of the list
        auto set_bit = [&](const int v, const int j) -> bool {
            const unsigned bit = 1u << (j & 31);
            return !(atomicOr(reinterpret_cast<unsigned *>(cur + ((v << lnc) + (j >> 7))) + ((j >> 5) & 3), bit) & bit);
        };
        for (int j = tid; j < ns; j += kBatchBlock) set_bit(full ? un.first + j : (int)__ldcg(lst + j), j);
        __syncthreads();

        unsigned long long tot = 0, reach = 0;   // weighted, this thread's
        const unsigned all = (unsigned)ns * (unsigned)n;
        unsigned seen = (unsigned)ns;            // pairs reached, the same in every thread
        int L = 1, last = 0;
        bool done = seen == all;
        // walk ends: levels 1, 2, .. while they are few (a pass visits every row)
        if (!full) {
            for (unsigned ends = (unsigned)d; !done; ends *= (unsigned)d, ++L) {
                if ((unsigned long long)ends * (unsigned)ns > (unsigned long long)kWalkItems * (unsigned)n) break;
                // a thread takes a walk of L - 1 steps and its d ends (the ids of one row)
                unsigned cnt = 0u, wcnt = 0u;
                const unsigned pre = ends / (unsigned)d;
                for (unsigned k = (unsigned)tid; k < pre * (unsigned)ns; k += kBatchBlock) {
                    const int j = (int)(k / pre);
                    unsigned w = k - (unsigned)j * pre;
                    int v = full ? un.first + j : (int)__ldcg(lst + j);
                    for (int l = 1; l < L; ++l) {
                        const unsigned q = w / (unsigned)d;
                        v = adj[v * d + (int)(w - q * (unsigned)d)];
                        w = q;
                    }
                    for (int i = 0; i < d; ++i) {
                        const int e = adj[v * d + i];
                        if (set_bit(e, j)) {
                            cnt += 1u;
                            wcnt += 2u - ((tb[e >> 5] >> (e & 31)) & 1u);
                        }
                    }
                }
                tot += (unsigned long long)L * wcnt;
                reach += wcnt;
                const unsigned wsum = __reduce_add_sync(0xffffffffu, cnt);
                if (lane == 0 && wsum) atomicAdd(&s_cnt[L % 3], wsum);
                __syncthreads();
                const unsigned c = s_cnt[L % 3];
                if (tid == 0) s_cnt[(L + 2) % 3] = 0u;
                seen += c;
                if (c) last = L;
                done = c == 0u || seen == all;
            }
        }
        for (; !done; ++L) {
            unsigned cnt = 0u, wcnt = 0u;
            switch (d) {
                case 3: level_pass<3>(cur, nxt, adj, d, items, lnc, tb, a.hist, a.hist_k, L, cnt, wcnt); break;
                case 4: level_pass<4>(cur, nxt, adj, d, items, lnc, tb, a.hist, a.hist_k, L, cnt, wcnt); break;
                case 5: level_pass<5>(cur, nxt, adj, d, items, lnc, tb, a.hist, a.hist_k, L, cnt, wcnt); break;
                case 6: level_pass<6>(cur, nxt, adj, d, items, lnc, tb, a.hist, a.hist_k, L, cnt, wcnt); break;
                case 7: level_pass<7>(cur, nxt, adj, d, items, lnc, tb, a.hist, a.hist_k, L, cnt, wcnt); break;
                case 8: level_pass<8>(cur, nxt, adj, d, items, lnc, tb, a.hist, a.hist_k, L, cnt, wcnt); break;
                default: level_pass<0>(cur, nxt, adj, d, items, lnc, tb, a.hist, a.hist_k, L, cnt, wcnt); break;
            }
            tot += (unsigned long long)L * wcnt;
            reach += wcnt;
            const unsigned wsum = __reduce_add_sync(0xffffffffu, cnt);
            if (lane == 0 && wsum) atomicAdd(&s_cnt[L % 3], wsum);
            __syncthreads();
            const unsigned c = s_cnt[L % 3];
            if (tid == 0) s_cnt[(L + 2) % 3] = 0u;
            seen += c;
            if (c) last = L;
            done = c == 0u || seen == all;
            uint4 *sw2 = cur; cur = nxt; nxt = sw2;
        }
        unsigned long long wt = tot, wr = reach;
        for (int o = 16; o; o >>= 1) {
            wt += __shfl_down_sync(0xffffffffu, wt, o);
            wr += __shfl_down_sync(0xffffffffu, wr, o);
        }
        if (lane == 0) { s_tot[warp] = wt; s_reach[warp] = wr; }
        __syncthreads();
        if (tid == 0) {
            unsigned long long bt = 0, br = (unsigned long long)ns;
            for (int w = 0; w < kBatchBlock / 32; ++w) { bt += s_tot[w]; br += s_reach[w]; }
            atomicAdd(reinterpret_cast<unsigned long long *>(&a.out[cand].total), bt);
            atomicAdd(reinterpret_cast<unsigned long long *>(&a.out[cand].reached), br);
            atomicMax(&a.out[cand].levels, last);
        }
        __syncthreads();  // the next unit overwrites shared memory
    }
}

// One warp per candidate: the result from the searched sources' counts.
__global__ void __launch_bounds__(128) batch_finalize(const BatchArgs a) {
    const int n_cand = a.ctl->n_cand;
    const int lane = threadIdx.x & 31;
    const int w0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), nw = (int)((gridDim.x * blockDim.x) >> 5);
    const bool dead = a.ctl->bad || a.ctl->timeout;
    for (int i = w0; i < n_cand; i += nw) {
        if (dead) {
            // a rejected or timed-out launch scores nothing: every result says so
            if (lane == 0) a.out[i] = gg_cand_result{0ull, 0ull, -1, 0};
            continue;
        }
        const BatchBase &B = a.bases[a.cands[i].base];
        const CandState cs = a.cs[i];
        gg_cand_result r = a.out[i];
        const unsigned long long nn = (unsigned long long)B.n * (unsigned long long)B.n;
        if (cs.mode != kFull) {
            const unsigned long long T = cs.count;
            r.total = B.total - (2ull * cs.old_sum - cs.tt_sum) + r.total;
            r.reached = B.reached - (2ull * T * B.n - T * T) + r.reached;
            // The largest distance between vertices outside T stays the base's diameter when
            // the pairs that T touches cannot be all there are at it.  Otherwise look for it:
            // from the diameter down, a source outside T with another such vertex there.
            int top = B.levels;
            if (B.at_top <= 2ull * cs.tops) {
                const uint32_t *tb = a.tbits + (size_t)i * a.tbits_stride;
                const uint32_t *pw = reinterpret_cast<const uint32_t *>(B.planes);
                const size_t ps = (size_t)B.n * B.cols * 4, cw = (size_t)B.cols * 4;
                const int words = (B.n + 31) / 32;
                for (bool found = false; top > r.levels; --top) {
                    for (int s0 = 0; s0 < B.n && !found; s0 += 32) {
                        const int s = s0 + lane;
                        const bool in = s < B.n && !((__ldcg(tb + (s0 >> 5)) >> lane) & 1u) && (int)__ldg(B.ecc + s) >= top;
                        for (unsigned m = __ballot_sync(0xffffffffu, in); m && !found; m &= m - 1u) {
                            const int v = s0 + __ffs((int)m) - 1;
                            bool hit = false;
                            for (int k = lane; k < words; k += 32) {
                                uint32_t live = ~__ldcg(tb + k);
                                if (k == words - 1 && (B.n & 31)) live &= (1u << (B.n & 31)) - 1u;
                                hit |= (dist4_eq(dist4_load(pw, ps, (size_t)v * cw + k), dist4_const((unsigned)top)) & live) != 0u;
                            }
                            found = __any_sync(0xffffffffu, hit);
                        }
                    }
                    if (found) break;
                }
            }
            r.levels = max(r.levels, top);
        }
        r.connected = r.reached == nn;
        if (lane == 0) a.out[i] = r;
    }
}

// Zeroes the results and range-checks every candidate (the device-array entry
// point gets candidates the host never saw): base registered, endpoints inside the
// base, distinct, mode 0 or 1.  One bad candidate sets ctl->bad, and the kernels
// after this one return before reading a base or a row through it.
// With force_full it makes the work units, too (a histogram pass is 3 to 8 us longer with a
// launch of batch_select for them).
__global__ void batch_reset(const BatchArgs a) {
    const int n_cand = a.ctl->n_cand;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_cand; i += gridDim.x * blockDim.x) {
        a.out[i] = gg_cand_result{0ull, 0ull, 0, 0};
        a.cs[i] = CandState{0ull, 0ull, 0u, 0u, 0u, kNear};
        const gg_swap sw = a.cands[i];
        bool ok = sw.base >= 0 && sw.base < a.ctl->n_bases;
        if (ok && sw.a >= 0) {
            const unsigned n = (unsigned)a.bases[sw.base].n;
            ok = (unsigned)sw.a < n && (unsigned)sw.b < n && (unsigned)sw.c < n && (unsigned)sw.d < n &&
                 (sw.mode == 0 || sw.mode == 1) && sw.a != sw.b && sw.a != sw.c && sw.a != sw.d &&
                 sw.b != sw.c && sw.b != sw.d && sw.c != sw.d;
        }
        if (!ok) {
            atomicExch(&a.ctl->bad, 1);
            atomicMin(&a.ctl->bad_index, i);
        } else if (a.force_full) {
            const BatchBase &B = a.bases[sw.base];
            const int S = 128 << B.log_nc, u0 = atomicAdd(&a.ctl->n_units, B.chunks);
            a.cs[i].mode = kFull;
            for (int k = 0; k < B.chunks; ++k) a.units[u0 + k] = Unit{i, k * S, min(S, B.n - k * S), B.log_nc};
        }
    }
}

// T of every candidate, and the work units.  A block of four warps takes a candidate and
// 1024 sources (32 a lane), a warp per endpoint: the distances of the endpoint's
// neighbours come as 4 plane words each (coalesced; a base's planes sit in the L2), four
// neighbours' loads in flight together, and every test is a few logic operations on 32
// sources at once.  The block that finishes a candidate cuts its list into units.  Bound
// by the dependent round trips (row ids, then planes) of a group of four neighbours.
// (One thread per (candidate, source), the plane bits gathered one by one, took 187 us
// for 2048 x 1024 + 512 x 3000 sources.)
__global__ void __launch_bounds__(128) batch_select(const BatchArgs a, const int max_n) {
    __shared__ uint32_t s_aff[4][32], s_near[4][32];
    if (a.ctl->bad) return;   // batch_reset rejected a candidate
    const unsigned n_cand = (unsigned)a.ctl->n_cand;
    const unsigned groups = ((unsigned)max_n + 1023u) / 1024u;
    const unsigned lane = threadIdx.x & 31u;
    const int i = (int)(threadIdx.x >> 5);   // the warp's endpoint
    const unsigned long long total = (unsigned long long)n_cand * groups;
    for (unsigned long long q = blockIdx.x; q < total; q += gridDim.x) {
        const unsigned cand = (unsigned)(q / groups), grp = (unsigned)(q % groups);
        const gg_swap sw = a.cands[cand];
        const BatchBase &B = a.bases[sw.base];
        const int n = B.n, d = B.d;
        if ((int)(grp * 1024u) >= n) continue;
        const SwapRows sr(sw);
        const int r = i == 0 ? sr.r[0] : i == 1 ? sr.r[1] : i == 2 ? sr.r[2] : sr.r[3];
        const int f = i == 0 ? sr.f[0] : i == 1 ? sr.f[1] : i == 2 ? sr.f[2] : sr.f[3];
        const int t = i == 0 ? sr.t[0] : i == 1 ? sr.t[1] : i == 2 ? sr.t[2] : sr.t[3];
        int mode = !B.valid ? kFull : (sw.a < 0 ? kBase : kNear);
        if (mode == kNear && !B.few_near && (long long)n_cand * B.chunks <= a.wave) mode = kFull;
        if (mode == kNear) {
            // both ends list each removed edge equally often (the edited graph is symmetric)
            int c[4] = {0, 0, 0, 0};
            for (int j0 = 0; j0 < d; j0 += 32)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    c[k] += __popc(__ballot_sync(0xffffffffu, j0 + (int)lane < d &&
                                                 __ldg(B.adj + (size_t)sr.r[k] * d + j0 + lane) == sr.f[k]));
            if (c[0] < 1 || c[0] != c[1] || c[2] < 1 || c[2] != c[3]) mode = kFull;
        }
        if (mode != kNear) {   // uniform over the block
            if (grp == 0u && threadIdx.x == 0u) a.cs[cand].mode = mode;
            if (grp == 0u && i == 0 && mode == kFull) {
                const int S = 128 << B.log_nc;
                unsigned u0 = 0u;
                if (lane == 0u) u0 = (unsigned)atomicAdd(&a.ctl->n_units, B.chunks);
                u0 = __shfl_sync(0xffffffffu, u0, 0);
                for (int k = (int)lane; k < B.chunks; k += 32)
                    a.units[u0 + k] = Unit{(int)cand, k * S, min(S, n - k * S), B.log_nc};
            }
            continue;
        }
        const unsigned w = grp * 32u + lane, words = ((unsigned)n + 31u) / 32u;
        const bool in = w < words;
        const uint32_t *pw = reinterpret_cast<const uint32_t *>(B.planes);
        const size_t ps = (size_t)n * B.cols * 4, cw = (size_t)B.cols * 4;
        const unsigned wl = in ? w : 0u;
        edit_masks(pw, ps, cw, B.adj, d, r, f, t, wl, (unsigned)B.radius, s_aff[i][lane], s_near[i][lane]);
        __syncthreads();
        if (i == 0) {
            uint32_t go = (s_near[0][lane] | s_near[1][lane] | s_near[2][lane] | s_near[3][lane]) &
                          (s_aff[0][lane] | s_aff[1][lane] | s_aff[2][lane] | s_aff[3][lane]);
            if (!in) go = 0u;
            else if (w == words - 1u && (n & 31)) go &= (1u << (n & 31)) - 1u;
            if (in) a.tbits[(size_t)cand * a.tbits_stride + w] = go;
            // these sources into the candidate's list
            const unsigned mine = __popc(go);
            unsigned incl = mine;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)lane >= o) incl += y;
            }
            const unsigned cnt = __shfl_sync(0xffffffffu, incl, 31);
            unsigned first = 0u;
            if (lane == 0u && cnt) first = atomicAdd(&a.cs[cand].count, cnt);
            unsigned at = __shfl_sync(0xffffffffu, first, 0) + incl - mine;
            unsigned sum = 0u, tops = 0u;
            uint16_t *lst = a.lists + (size_t)cand * a.list_stride;
            for (uint32_t m = go; m; m &= m - 1u) {
                const unsigned s = w * 32u + (unsigned)__ffs((int)m) - 1u;
                lst[at++] = (uint16_t)s;
                sum += __ldg(B.rowsum + s);
                tops += __ldg(B.top + s);
            }
            // (32 lanes x 32 sources x a sum below 16 n: below 2^32 for n < 2^18)
            sum = __reduce_add_sync(0xffffffffu, sum);
            tops = __reduce_add_sync(0xffffffffu, tops);
            unsigned prev = 0u;
            if (lane == 0u) {
                if (cnt) {
                    atomicAdd(&a.cs[cand].old_sum, (unsigned long long)sum);
                    atomicAdd(&a.cs[cand].tops, tops);
                }
                __threadfence();
                prev = atomicAdd(&a.cs[cand].groups_done, 1u);
            }
            prev = __shfl_sync(0xffffffffu, prev, 0);
            if (prev + 1u == ((unsigned)n + 1023u) / 1024u) {
                // every group of the candidate is in: equal units of at most 128 << l sources,
                // l the least that takes them at once within the base's chunk width
                unsigned T = 0u, u0 = 0u;
                if (lane == 0u) T = atomicAdd(&a.cs[cand].count, 0u);
                T = __shfl_sync(0xffffffffu, T, 0);
                int l = 0;
                while (l < B.log_nc && (128u << l) < T) ++l;
                const unsigned nu = (T + (128u << l) - 1u) >> (7 + l);
                if (nu) {
                    const unsigned per = (T + nu - 1u) / nu;
                    if (lane == 0u) u0 = (unsigned)atomicAdd(&a.ctl->n_units, (int)nu);
                    u0 = __shfl_sync(0xffffffffu, u0, 0);
                    for (unsigned k = lane; k < nu; k += 32u)
                        a.units[u0 + k] = Unit{(int)cand, (int)(k * per), (int)min(per, T - k * per), l};
                }
            }
        }
        __syncthreads();
    }
}

gg_status bfail(gg_status s, const std::string &m) {
    (void)cudaGetLastError();
    gg::set_last_error(m.c_str());
    return s;
}

#define GB_CK(call)                                                                          \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess)                                                               \
            return bfail(e_ == cudaErrorMemoryAllocation ? GG_OUT_OF_MEMORY : GG_CUDA_ERROR, \
                         std::string(#call) + ": " + cudaGetErrorString(e_));                \
    } while (0)

}  // namespace

struct gg_batch {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    std::vector<BatchBase> bases;          // host copy (adj = device pointers)
    std::vector<int32_t *> base_adj;       // device adjacency per base
    std::vector<uint16_t *> base_adj16;    // the same, packed as uint16 for the bulk copy
    BatchBase *d_bases = nullptr;
    BatchCtl *d_ctl = nullptr, *h_ctl = nullptr;
    int cap = 0;                           // candidates the buffers hold
    gg_swap *d_cands = nullptr, *h_cands = nullptr;
    gg_cand_result *d_out = nullptr, *h_out = nullptr;
    size_t smem = 0;
    int grid = 0;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    const gg_swap *graph_cands = nullptr;  // pointers baked into the graph
    gg_cand_result *graph_out = nullptr;
    cudaStream_t graph_stream = nullptr;
    unsigned *d_hist = nullptr;            // vertex histogram output
    size_t hist_cap = 0;
    double last_ms = 0.0;
    // near-source mode
    bool full_only = false;                // GG_BATCH_FULL=1: every candidate searches every source
    bool any_near = false;                 // some base is valid (batch_select is launched)
    bool near_always = false;              // GG_BATCH_FULL=0: near sources also where they do not pay
    std::vector<uint4 *> base_planes;      // per base: [kPlanes][n][cols]
    std::vector<unsigned *> base_stats;    // per base: rowsum[n], ecc[n], top[n]
    std::vector<std::pair<std::pair<int, int>, gg_engine *>> engines;  // per (n, degree): base passes
    int *d_flag = nullptr, *h_flag = nullptr;
    CandState *d_cs = nullptr;             // [cap]
    uint16_t *d_lists = nullptr;           // [cap][list_stride]
    int list_stride = 0;                   // largest base n
    uint32_t *d_tbits = nullptr;           // [cap][tbits_stride]
    int tbits_stride = 0;
    Unit *d_units = nullptr;               // [cap * max_chunks]
    int units_per_cand = 0;
    int max_chunks = 1;                    // most units a candidate can take
};

namespace {

void drop_graph(gg_batch *b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
}

// Shared memory of a unit with rows of 1 << l chunks: adjacency, T's bits, two bitsets.
size_t unit_smem(int n, int d, int l) {
    const size_t adj = ((size_t)n * d * 2 + 15) / 16 * 16, tb = ((size_t)(n + 31) / 32 * 4 + 15) / 16 * 16;
    return adj + tb + 2 * (size_t)n * (16u << l);
}
// (T's bits, at most 4 KB, come on top of the budget that decides which bases fit)
bool log_nc_fits(int n, int d, int l) {
    return unit_smem(n, d, l) - ((size_t)(n + 31) / 32 * 4 + 15) / 16 * 16 <= kSmemBudget;
}

std::string batch_tune_key(int device, int n, int d) { return gg::tune_key(device, "batch", {n, d}); }

// Chunk count per task row (a power of two): the one gg_batch_autotune recorded for
// this base shape on this kind of GPU, else the widest whose bitsets and adjacency
// fit the shared-memory budget.
int auto_log_nc(int device, int n, int d) {
    std::vector<int> tuned;
    if (gg::tune_get(batch_tune_key(device, n, d), &tuned) && !tuned.empty() && tuned[0] >= 0 &&
        tuned[0] <= 4 && log_nc_fits(n, d, tuned[0]))
        return tuned[0];
    int best = -1;
    for (int l = 0; l <= 4; ++l) {
        if (log_nc_fits(n, d, l)) best = l;
        if ((128 << l) >= n) break;
    }
    return best;
}

gg_status refresh_plan(gg_batch *b) {
    size_t smem = 0;
    int max_chunks = 1;
    for (auto &B : b->bases) {
        smem = std::max(smem, unit_smem(B.n, B.d, B.log_nc));
        max_chunks = std::max(max_chunks, B.chunks);
    }
    b->smem = smem;
    b->max_chunks = max_chunks;
    // (the limit belongs to the kernel, which handles with other bases launch too)
    GB_CK(cudaFuncSetAttribute(batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMost));
    int per_sm = 0, sms = 0;
    GB_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_kernel, kBatchBlock, smem));
    GB_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device));
    if (per_sm < 1) return bfail(GG_BAD_ARG, "batch task does not fit in shared memory");
    b->grid = per_sm * sms;
    GB_CK(cudaMemcpyAsync(b->d_bases, b->bases.data(), b->bases.size() * sizeof(BatchBase), cudaMemcpyHostToDevice, b->stream));
    GB_CK(cudaStreamSynchronize(b->stream));   // a population may come on another stream
    drop_graph(b);
    return GG_OK;
}

gg_status ensure_cap(gg_batch *b, int n) {
    int max_n = 0;
    for (auto &B : b->bases) max_n = std::max(max_n, B.n);
    if (n <= b->cap && max_n <= b->list_stride && b->max_chunks <= b->units_per_cand) return GG_OK;
    const int cap = std::max({n, n > b->cap ? 2 * b->cap : b->cap, 1});
    cudaFree(b->d_cands); cudaFree(b->d_out); cudaFree(b->d_cs); cudaFree(b->d_lists);
    cudaFree(b->d_tbits); cudaFree(b->d_units);
    cudaFreeHost(b->h_cands); cudaFreeHost(b->h_out);
    b->d_cands = nullptr; b->d_out = nullptr; b->h_cands = nullptr; b->h_out = nullptr;
    b->d_cs = nullptr; b->d_lists = nullptr; b->d_tbits = nullptr; b->d_units = nullptr;
    b->cap = 0;
    b->list_stride = std::max(max_n, 1);
    b->tbits_stride = (b->list_stride + 31) / 32;
    b->units_per_cand = b->max_chunks;
    GB_CK(cudaMalloc(&b->d_cands, (size_t)cap * sizeof(gg_swap)));
    GB_CK(cudaMalloc(&b->d_out, (size_t)cap * sizeof(gg_cand_result)));
    GB_CK(cudaMallocHost(&b->h_cands, (size_t)cap * sizeof(gg_swap)));
    GB_CK(cudaMallocHost(&b->h_out, (size_t)cap * sizeof(gg_cand_result)));
    GB_CK(cudaMalloc(&b->d_cs, (size_t)cap * sizeof(CandState)));
    GB_CK(cudaMalloc(&b->d_lists, (size_t)cap * b->list_stride * sizeof(uint16_t)));
    GB_CK(cudaMalloc(&b->d_tbits, (size_t)cap * b->tbits_stride * sizeof(uint32_t)));
    GB_CK(cudaMalloc(&b->d_units, (size_t)cap * b->units_per_cand * sizeof(Unit)));
    b->cap = cap;
    drop_graph(b);
    return GG_OK;
}

// Enqueue reset -> select (unless every candidate is searched in full) -> batch kernel ->
// finalize on `st` for candidates `cands`, results `out`; the candidate count comes from d_ctl.
gg_status enqueue(gg_batch *b, const gg_swap *cands, gg_cand_result *out, cudaStream_t st,
                  unsigned *hist = nullptr, int hist_k = 0) {
    BatchArgs a{};
    a.bases = b->d_bases; a.cands = cands; a.out = out; a.ctl = b->d_ctl;
    a.hist = hist; a.hist_k = hist_k;
    a.cs = b->d_cs;
    a.lists = b->d_lists; a.list_stride = b->list_stride;
    a.tbits = b->d_tbits; a.tbits_stride = b->tbits_stride;
    a.units = b->d_units;
    a.force_full = !b->any_near || hist;   // the histogram pass searches every source of its one candidate
    a.wave = b->near_always ? 0 : b->grid;
    batch_reset<<<64, 256, 0, st>>>(a);
    const unsigned long long blocks = (unsigned long long)b->cap * ((b->list_stride + 1023) / 1024);
    if (!a.force_full) batch_select<<<(int)std::min<unsigned long long>(blocks, 148ull * 16), 128, 0, st>>>(a, b->list_stride);
    batch_kernel<<<b->grid, kBatchBlock, b->smem, st>>>(a);
    batch_finalize<<<(int)std::min((b->cap + 3) / 4, 148 * 8), 128, 0, st>>>(a);
    GB_CK(cudaGetLastError());
    return GG_OK;
}

constexpr int kIncMaxN = 16384;   // larger bases search every source (planes of 4 n^2/8 bytes)
// ... and smaller ones than this, whose T is most of them: populations of 1 to 2048, near /
// full: n = 256, d = 4: 60 to 223 us / 48 to 184; n = 64, d = 3: 60 to 207 / 48 to 163 (n = 300, d = 6:
// 60 to 213 / 51 to 213; and no base pass: set_base and 32 moves 165 / 72).
constexpr int kIncMinN = 257;

// Whether T is so small that a unit of it is worth finding even where the full searches of
// a population run side by side (each then costs one unit's time, and batch_select 12 us):
// rows at most a quarter as wide, of a base of more than 512 vertices.  32 moves, near /
// full: n = 1000, d = 6: 62 / 73 us, d = 3: 110 / 75; n = 1500, d = 4: 97 / 77; n = 512, d = 3: 75 / 62;
// n = 700, d = 12: 60 / 73.  T is put at 0.8 of four balls of the radius in the tree.
bool worth_near(const BatchBase &B) {
    double ball = 1.0, ring = B.d;
    for (int k = 1; k <= B.radius && ball < B.n; ++k, ring *= B.d - 1) ball += ring;
    int l = 0;
    while (l < B.log_nc && (128 << l) < 0.8 * 4.0 * std::min<double>(ball, B.n)) ++l;
    return B.n > 512 && l + 2 <= B.log_nc;
}

// The base pass of base `id` (near-source mode): the single-graph engine
// evaluates the base with its distance planes (at most 16 levels), then every
// source's distance sum and eccentricity follow from the planes.  valid = 0
// (every candidate of the base searches every source) unless the base is
// symmetric, connected and of diameter <= 15.
gg_status base_pass(gg_batch *b, int id) {
    BatchBase &B = b->bases[id];
    const cudaStream_t st = b->stream;
    B.valid = 0;
    if (!b->full_only && (B.n >= kIncMinN || b->near_always) && B.n <= kIncMaxN) {
        gg_engine *eng = nullptr;
        for (auto &pe : b->engines)
            if (pe.first == std::make_pair(B.n, B.d)) eng = pe.second;
        if (!eng) {
            gg_status s = gg::graph_engine(B.n, B.d, b->device, &eng);
            if (s != GG_OK) return s;
            b->engines.push_back({{B.n, B.d}, eng});
            GB_CK(cudaSetDevice(b->device));
        }
        if (!b->base_planes[id]) {
            B.cols = (unsigned)gg::engine_plane_cols(eng);
            GB_CK(cudaMalloc(&b->base_planes[id], (size_t)kPlanes * B.n * B.cols * sizeof(uint4)));
            GB_CK(cudaMalloc(&b->base_stats[id], 3 * (size_t)B.n * sizeof(unsigned)));
        }
        GB_CK(cudaMemsetAsync(b->d_flag, 0, sizeof(int), st));
        const long long ent = (long long)B.n * B.d;
        table_symmetry<<<(int)((ent + 255) / 256), 256, 0, st>>>(b->base_adj[id], B.n, B.d, b->d_flag);
        GB_CK(cudaGetLastError());
        gg_eval_opts o{};
        o.max_levels = 1 << kPlanes;      // a base that needs more levels searches every source
        uint64_t counts[(1 << kPlanes) + 1] = {};
        o.level_counts = counts;
        gg::EvalExtra x;
        x.planes = b->base_planes[id];
        x.nplanes = kPlanes;
        x.no_graph = true;
        gg_result r{};
        gg_status s = gg::engine_eval(eng, b->base_adj[id], &o, &r, st, &x);
        if (s != GG_OK) return s;
        int sms = 0;
        GB_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device));
        // rows of the planes = sources: valid only on a symmetric base, which
        // `valid` below requires
        plane_row_stats<kPlanes><<<plane_row_stats_grid(B.n, sms), 256, 0, st>>>(
            b->base_planes[id], (unsigned long long)B.n * B.cols, B.cols, B.n, b->base_stats[id],
            b->base_stats[id] + B.n, b->base_stats[id] + 2 * B.n, (unsigned)r.levels);
        GB_CK(cudaGetLastError());
        GB_CK(cudaMemcpyAsync(b->h_flag, b->d_flag, sizeof(int), cudaMemcpyDeviceToHost, st));
        GB_CK(cudaStreamSynchronize(st));
        if (!*b->h_flag && r.connected && !r.capped && r.levels < (1 << kPlanes)) {
            B.valid = 1;
            B.total = r.total;
            B.reached = r.reached;
            B.levels = r.levels;
            B.at_top = counts[r.levels];
            B.radius = (std::max(r.levels, 1) - 1) / 2;
            B.top = b->base_stats[id] + 2 * B.n;
            B.planes = b->base_planes[id];
            B.rowsum = b->base_stats[id];
            B.ecc = b->base_stats[id] + B.n;
            B.few_near = worth_near(B);
        }
    }
    GB_CK(cudaMemcpyAsync(b->d_bases + id, &B, sizeof(BatchBase), cudaMemcpyHostToDevice, st));
    GB_CK(cudaStreamSynchronize(st));
    bool any = false;
    for (auto &x : b->bases) any |= x.valid != 0;
    if (any != b->any_near) drop_graph(b);
    b->any_near = any;
    return GG_OK;
}

__global__ void set_ctl(BatchCtl *ctl, const BatchCtl v) { *ctl = v; }

// int32 rows -> uint16 rows (vertex ids < 65536), zero padding to `padded` entries.
__global__ void pack16_kernel(const int32_t *adj, uint16_t *out, int n_ent, int padded) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < padded; k += gridDim.x * blockDim.x)
        out[k] = k < n_ent ? (uint16_t)adj[k] : (uint16_t)0;
}

unsigned adj16_bytes(int n, int d) { return (unsigned)((((size_t)n * d * 2) + 15) / 16 * 16); }

// The device-side candidate check starts clean for every launch.
void arm_check(gg_batch *b) {
    b->h_ctl->unit_ctr = 0;
    b->h_ctl->n_units = 0;
    b->h_ctl->bad = 0;
    b->h_ctl->timeout = 0;
    b->h_ctl->bad_index = 0x7fffffff;
    b->h_ctl->n_bases = (int)b->bases.size();
}

gg_status validate(const gg_batch *b, int n_cand, const gg_swap *c) {
    for (int i = 0; i < n_cand; ++i) {
        const gg_swap &s = c[i];
        if (s.base < 0 || s.base >= (int)b->bases.size())
            return bfail(GG_BAD_ARG, "candidate " + std::to_string(i) + ": unknown base");
        if (s.a < 0) continue;
        const int n = b->bases[s.base].n;
        if (s.a >= n || s.b < 0 || s.b >= n || s.c < 0 || s.c >= n || s.d < 0 || s.d >= n ||
            (s.mode != 0 && s.mode != 1))
            return bfail(GG_BAD_ARG, "candidate " + std::to_string(i) + ": vertex or mode out of range");
        if (s.a == s.b || s.a == s.c || s.a == s.d || s.b == s.c || s.b == s.d || s.c == s.d)
            return bfail(GG_BAD_ARG, "candidate " + std::to_string(i) + ": endpoints must be distinct");
    }
    return GG_OK;
}

}  // namespace

extern "C" {

gg_status gg_batch_create(int device, gg_batch **out) {
    if (!out) return bfail(GG_BAD_ARG, "null out");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return bfail(GG_NO_DEVICE, "no CUDA device");
    if (device < 0 || device >= ndev) return bfail(GG_NO_DEVICE, "device index out of range");
    gg_batch *b = new gg_batch();
    b->device = device;
    auto fail_and_free = [&](gg_status s) { gg_batch_destroy(b); return s; };
    if (cudaSetDevice(device) != cudaSuccess ||
        cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&b->ev0) != cudaSuccess || cudaEventCreate(&b->ev1) != cudaSuccess ||
        cudaMalloc(&b->d_ctl, sizeof(BatchCtl)) != cudaSuccess ||
        cudaMallocHost(&b->h_ctl, sizeof(BatchCtl)) != cudaSuccess ||
        cudaMalloc(&b->d_bases, 256 * sizeof(BatchBase)) != cudaSuccess ||
        cudaMalloc(&b->d_flag, sizeof(int)) != cudaSuccess ||
        cudaMallocHost(&b->h_flag, sizeof(int)) != cudaSuccess)
        return fail_and_free(bfail(GG_CUDA_ERROR, "batch set-up failed"));
    std::memset(b->h_ctl, 0, sizeof(BatchCtl));
    const char *f = std::getenv("GG_BATCH_FULL");
    b->full_only = f && std::atoi(f) != 0;
    b->near_always = f && !b->full_only;
    *out = b;
    return GG_OK;
}

gg_status gg_batch_add_base(gg_batch *b, int n, int degree, const int32_t *adj, int *base_id) {
    if (!b || !adj || !base_id || n < 1 || n > 65535 || degree < 1 || b->bases.size() >= 256)
        return bfail(GG_BAD_ARG, "need 1 <= n <= 65535, degree >= 1, at most 256 bases");
    for (long long k = 0; k < (long long)n * degree; ++k)
        if (adj[k] < 0 || adj[k] >= n) return bfail(GG_BAD_ARG, "adjacency entry outside [0, n)");
    const int lnc = auto_log_nc(b->device, n, degree);
    if (lnc < 0) return bfail(GG_BAD_ARG, "base graph too large for a shared-memory task");
    GB_CK(cudaSetDevice(b->device));
    int32_t *d = nullptr;
    uint16_t *d16 = nullptr;
    const unsigned b16 = adj16_bytes(n, degree);
    GB_CK(cudaMalloc(&d, (size_t)n * degree * sizeof(int32_t)));
    cudaError_t me = cudaMalloc(&d16, b16);
    if (me != cudaSuccess) { cudaFree(d); GB_CK(me); }
    // (on the stream that reads it: a copy on another one may still be under way)
    GB_CK(cudaMemcpyAsync(d, adj, (size_t)n * degree * sizeof(int32_t), cudaMemcpyHostToDevice, b->stream));
    pack16_kernel<<<64, 256, 0, b->stream>>>(d, d16, n * degree, (int)(b16 / 2));
    GB_CK(cudaGetLastError());
    BatchBase B{};
    B.adj = d; B.adj16 = d16; B.adj16_bytes = b16;
    B.n = n; B.d = degree; B.log_nc = lnc; B.chunks = (n + (128 << lnc) - 1) / (128 << lnc);
    b->bases.push_back(B);
    b->base_adj.push_back(d);
    b->base_adj16.push_back(d16);
    b->base_planes.push_back(nullptr);
    b->base_stats.push_back(nullptr);
    const int id = (int)b->bases.size() - 1;
    gg_status s = refresh_plan(b);
    if (s == GG_OK) s = base_pass(b, id);
    if (s != GG_OK) return s;
    *base_id = id;
    return GG_OK;
}

gg_status gg_batch_set_base(gg_batch *b, int base_id, const int32_t *adj) {
    if (!b || !adj || base_id < 0 || base_id >= (int)b->bases.size())
        return bfail(GG_BAD_ARG, "bad base or adjacency");
    const BatchBase &B = b->bases[base_id];
    for (long long k = 0; k < (long long)B.n * B.d; ++k)
        if (adj[k] < 0 || adj[k] >= B.n) return bfail(GG_BAD_ARG, "adjacency entry outside [0, n)");
    GB_CK(cudaSetDevice(b->device));
    // ordered on the batch stream: launches already enqueued see the old table
    GB_CK(cudaMemcpyAsync(b->base_adj[base_id], adj, (size_t)B.n * B.d * sizeof(int32_t),
                          cudaMemcpyHostToDevice, b->stream));
    pack16_kernel<<<64, 256, 0, b->stream>>>(b->base_adj[base_id], b->base_adj16[base_id], B.n * B.d,
                                            (int)(B.adj16_bytes / 2));
    GB_CK(cudaGetLastError());
    return base_pass(b, base_id);
}

gg_status gg_batch_set_chunk(gg_batch *b, int base_id, int sources) {
    if (!b || base_id < 0 || base_id >= (int)b->bases.size() || sources < 128 || sources % 128)
        return bfail(GG_BAD_ARG, "bad base or chunk width");
    int l = 0;
    while ((128 << l) < sources) ++l;
    if ((128 << l) != sources) return bfail(GG_BAD_ARG, "chunk width must be 128 * 2^k");
    BatchBase &B = b->bases[base_id];
    if (!log_nc_fits(B.n, B.d, l)) return bfail(GG_BAD_ARG, "chunk does not fit in shared memory");
    B.log_nc = l;
    B.chunks = (B.n + (128 << l) - 1) / (128 << l);
    B.few_near = worth_near(B);
    GB_CK(cudaSetDevice(b->device));
    return refresh_plan(b);
}

gg_status gg_batch_autotune(gg_batch *b, int n_cand, const gg_swap *cands, int trials, double *best_ms) {
    if (!b || n_cand < 1 || !cands || trials < 1) return bfail(GG_BAD_ARG, "bad arguments");
    gg_status s = validate(b, n_cand, cands);
    if (s != GG_OK) return s;
    std::vector<gg_cand_result> out((size_t)n_cand);
    auto time_it = [&](double *t) -> gg_status {
        gg_status r = gg_batch_eval(b, n_cand, cands, out.data());  // warm (and capture)
        if (r != GG_OK) return r;
        *t = 1e300;
        for (int k = 0; k < trials; ++k) {
            r = gg_batch_eval(b, n_cand, cands, out.data());
            if (r != GG_OK) return r;
            *t = std::min(*t, b->last_ms);
        }
        return GG_OK;
    };
    std::vector<char> used(b->bases.size(), 0);
    for (int i = 0; i < n_cand; ++i) used[cands[i].base] = 1;
    double best_t = 1e300;
    s = time_it(&best_t);
    if (s != GG_OK) return s;
    // coordinate descent over the bases the candidates use: each base's chunk width
    // with the others fixed
    for (size_t id = 0; id < b->bases.size(); ++id) {
        if (!used[id]) continue;
        const int n = b->bases[id].n, d = b->bases[id].d;
        int best_l = b->bases[id].log_nc;
        for (int l = 0; l <= 4; ++l) {
            if (l == best_l || !log_nc_fits(n, d, l)) continue;
            if (l > 0 && (128 << (l - 1)) >= n) break;   // wider than the base's sources
            s = gg_batch_set_chunk(b, (int)id, 128 << l);
            if (s != GG_OK) return s;
            double t = 0;
            s = time_it(&t);
            if (s != GG_OK) return s;
            if (t < best_t) { best_t = t; best_l = l; }
        }
        s = gg_batch_set_chunk(b, (int)id, 128 << best_l);
        if (s != GG_OK) return s;
        gg::tune_put(batch_tune_key(b->device, n, d), {best_l});
    }
    if (best_ms) *best_ms = best_t;
    return GG_OK;
}

gg_status gg_batch_chunk(gg_batch *b, int base_id, int *sources) {
    if (!b || !sources || base_id < 0 || base_id >= (int)b->bases.size()) return bfail(GG_BAD_ARG, "bad base");
    *sources = 128 << b->bases[base_id].log_nc;
    return GG_OK;
}

gg_status gg_batch_eval(gg_batch *b, int n_cand, const gg_swap *cands, gg_cand_result *out) {
    if (!b || n_cand < 0 || (n_cand && (!cands || !out))) return bfail(GG_BAD_ARG, "bad arguments");
    if (n_cand == 0) return GG_OK;
    gg_status s = validate(b, n_cand, cands);
    if (s != GG_OK) return s;
    GB_CK(cudaSetDevice(b->device));
    s = ensure_cap(b, n_cand);
    if (s != GG_OK) return s;
    std::memcpy(b->h_cands, cands, (size_t)n_cand * sizeof(gg_swap));
    b->h_ctl->n_cand = n_cand;
    arm_check(b);
    GB_CK(cudaMemcpyAsync(b->d_cands, b->h_cands, (size_t)n_cand * sizeof(gg_swap),
                          cudaMemcpyHostToDevice, b->stream));
    GB_CK(cudaMemcpyAsync(b->d_ctl, b->h_ctl, sizeof(BatchCtl), cudaMemcpyHostToDevice, b->stream));
    if (!b->exec) {  // capture reset -> kernel -> finalize once per buffer set
        GB_CK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
        gg_status es = enqueue(b, b->d_cands, b->d_out, b->stream);
        cudaGraph_t g = nullptr;
        cudaError_t ce = cudaStreamEndCapture(b->stream, &g);
        if (es != GG_OK) { if (g) cudaGraphDestroy(g); return es; }
        GB_CK(ce);
        b->graph = g;
        GB_CK(cudaGraphInstantiate(&b->exec, b->graph, 0));
    }
    GB_CK(cudaEventRecord(b->ev0, b->stream));
    GB_CK(cudaGraphLaunch(b->exec, b->stream));
    GB_CK(cudaEventRecord(b->ev1, b->stream));
    GB_CK(cudaMemcpyAsync(b->h_out, b->d_out, (size_t)n_cand * sizeof(gg_cand_result),
                          cudaMemcpyDeviceToHost, b->stream));
    GB_CK(cudaStreamSynchronize(b->stream));
    float ms = 0.f;
    GB_CK(cudaEventElapsedTime(&ms, b->ev0, b->ev1));
    b->last_ms = ms;
    std::memcpy(out, b->h_out, (size_t)n_cand * sizeof(gg_cand_result));
    if (out[0].levels < 0) return gg_batch_device_status(b, b->stream, nullptr);  // a flagged launch
    return GG_OK;
}

gg_status gg_batch_eval_device(gg_batch *b, int n_cand, const gg_swap *d_cands,
                               gg_cand_result *d_out, void *stream) {
    if (!b || n_cand < 0 || (n_cand && (!d_cands || !d_out))) return bfail(GG_BAD_ARG, "bad arguments");
    if (n_cand == 0) return GG_OK;
    GB_CK(cudaSetDevice(b->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : b->stream;
    gg_status cs = ensure_cap(b, n_cand);   // per-candidate lists of the near-source mode
    if (cs != GG_OK) return cs;
    b->h_ctl->n_cand = n_cand;
    arm_check(b);
    // the control block goes by value as a kernel argument: this call returns
    // before the GPU runs it, and the next call may change the host copy
    set_ctl<<<1, 1, 0, st>>>(b->d_ctl, *b->h_ctl);
    GB_CK(cudaGetLastError());
    GB_CK(cudaEventRecord(b->ev0, st));
    gg_status s = enqueue(b, d_cands, d_out, st);
    if (s != GG_OK) return s;
    GB_CK(cudaEventRecord(b->ev1, st));
    return GG_OK;
}

gg_status gg_batch_device_status(gg_batch *b, void *stream, int *first_bad) {
    if (!b) return bfail(GG_BAD_ARG, "null batch");
    GB_CK(cudaSetDevice(b->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : b->stream;
    GB_CK(cudaStreamSynchronize(st));
    BatchCtl c{};
    GB_CK(cudaMemcpy(&c, b->d_ctl, sizeof(BatchCtl), cudaMemcpyDeviceToHost));
    if (first_bad) *first_bad = c.bad ? c.bad_index : -1;
    if (c.timeout) return bfail(GG_TIMEOUT, "a CTA's wait for its adjacency copy ran past its limit");
    if (c.bad)
        return bfail(GG_BAD_ARG, "device candidate " + std::to_string(c.bad_index) +
                                     ": unknown base, vertex or mode out of range, or repeated endpoint");
    return GG_OK;
}

gg_status gg_batch_vertex_hist(gg_batch *b, int base_id, int K, uint32_t *hist) {
    if (!b || !hist || base_id < 0 || base_id >= (int)b->bases.size() || K < 1 || K > 64)
        return bfail(GG_BAD_ARG, "bad base, K or output");
    GB_CK(cudaSetDevice(b->device));
    gg_status s = ensure_cap(b, 1);
    if (s != GG_OK) return s;
    const int n = b->bases[base_id].n;
    const size_t need = (size_t)n * K;
    if (need > b->hist_cap) {
        cudaFree(b->d_hist);
        b->d_hist = nullptr;
        b->hist_cap = 0;
        GB_CK(cudaMalloc(&b->d_hist, need * sizeof(unsigned)));
        b->hist_cap = need;
    }
    unsigned *d_hist = b->d_hist;
    const gg_swap self{base_id, -1, -1, -1, -1, 0};
    b->h_cands[0] = self;
    b->h_ctl->n_cand = 1;
    arm_check(b);
    cudaError_t e = cudaMemsetAsync(d_hist, 0, (size_t)n * K * sizeof(unsigned), b->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(b->d_cands, b->h_cands, sizeof(gg_swap), cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(b->d_ctl, b->h_ctl, sizeof(BatchCtl), cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess) s = enqueue(b, b->d_cands, b->d_out, b->stream, d_hist, K);
    if (e == cudaSuccess && s == GG_OK)
        e = cudaMemcpyAsync(hist, d_hist, (size_t)n * K * sizeof(unsigned), cudaMemcpyDeviceToHost, b->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
    if (s != GG_OK) return s;
    GB_CK(e);
    return GG_OK;
}

gg_status gg_batch_last_ms(gg_batch *b, double *ms) {
    if (!b || !ms) return bfail(GG_BAD_ARG, "null argument");
    float f = 0.f;
    if (cudaEventElapsedTime(&f, b->ev0, b->ev1) == cudaSuccess) b->last_ms = f;
    else (void)cudaGetLastError();
    *ms = b->last_ms;
    return GG_OK;
}

gg_status gg_batch_destroy(gg_batch *b) {
    if (!b) return GG_OK;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    drop_graph(b);
    for (auto p : b->base_adj) cudaFree(p);
    for (auto p : b->base_adj16) cudaFree(p);
    for (auto p : b->base_planes) cudaFree(p);
    for (auto p : b->base_stats) cudaFree(p);
    for (auto &pe : b->engines) gg_destroy(pe.second);
    cudaFree(b->d_cs); cudaFree(b->d_lists); cudaFree(b->d_tbits); cudaFree(b->d_units);
    cudaFree(b->d_flag); cudaFreeHost(b->h_flag);
    cudaFree(b->d_bases); cudaFree(b->d_ctl); cudaFreeHost(b->h_ctl);
    cudaFree(b->d_cands); cudaFree(b->d_out); cudaFreeHost(b->h_cands); cudaFreeHost(b->h_out);
    cudaFree(b->d_hist);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return GG_OK;
}

}  // extern "C"
