// gg_direct.cuh -- all-pairs BFS of small graphs, one block a group of sources.
//
// Where a group's two visited sets fit a block's shared memory (up to about 28,000
// vertices at 32 sources a group), the level loop needs no grid barrier: a block keeps one
// word of W x 32 source bits per vertex, a level is next[v] = cur[v] | OR of cur[u] over
// v's pull neighbours (cudaASPLconv.cu:35-56), and only the counts of new pairs leave the
// SM.  The level loop of bfs_batch_kernel costs 3.4-4.4 us a level here however little
// there is to do (L2 round trips and a grid barrier).
//
// The first levels come from the sources' walk ends (a walk of length L from a source
// sets its bit at the end) while those are few.  A walk follows the table's rows from the
// source, so its ends are what the source pulls from; they are the vertices that reach it,
// too, when the table has no one-way entries.  The blocks check that between them (a share
// of the rows each, d look-ups an entry) and the last one tells the host, which runs a
// table that has some again without walks, every level a pass.
//
// The last block to finish writes the counters to host memory, clears them for the next
// launch and stores the launch's number, which the host waits for: an evaluation is this
// launch and, for larger tables, the copy before it.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "gg_kernels.cuh"

namespace gg {

constexpr int kDirectBlock = 1024;
constexpr int kDirectWalk = 2;   // walk ends of a group, at most this many times the rows

struct DirectCtl {
    unsigned done;       // blocks that finished
    int levels_run;      // last level executed by any block
    int bad;             // an adjacency entry outside [0, rows)
    int oneway;          // the walk met a table with one-way entries: the counters are not its counts
    unsigned seq;        // host: the number of the launch that handed its counters over
};

struct DirectArgs {
    const int32_t *adj;       // [rows][d]
    const int32_t *src;       // vertex of entry i of the source list, or nullptr: src_first + i
    int src_first, src_begin, ns_total;
    int rows, d;              // d >= 1
    int max_levels;
    const uint16_t *adj16;    // the same ids, checked by the caller (device or pinned host memory), or nullptr
    int adj_smem;             // the rows as 16-bit ids in shared memory (range-checked on the way from adj)
    // The first levels by walks: rows to check for one-way entries (0: no walks, nothing to
    // check): all of them, or, for a lift whose orbits translate onto one another, those of
    // its sources (check_src: the list's vertices, else src_first ..)
    int check;
    int check_src;
    unsigned seq;             // number of this launch
    const int *bad_table;     // or set by a check kernel before; nullptr: checked already
    DirectCtl *ctl, *h_ctl;   // device (zero between launches), host
    unsigned long long *counts, *h_counts;   // [max_levels + 1]; device ones zero between launches
    unsigned *masks, *h_masks;               // WVC: AND of every visited word after level L (ones between launches), or nullptr
    unsigned long long *batch_ns;            // host [2]: start and end of the launch's first and last block
};

template <int W>
struct DirectWord {
    uint32_t w[W];
};
template <int W>
__device__ __forceinline__ DirectWord<W> dw_load(const uint32_t *p) {
    DirectWord<W> r;
    if constexpr (W == 1) {
        r.w[0] = *p;
    } else if constexpr (W == 2) {
        const uint2 q = *reinterpret_cast<const uint2 *>(p);
        r.w[0] = q.x; r.w[1] = q.y;
    } else {
        const uint4 q = *reinterpret_cast<const uint4 *>(p);
        r.w[0] = q.x; r.w[1] = q.y; r.w[2] = q.z; r.w[3] = q.w;
    }
    return r;
}
template <int W>
__device__ __forceinline__ void dw_store(uint32_t *p, const DirectWord<W> r) {
    if constexpr (W == 1) *p = r.w[0];
    else if constexpr (W == 2) *reinterpret_cast<uint2 *>(p) = make_uint2(r.w[0], r.w[1]);
    else *reinterpret_cast<uint4 *>(p) = make_uint4(r.w[0], r.w[1], r.w[2], r.w[3]);
}

// The D neighbour ids of row v (D > 0), from 16-bit rows in shared memory or the table.
template <int D>
__device__ __forceinline__ void direct_ids(const uint16_t *srow, const int32_t *grow, const bool smem, unsigned (&id)[D]) {
    if (smem) {
        if constexpr (D % 4 == 0) {
#pragma unroll
            for (int k = 0; k < D / 4; ++k) {
                const uint2 q = reinterpret_cast<const uint2 *>(srow)[k];
                id[4 * k] = q.x & 0xffffu; id[4 * k + 1] = q.x >> 16;
                id[4 * k + 2] = q.y & 0xffffu; id[4 * k + 3] = q.y >> 16;
            }
        } else if constexpr (D % 2 == 0) {
#pragma unroll
            for (int k = 0; k < D / 2; ++k) {
                const unsigned q = reinterpret_cast<const unsigned *>(srow)[k];
                id[2 * k] = q & 0xffffu; id[2 * k + 1] = q >> 16;
            }
        } else {
#pragma unroll
            for (int k = 0; k < D; ++k) id[k] = srow[k];
        }
    } else if constexpr (D % 4 == 0) {
#pragma unroll
        for (int k = 0; k < D / 4; ++k) {
            const int4 q = __ldg(reinterpret_cast<const int4 *>(grow) + k);
            id[4 * k] = (unsigned)q.x; id[4 * k + 1] = (unsigned)q.y; id[4 * k + 2] = (unsigned)q.z; id[4 * k + 3] = (unsigned)q.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < D; ++k) id[k] = (unsigned)__ldg(grow + k);
    }
}

// One level: the thread's new pairs, and (masks) the AND of its rows' words.  D > 0: the
// degrees of the contest's usual graphs, a row's ids and gathers all in flight together; the
// others (D = 0) loop over the slots, up to a quarter longer a row at 7 to 15 (a row of 9000
// vertices, two words: d = 8 5.6 ns, 9 6.0, 12 6.0, 13 7.3).
template <int W, int D>
__device__ __forceinline__ unsigned direct_pass(const uint32_t *cur, uint32_t *nxt, const uint16_t *sadj,
                                                const int32_t *gadj, const bool smem, const int rows, const int d,
                                                unsigned &and_all) {
    unsigned cnt = 0u;
    for (int v = (int)threadIdx.x; v < rows; v += (int)blockDim.x) {
        const DirectWord<W> own = dw_load<W>(cur + (size_t)v * W);
        DirectWord<W> out = own;
        uint32_t full = ~0u;
#pragma unroll
        for (int k = 0; k < W; ++k) full &= own.w[k];
        if (full != ~0u) {
            if constexpr (D > 0) {
                unsigned id[D];
                direct_ids<D>(sadj + (size_t)v * D, gadj + (size_t)v * D, smem, id);
#pragma unroll
                for (int i = 0; i < D; ++i) {
                    const DirectWord<W> x = dw_load<W>(cur + (size_t)id[i] * W);
#pragma unroll
                    for (int k = 0; k < W; ++k) out.w[k] |= x.w[k];
                }
            } else {
#pragma unroll 4
                for (int i = 0; i < d; ++i) {
                    const unsigned u = smem ? (unsigned)sadj[(size_t)v * d + i] : (unsigned)__ldg(gadj + (size_t)v * d + i);
                    const DirectWord<W> x = dw_load<W>(cur + (size_t)u * W);
#pragma unroll
                    for (int k = 0; k < W; ++k) out.w[k] |= x.w[k];
                }
            }
#pragma unroll
            for (int k = 0; k < W; ++k) cnt += __popc(out.w[k] & ~own.w[k]);
        }
        dw_store<W>(nxt + (size_t)v * W, out);
#pragma unroll
        for (int k = 0; k < W; ++k) and_all &= out.w[k];
    }
    return cnt;
}

template <int W>
__global__ void __launch_bounds__(kDirectBlock, 1) direct_kernel(const DirectArgs a) {
    extern __shared__ uint4 dsm[];
    __shared__ unsigned s_cnt[3], s_and[3];
    __shared__ int s_last;
    const int tid = (int)threadIdx.x, nthr = (int)blockDim.x, lane = tid & 31;
    const int rows = a.rows, d = a.d;
    if (blockIdx.x == 0 && tid == 0) a.batch_ns[0] = gtimer();
    const bool smem = a.adj_smem != 0;
    uint16_t *sadj = reinterpret_cast<uint16_t *>(dsm);
    const size_t adj_b = smem ? ((size_t)rows * d * 2 + 15) / 16 * 16 : 0;
    uint32_t *cur = reinterpret_cast<uint32_t *>(reinterpret_cast<unsigned char *>(dsm) + adj_b);
    uint32_t *nxt = cur + ((size_t)rows * W + 3) / 4 * 4;
    const int first = (int)blockIdx.x * 32 * W, ns = min(32 * W, a.ns_total - first);
    if (tid < 3) { s_cnt[tid] = 0u; s_and[tid] = ~0u; }
    bool bad = a.bad_table && *a.bad_table;   // (a check kernel's answer)
    if (smem && a.adj16) {
        const int n8 = (rows * d + 7) / 8;   // (the buffer is padded to 16 bytes)
        for (int k = tid; k < n8; k += nthr)
            reinterpret_cast<uint4 *>(sadj)[k] = *(reinterpret_cast<const uint4 *>(a.adj16) + k);
    } else if (smem) {
        const int n = rows * d;
        if ((n & 3) == 0) {
            for (int k = tid; k < n / 4; k += nthr) {
                const int4 q = __ldg(reinterpret_cast<const int4 *>(a.adj) + k);
                unsigned x[4] = {(unsigned)q.x, (unsigned)q.y, (unsigned)q.z, (unsigned)q.w};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (x[j] >= (unsigned)rows) { bad = true; x[j] = 0u; }
                reinterpret_cast<uint2 *>(sadj)[k] = make_uint2(x[0] | (x[1] << 16), x[2] | (x[3] << 16));
            }
        } else {
            for (int k = tid; k < n; k += nthr) {
                unsigned x = (unsigned)__ldg(a.adj + k);
                if (x >= (unsigned)rows) { bad = true; x = 0u; }
                sadj[k] = (uint16_t)x;
            }
        }
    }
    // visited before level 1: the bits past the last source, and the diagonal
    for (int v = tid; v < rows; v += nthr) {
        DirectWord<W> x;
#pragma unroll
        for (int k = 0; k < W; ++k) x.w[k] = pad_word(32 * k, ns);
        dw_store<W>(cur + (size_t)v * W, x);
    }
    const bool any_bad = __syncthreads_or(bad) != 0;
    auto vertex = [&](const int j) {
        const int i = a.src_begin + first + j;
        return a.src ? __ldg(a.src + i) : a.src_first + i;
    };
    auto set_bit = [&](const int v, const int j) -> bool {
        const unsigned bit = 1u << (j & 31);
        return !(atomicOr(cur + (size_t)v * W + (j >> 5), bit) & bit);
    };
    int L = 0, executed = 0;
    if (!any_bad) {
        for (int j = tid; j < ns; j += nthr) set_bit(vertex(j), j);
        if (a.check) {
            // the block's share of the one-way check: is v among the neighbours of its neighbour u?
            auto entry = [&](const size_t at) { return smem ? (int)sadj[at] : __ldg(a.adj + at); };
            const int lo = (int)((long long)a.check * blockIdx.x / gridDim.x);
            const int hi = (int)((long long)a.check * (blockIdx.x + 1) / gridDim.x);
            for (int k = tid; k < (hi - lo) * d; k += nthr) {
                const int i = lo + k / d;
                const int v = !a.check_src ? i : a.src ? __ldg(a.src + i) : a.src_first + i;
                const size_t u = (size_t)entry((size_t)v * d + k % d) * d;
                bool back = false;
#pragma unroll 4
                for (int l = 0; l < d; ++l) back |= entry(u + l) == v;
                if (!back) a.ctl->oneway = 1;
            }
        }
        __syncthreads();
        const unsigned all = (unsigned)ns * (unsigned)rows;   // (rows < 2^16, ns <= 128)
        unsigned seen = (unsigned)ns;
        bool done = false;
        if (a.masks) {
            unsigned m = ~0u;
            for (size_t k = tid; k < (size_t)rows * W; k += nthr) m &= cur[k];
            m = __reduce_and_sync(0xffffffffu, m);
            if (lane == 0) atomicAnd(a.masks, m);
        }
        // End of level L: the block's new pairs (the same in every thread), its counters.
        auto end_level = [&](const unsigned cnt, const unsigned and_all) {
            const unsigned wsum = __reduce_add_sync(0xffffffffu, cnt);
            if (lane == 0 && wsum) atomicAdd(&s_cnt[L % 3], wsum);
            if (a.masks) {
                const unsigned m = __reduce_and_sync(0xffffffffu, and_all);
                if (lane == 0) atomicAnd(&s_and[L % 3], m);
            }
            __syncthreads();
            const unsigned c = s_cnt[L % 3];
            if (tid == 0) {
                if (c) atomicAdd(a.counts + L, (unsigned long long)c);
                if (a.masks) atomicAnd(a.masks + L, s_and[L % 3]);
                s_cnt[(L + 2) % 3] = 0u;
                s_and[(L + 2) % 3] = ~0u;
            }
            seen += c;
            executed = L;
            done = c == 0u || seen == all || L >= a.max_levels;
        };
        L = 1;
        for (unsigned ends = (unsigned)d; a.check && !done; ends *= (unsigned)d, ++L) {
            if ((unsigned long long)ends * (unsigned)ns > (unsigned long long)kDirectWalk * (unsigned)rows) break;
            // a thread takes a walk of L - 1 steps and its d ends (the ids of one row)
            unsigned cnt = 0u;
            const unsigned pre = ends / (unsigned)d;
            for (unsigned k = (unsigned)tid; k < pre * (unsigned)ns; k += (unsigned)nthr) {
                const int j = (int)(k / pre);
                unsigned w = k - (unsigned)j * pre;
                int v = vertex(j);
                for (int l = 1; l < L; ++l) {
                    const unsigned q = w / (unsigned)d;
                    const size_t at = (size_t)v * d + (w - q * (unsigned)d);
                    v = smem ? (int)sadj[at] : __ldg(a.adj + at);
                    w = q;
                }
                for (int i = 0; i < d; ++i)
                    cnt += set_bit(smem ? (int)sadj[(size_t)v * d + i] : __ldg(a.adj + (size_t)v * d + i), j);
            }
            unsigned and_all = ~0u;
            if (a.masks) {   // over every row, once all ends are in
                __syncthreads();
                for (size_t k = tid; k < (size_t)rows * W; k += nthr) and_all &= cur[k];
            }
            end_level(cnt, and_all);
        }
        for (; !done; ++L) {
            unsigned and_all = ~0u, cnt;
            switch (d) {
                case 3: cnt = direct_pass<W, 3>(cur, nxt, sadj, a.adj, smem, rows, d, and_all); break;
                case 4: cnt = direct_pass<W, 4>(cur, nxt, sadj, a.adj, smem, rows, d, and_all); break;
                case 5: cnt = direct_pass<W, 5>(cur, nxt, sadj, a.adj, smem, rows, d, and_all); break;
                case 6: cnt = direct_pass<W, 6>(cur, nxt, sadj, a.adj, smem, rows, d, and_all); break;
                case 8: cnt = direct_pass<W, 8>(cur, nxt, sadj, a.adj, smem, rows, d, and_all); break;
                case 12: cnt = direct_pass<W, 12>(cur, nxt, sadj, a.adj, smem, rows, d, and_all); break;
                case 16: cnt = direct_pass<W, 16>(cur, nxt, sadj, a.adj, smem, rows, d, and_all); break;
                default: cnt = direct_pass<W, 0>(cur, nxt, sadj, a.adj, smem, rows, d, and_all); break;
            }
            end_level(cnt, and_all);
            uint32_t *t = cur; cur = nxt; nxt = t;
        }
        // a group that ends before it reached everything keeps its mask at the later levels
        if (a.masks && seen != all) {
            const unsigned m = s_and[executed % 3];
            for (int l = executed + 1 + tid; l <= a.max_levels; l += nthr) atomicAnd(a.masks + l, m);
        }
    }
    // the last block hands the counters over and clears them
    if (tid == 0) {
        if (any_bad) a.ctl->bad = 1;
        else atomicMax(&a.ctl->levels_run, executed);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&a.ctl->done, 1u) + 1u == gridDim.x;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int run = ld_acquire_i(&a.ctl->levels_run), is_bad = ld_acquire_i(&a.ctl->bad);
    const int is_oneway = ld_acquire_i(&a.ctl->oneway);
    for (int l = tid; l <= run; l += nthr) {
        a.h_counts[l] = l == 0 ? (unsigned long long)a.ns_total : __ldcg(a.counts + l);
        a.counts[l] = 0ull;
    }
    if (a.masks)
        for (int l = tid; l <= a.max_levels; l += nthr) {
            if (l <= run) a.h_masks[l] = __ldcg(a.masks + l);
            a.masks[l] = ~0u;
        }
    if (tid == 0) {
        a.h_ctl->levels_run = run;
        a.h_ctl->bad = is_bad;
        a.h_ctl->oneway = is_oneway;
        a.ctl->done = 0u;
        a.ctl->levels_run = 0;
        a.ctl->bad = 0;
        a.ctl->oneway = 0;
        a.batch_ns[1] = gtimer();
    }
    // everything above reaches the host before the launch's number does
    __threadfence_system();
    __syncthreads();
    if (tid == 0) *reinterpret_cast<volatile unsigned *>(&a.h_ctl->seq) = a.seq;
}

}  // namespace gg
