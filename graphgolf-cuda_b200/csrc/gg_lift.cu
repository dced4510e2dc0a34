// gg_lift.cu -- batched exact evaluation of lifted candidates (gg_lift_* in gg.h):
// cyclic lifts ("part"), 2-D and 3-D torus lifts ("piece", "box").
//
// The part form of cudaASPLconv: M orbit vertices with d diffs each; vertex v of
// the N-vertex lift has the neighbours (v + diffs[v % M][i]) mod N, and the BFS
// runs from the M vertices 0..M-1 (cudaASPLconv.cu:197-243).  Piece and box
// tables hold 2- or 3-component diffs per orbit of a corner tile, the BFS runs
// from that tile (cudaASPLpiece.cu:159-216, cudaASPLbox.cu:166-226).  The
// reference's annealers change 2 or 4 slots of the table per proposal
// (cppcode/annealing.cpp:112-197, pieceannealing.cpp:113-204) and score each with
// one calculator call.
//
// Here one cooperative launch scores a population.  `lift_tables` writes every
// candidate's table (base + edit, diffs reduced to [0, n) per axis); for piece and
// box, `lift_expand` turns each into a pull adjacency and the kernel's EXPL
// variant reads adjacency rows and finds sources through a vertex ->
// representative map.  `lift_kernel`
// runs the candidates in rounds of G side by side: a round's bitsets hold, per
// vertex, W = G * cpc uint4 chunks (cpc = ceil(M/128)), chunk group g being the
// M sources of candidate g of the round, source s at bit s % 128 of chunk s / 128
// of its group.  A level is one pass over all (vertex, chunk) items:
//     new = (OR_i F[(v + diff_g[v % M][i]) mod N][w]) & ~V[v][w];  V |= new;  F' = new
// where g is the item's group, so neighbours always come from the item's own
// candidate.  Each thread owns one chunk column w (so one group, one counter and
// one table) and walks the vertices v = v0, v0 + VS, ...; consecutive lanes own
// consecutive columns, so the gathers of a neighbour row are contiguous 16-byte
// loads, all issued before the first is used.  Level 1 is the round's reset pass
// (a chunk's level-1 pairs are the sources among its own neighbours: no gather).
// Late in a round (past 85 % of its
// pairs reached) a chunk gathers half its neighbours first and the rest only
// while it still misses sources.  New pairs are counted per thread, reduced per
// group at the end of the level (shared atomics, then one global atomic per block
// and group into counts[L][k]); after the grid barrier every block reads the
// round's counts, and the round ends when no candidate found a pair or every
// candidate reached all M*N pairs.
//
// Moves by change (within the limits of delta_fits, where delta_pays says so): the base's
// distance rows are kept (delta_base: one search of the base that also writes bit-planes),
// and a candidate is scored by following what its edit changes in the rows near it
// (gg_delta.cuh): lift_select lists the rows, lift_delta follows them.  Edits that leave
// the lift asymmetric, changes that outgrow the lists or reach distances past kDeltaMax,
// bases that are asymmetric, disconnected or of diameter above 15, and handles with an
// explicit group run the search above.
#include "gg.h"
#include "gg_delta.cuh"
#include "gg_internal.h"
#include "gg_kernels.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

namespace {

constexpr int kLiftBlock = 256;
constexpr int kMaxGroup = 32;
constexpr int kFirstLevels = 256;   // count rows a launch starts with (see gg_lift_eval)

struct LiftArgs {
    const int32_t *tab;              // part form: [K][M][d] diffs in [0, N), rows 16-byte aligned when d % 4 == 0
    const int32_t *adj;              // piece / box: [K][N][d] pull adjacency of each candidate
    const int32_t *inv;              // piece / box: [N] representative index of a vertex, or -1
    int N, M, d, K, G, cpc, W;       // W = G * cpc chunks per vertex
    unsigned cols_threads;           // threads that own a column: the largest multiple of W <= grid threads
    unsigned vstep;                  // cols_threads / W: vertices between a thread's items
    int half_ppm;                    // past this share of the round's pairs reached: half gathers
    uint4 *V, *F0, *F1;              // [N][W]
    unsigned long long *counts;      // [max_levels + 1][K]: pairs first reached at level L
    int max_levels;
    unsigned long long *level_ns;    // [max_levels + 1]: device clock at the start ([0]) and
                                     // at the end of each level of the first round
    gg::Ctl *ctl;
    unsigned expected;
    long long wait_ns;
    // Distance bit-planes of a single candidate (the base), all zero before: bit s % 128 of
    // planes[(p * N + v) * cpc + s / 128] is bit p of the distance of (source s, vertex v);
    // distances up to 15.  nullptr: none.
    uint4 *planes;
};

// New pairs of chunk t at level L into the planes (one writer a chunk).
__device__ __forceinline__ void put_planes(const LiftArgs &a, const size_t t, const int L, const uint4 nw) {
    for (int p = 0; p < 4; ++p)
        if ((L >> p) & 1) {
            uint4 *q = a.planes + (size_t)p * a.N * a.cpc + t;
            *q = gg::u4or(*q, nw);
        }
}

// Candidate tables ([K][M][d][comps], comps = axes of the lift): slot (k, r, i)
// is the base slot unless candidate k's edit names slot (r, i).
__global__ void lift_tables(const int32_t *base, const gg_lift_edit *ed, int K, int M, int d, int comps,
                            int32_t *tab) {
    const long long per = (long long)M * d, total = per * K;
    for (long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x; x < total;
         x += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(x / per);
        const int e = (int)(x - (long long)k * per);
        const int r = e / d, i = e - r * d;
        const gg_lift_edit &q = ed[k];
        int hit = -1;
        for (int j = 0; j < q.count; ++j)
            if (q.row[j] == r && q.slot[j] == i) hit = j;
        for (int c = 0; c < comps; ++c)
            tab[x * comps + c] = hit >= 0 ? q.diff[hit][c] : __ldg(base + (size_t)e * comps + c);
    }
}

// Pull adjacency of every candidate of a 2-D or 3-D torus lift (axes sizes n,
// orbit sizes m; vertex (x * ny + y) * nz + z), from its table of diffs already
// reduced to [0, n): the expansion of cudaASPLpiece.cu:41-50 / cudaASPLbox.cu:44-57.
// One thread per (candidate, vertex): the coordinates and the orbit row once, then
// the row's d entries.
__global__ void lift_expand(const int32_t *tab, int K, int M, int d, int comps, int nx, int ny, int nz, int mx,
                            int my, int mz, int32_t *adj) {
    const long long N = (long long)nx * ny * nz, total = N * K;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(q / N);
        const int v = (int)(q - (long long)k * N);
        const int x = v / (ny * nz), rem = v - x * (ny * nz), y = rem / nz, z = rem - y * nz;
        const int r = ((x % mx) * my + (y % my)) * mz + (z % mz);
        const int32_t *t = tab + ((size_t)k * M + r) * d * comps;
        int32_t *out = adj + (size_t)q * d;
        for (int i = 0; i < d; ++i) {
            int tx = x + __ldg(t + i * comps), ty = y + __ldg(t + i * comps + 1);
            int tz = comps > 2 ? z + __ldg(t + i * comps + 2) : z;
            tx -= tx >= nx ? nx : 0;
            ty -= ty >= ny ? ny : 0;
            tz -= tz >= nz ? nz : 0;
            out[i] = (tx * ny + ty) * nz + tz;
        }
    }
}

// OR of F[u][w] over the neighbours u of slots [B, E) of `row` (u = v + diff,
// diff in [0, N)): every load of the span is issued before the first is used.
template <int B, int E, bool EXPL>
__device__ __forceinline__ void gather_span(const int32_t *row, unsigned v, unsigned w, unsigned N, unsigned W,
                                            const uint4 *Fc, uint4 &acc) {
    int32_t df[E - B];
    if constexpr (B % 4 == 0 && (E - B) % 4 == 0) {
#pragma unroll
        for (int i = 0; i < E - B; i += 4) {
            const int4 q = __ldg(reinterpret_cast<const int4 *>(row + B + i));
            df[i] = q.x; df[i + 1] = q.y; df[i + 2] = q.z; df[i + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < E - B; ++i) df[i] = __ldg(row + B + i);
    }
    uint4 x[E - B];
#pragma unroll
    for (int i = 0; i < E - B; ++i) {
        unsigned u = (unsigned)df[i];
        if constexpr (!EXPL) {   // a diff: u = (v + diff) mod N
            u += v;
            u -= u >= N ? N : 0u;
        }
        x[i] = __ldcg(Fc + (size_t)u * W + w);
    }
#pragma unroll
    for (int i = 0; i < E - B; ++i) gg::or_into(acc, x[i]);
}

// The same for a run-time degree: slots [b, e).
template <bool EXPL>
__device__ __forceinline__ void gather_any(const int32_t *row, int b, int e, unsigned v, unsigned w, unsigned N,
                                           unsigned W, const uint4 *Fc, uint4 &acc) {
#pragma unroll 4
    for (int i = b; i < e; ++i) {
        unsigned u = (unsigned)__ldg(row + i);
        if constexpr (!EXPL) {
            u += v;
            u -= u >= N ? N : 0u;
        }
        gg::or_into(acc, __ldcg(Fc + (size_t)u * W + w));
    }
}

// Representative index of vertex u: u itself for a part (sources 0..M-1),
// inv[u] for a piece or box; -1 for a vertex that is no source.
template <bool EXPL>
__device__ __forceinline__ int source_of(unsigned u, unsigned M, const int32_t *inv) {
    if constexpr (EXPL) return __ldg(inv + u);
    else return u < M ? (int)u : -1;
}

// The sources among the pull neighbours of v (row `row`, slots [B, E)) that lie in
// the chunk of sources [lo, lo + 128), as bits.
template <int B, int E, bool EXPL>
__device__ __forceinline__ void sources_span(const int32_t *row, unsigned v, unsigned lo, unsigned N, unsigned M,
                                             const int32_t *inv, unsigned nb[4]) {
    int32_t df[E - B];
    if constexpr (B % 4 == 0 && (E - B) % 4 == 0) {
#pragma unroll
        for (int i = 0; i < E - B; i += 4) {
            const int4 q = __ldg(reinterpret_cast<const int4 *>(row + B + i));
            df[i] = q.x; df[i + 1] = q.y; df[i + 2] = q.z; df[i + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < E - B; ++i) df[i] = __ldg(row + B + i);
    }
#pragma unroll
    for (int i = 0; i < E - B; ++i) {
        unsigned u = (unsigned)df[i];
        if constexpr (!EXPL) {
            u += v;
            u -= u >= N ? N : 0u;
        }
        const int sv = source_of<EXPL>(u, M, inv);
        const unsigned o = (unsigned)sv - lo;
        if (sv >= 0 && o < 128u) nb[o >> 5] |= 1u << (o & 31u);
    }
}

// The reset pass of a round with level 1 folded in: the pairs a chunk (v, w)
// reaches at level 1 are the sources among its pull neighbours that lie in the
// chunk, so the pass writes the padding bits, the diagonal and those pairs into V
// and their frontier into F1 (`Fn`) without a gather.  Columns of candidates past
// the last one (mine == false) start full.  `rows`: the column's candidate's diff
// table (part, row v % M) or pull adjacency (piece / box, row v).  Returns the
// thread's new pairs.
template <int D, bool EXPL>
__device__ __forceinline__ unsigned level1_pass(const LiftArgs &a, const int32_t *rows, unsigned v0,
                                                unsigned vstep, unsigned rstep, unsigned w, unsigned cc,
                                                bool mine, uint4 *Fn) {
    const unsigned N = (unsigned)a.N, M = (unsigned)a.M, W = (unsigned)a.W;
    const uint4 pad = mine ? gg::pad_mask((int)cc, a.M)
                           : make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
    const unsigned lo = cc * 128u;     // sources of this chunk: [lo, lo + 128) of the group
    unsigned cnt = 0, r = v0 % M;
    for (unsigned v = v0; v < N; v += vstep) {
        uint4 vis = pad, n1 = gg::u4zero();
        if (mine) {
            const int sv = source_of<EXPL>(v, M, a.inv);
            const unsigned o = (unsigned)sv - lo;
            if (sv >= 0 && o < 128u) {   // the diagonal
                const unsigned bit = 1u << (o & 31u);
                switch (o >> 5) {
                    case 0: vis.x |= bit; break;
                    case 1: vis.y |= bit; break;
                    case 2: vis.z |= bit; break;
                    default: vis.w |= bit; break;
                }
            }
            const int32_t *row = rows + (size_t)(EXPL ? v : r) * a.d;
            unsigned nb[4] = {0u, 0u, 0u, 0u};
            if constexpr (D > 0) {
                sources_span<0, D, EXPL>(row, v, lo, N, M, a.inv, nb);
            } else {
                for (int i = 0; i < a.d; ++i) {
                    unsigned u = (unsigned)__ldg(row + i);
                    if constexpr (!EXPL) {
                        u += v;
                        u -= u >= N ? N : 0u;
                    }
                    const int su = source_of<EXPL>(u, M, a.inv);
                    const unsigned ou = (unsigned)su - lo;
                    if (su >= 0 && ou < 128u) nb[ou >> 5] |= 1u << (ou & 31u);
                }
            }
            n1 = gg::andnot(make_uint4(nb[0], nb[1], nb[2], nb[3]), vis);
            gg::or_into(vis, n1);
            cnt += gg::u4popc(n1);
            if (a.planes && gg::u4any(n1)) put_planes(a, (size_t)v * W + w, 1, n1);
        }
        a.V[(size_t)v * W + w] = vis;
        Fn[(size_t)v * W + w] = n1;
        r += rstep;
        r -= r >= M ? M : 0u;
    }
    return cnt;
}

// D > 0: the degree at compile time; D == 0: a.d at run time.  EXPL: piece / box
// (per-candidate pull adjacency and representative map); otherwise part (diffs).
template <int D, bool EXPL>
__global__ void __launch_bounds__(kLiftBlock, 4) lift_kernel(const LiftArgs a) {
    __shared__ unsigned s_cnt[kMaxGroup];
    __shared__ unsigned long long s_reached[kMaxGroup];
    __shared__ int s_half;
    if (threadIdx.x < kMaxGroup) s_cnt[threadIdx.x] = 0u;
    unsigned epoch = 0;
    const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x;
    // this thread's column (threads past cols_threads own none)
    const bool owner = tid < a.cols_threads;
    const unsigned w = owner ? tid % (unsigned)a.W : 0u;
    const unsigned g = w / (unsigned)a.cpc, cc = w - g * (unsigned)a.cpc;
    const unsigned v0 = owner ? tid / (unsigned)a.W : (unsigned)a.N;
    const unsigned N = (unsigned)a.N, W = (unsigned)a.W, M = (unsigned)a.M;
    const unsigned vstep = a.vstep, rstep = vstep % M;
    const unsigned long long all_pairs = (unsigned long long)a.M * (unsigned long long)a.N;
    const int dh = a.d / 2;
    const int rounds = (a.K + a.G - 1) / a.G;
    int zeroed = 1;        // rows 0 and 1 of counts are zeroed by the host
    int levels_run = 0;
    for (int rd = 0; rd < rounds; ++rd) {
        const int k0 = rd * a.G;
        const int live = min(a.G, a.K - k0);
        const bool mine = owner && (int)g < live;   // a column of a live candidate
        const int kc = k0 + (mine ? (int)g : 0);
        const int32_t *rows = EXPL ? a.adj + (size_t)kc * a.N * a.d : a.tab + (size_t)kc * a.M * a.d;
        if (threadIdx.x == 0) s_half = 0;   // read after the next barrier
        if (rd == 0 && a.level_ns && blockIdx.x == 0 && threadIdx.x == 0) a.level_ns[0] = gg::gtimer();
        unsigned long long reached = threadIdx.x < (unsigned)live ? (unsigned long long)a.M : 0ull;
        for (int L = 1; L <= a.max_levels; ++L) {
            const uint4 *Fc = (L & 1) ? a.F0 : a.F1;
            uint4 *Fn = (L & 1) ? a.F1 : a.F0;
            // the next level's count row, before any block can add to it
            if (blockIdx.x == 0 && L + 1 > zeroed && L + 1 <= a.max_levels)
                for (int k = threadIdx.x; k < a.K; k += blockDim.x) a.counts[(size_t)(L + 1) * a.K + k] = 0ull;
            zeroed = max(zeroed, L + 1);
            unsigned cnt = 0;
            unsigned r = v0 % M;
            if (L == 1) {
                // level 1 is the round's reset pass
                cnt = level1_pass<D, EXPL>(a, rows, v0, vstep, rstep, w, cc, mine, Fn);
            } else {
                const bool half = s_half != 0;
                for (unsigned v = v0; v < N; v += vstep) {
                    const size_t t = (size_t)v * W + w;
                    const uint4 own = __ldcg(a.V + t);
                    uint4 nw = gg::u4zero();
                    if (!gg::u4full(own)) {
                        // full from the reset pass unless the column is a live candidate's
                        const int32_t *row = rows + (size_t)(EXPL ? v : r) * a.d;
                        uint4 acc = gg::u4zero();
                        if constexpr (D > 0) {
                            if (!half && D <= 12) {
                                gather_span<0, D, EXPL>(row, v, w, N, W, Fc, acc);
                            } else if (!half) {   // two spans keep the loads within the registers
                                gather_span<0, D / 2, EXPL>(row, v, w, N, W, Fc, acc);
                                gather_span<D / 2, D, EXPL>(row, v, w, N, W, Fc, acc);
                            } else {
                                gather_span<0, D / 2, EXPL>(row, v, w, N, W, Fc, acc);
                                if (!gg::u4full(gg::u4or(own, acc))) gather_span<D / 2, D, EXPL>(row, v, w, N, W, Fc, acc);
                            }
                        } else {
                            gather_any<EXPL>(row, 0, half ? dh : a.d, v, w, N, W, Fc, acc);
                            if (half && !gg::u4full(gg::u4or(own, acc))) gather_any<EXPL>(row, dh, a.d, v, w, N, W, Fc, acc);
                        }
                        nw = gg::andnot(acc, own);
                        if (gg::u4any(nw)) {
                            a.V[t] = gg::u4or(own, nw);
                            cnt += gg::u4popc(nw);
                            if (a.planes) put_planes(a, t, L, nw);
                        }
                    }
                    Fn[t] = nw;
                    r += rstep;   // (v + vstep) % M
                    r -= r >= M ? M : 0u;
                }
            }
            // per group: lanes of one group share a key
            const int key = cnt ? (int)g : -1;
            const unsigned peers = __match_any_sync(0xffffffffu, key);
            const unsigned sum = __reduce_add_sync(peers, cnt);
            if (key >= 0 && (int)(threadIdx.x & 31u) == __ffs((int)peers) - 1) atomicAdd(&s_cnt[key], sum);
            __syncthreads();
            if (threadIdx.x < (unsigned)live && s_cnt[threadIdx.x]) {
                atomicAdd(a.counts + (size_t)L * a.K + k0 + threadIdx.x, (unsigned long long)s_cnt[threadIdx.x]);
                s_cnt[threadIdx.x] = 0u;
            }
            if (!gg::grid_sync(a.ctl, a.expected, a.wait_ns, L, epoch)) return;
            if (rd == 0 && a.level_ns && blockIdx.x == 0 && threadIdx.x == 0) a.level_ns[L] = gg::gtimer();
            levels_run = max(levels_run, L);
            int more = 0;
            if (threadIdx.x < (unsigned)live) {
                const unsigned long long n = gg::ld_relaxed_u64(a.counts + (size_t)L * a.K + k0 + threadIdx.x);
                reached += n;
                more = n != 0ull && reached < all_pairs;
                s_reached[threadIdx.x] = reached;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                unsigned long long sum_r = 0;
                for (int q = 0; q < live; ++q) sum_r += s_reached[q];
                s_half = (double)sum_r > (double)a.half_ppm * 1e-6 * (double)live * (double)all_pairs;
            }
            if (!__syncthreads_or(more)) break;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.ctl->levels_run = levels_run;
}

// ---- moves by change ---------------------------------------------------------------

// The lift's axes: n lifted and m orbit sizes; a part has one axis.
struct LiftAxes {
    int axes;
    int n[3], m[3];
    // vertex of copy c of orbit o
    __device__ __forceinline__ int vertex(int o, int c) const {
        int v = 0, mul = 1;
        for (int j = axes - 1; j >= 0; --j) {
            const int k = n[j] / m[j], x = o % m[j] + m[j] * (c % k);
            o /= m[j];
            c /= k;
            v += x * mul;
            mul *= n[j];
        }
        return v;
    }
    // orbit and copy of vertex v
    __device__ __forceinline__ void place(int v, int &o, int &c) const {
        int mo = 1, mc = 1;
        o = c = 0;
        for (int j = axes - 1; j >= 0; --j) {
            const int x = v % n[j];
            v /= n[j];
            o += x % m[j] * mo;
            c += x / m[j] * mc;
            mo *= m[j];
            mc *= n[j] / m[j];
        }
    }
    // v moved by the diff df (components in [0, n))
    __device__ __forceinline__ int move(int v, const int32_t *df) const {
        int r = 0, mul = 1;
        for (int j = axes - 1; j >= 0; --j) {
            int x = v % n[j] + df[j];
            v /= n[j];
            x -= x >= n[j] ? n[j] : 0;
            r += x * mul;
            mul *= n[j];
        }
        return r;
    }
    // orbit that the diff df leads to from orbit o, and the reverse diff
    __device__ __forceinline__ int orbit_at(int o, const int32_t *df) const {
        int r = 0, mul = 1;
        for (int j = axes - 1; j >= 0; --j) {
            r += (o % m[j] + df[j]) % m[j] * mul;
            o /= m[j];
            mul *= m[j];
        }
        return r;
    }
    __device__ __forceinline__ bool reverse(const int32_t *a, const int32_t *b) const {
        for (int j = 0; j < axes; ++j)
            if ((a[j] + b[j]) % n[j] != 0) return false;
        return true;
    }
    __device__ __forceinline__ bool same(const int32_t *a, const int32_t *b) const {
        for (int j = 0; j < axes; ++j)
            if (a[j] != b[j]) return false;
        return true;
    }
};

// A row of the base adjacency: rw 16-bit words -- the d neighbours, padding with the vertex
// itself, then its orbit and its copy in the last two.
__global__ void delta_rows_kernel(const int32_t *table, const LiftAxes ax, int N, int d, int rw, uint16_t *rows) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < N; v += gridDim.x * blockDim.x) {
        int o, c;
        ax.place(v, o, c);
        uint16_t *out = rows + (size_t)v * rw;
        for (int i = 0; i < rw - 2; ++i)
            out[i] = (uint16_t)(i < d ? ax.move(v, table + ((size_t)o * d + i) * ax.axes) : v);
        out[rw - 2] = (uint16_t)o;
        out[rw - 1] = (uint16_t)c;
    }
}

// A part's diffs as 16-bit words, dp a row, padded with 0.
__global__ void delta_diffs_kernel(const int32_t *table, int M, int d, int dp, uint16_t *diffs) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < M * dp; k += gridDim.x * blockDim.x) {
        const int o = k / dp, i = k % dp;
        diffs[k] = (uint16_t)(i < d ? table[(size_t)o * d + i] : 0);
    }
}

// 1 into *asym when some entry of the table and its reverse entry are not listed equally
// often by their rows.
__global__ void delta_symmetry(const int32_t *table, const LiftAxes ax, int M, int d, int *asym) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < M * d; k += gridDim.x * blockDim.x) {
        const int o = k / d;
        const int32_t *df = table + (size_t)k * ax.axes;
        const int q = ax.orbit_at(o, df);
        int here = 0, back = 0;
        for (int j = 0; j < d; ++j) {
            here += ax.same(table + ((size_t)o * d + j) * ax.axes, df);
            back += ax.reverse(table + ((size_t)q * d + j) * ax.axes, df);
        }
        if (here != back) *asym = 1;
    }
}

// Distance planes -> byte rows dist[s][v] (pitch bytes a row).  A block takes 128 vertices
// and 128 sources: a thread holds its vertex's four plane words, and each source's bytes go
// out 32 a warp.
__global__ void __launch_bounds__(128) delta_bytes(const uint4 *planes, int N, int M, int cpc, uint8_t *dist, int pitch) {
    const int v = blockIdx.x * 128 + (int)threadIdx.x, c = blockIdx.y;
    uint4 x[4];
#pragma unroll
    for (int p = 0; p < 4; ++p)
        x[p] = v < N ? __ldg(planes + ((size_t)p * N + v) * cpc + c) : gg::u4zero();
    if (v >= pitch) return;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        unsigned w[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) w[p] = gg::comp_of(x[p], k);
        const int s0 = c * 128 + k * 32;
#pragma unroll 8
        for (int i = 0; i < 32; ++i) {
            if (s0 + i >= M) break;
            dist[(size_t)(s0 + i) * pitch + v] =
                (uint8_t)(((w[0] >> i) & 1u) | (((w[1] >> i) & 1u) << 1) | (((w[2] >> i) & 1u) << 2) | (((w[3] >> i) & 1u) << 3));
        }
    }
}

// ball[o]: the orbits with a vertex within `radius` of representative o, one bit each.
__global__ void __launch_bounds__(256) delta_balls(const uint8_t *dist, int pitch, int N, const uint16_t *rows, int rw,
                                                   int words, unsigned radius, uint32_t *ball) {
    extern __shared__ uint32_t s_ball[];
    const int o = blockIdx.x;
    for (int k = threadIdx.x; k < words; k += blockDim.x) s_ball[k] = 0u;
    __syncthreads();
    const uint4 *row = reinterpret_cast<const uint4 *>(dist + (size_t)o * pitch);
    const unsigned r4 = radius * 0x01010101u;
    for (int k = threadIdx.x; k < pitch / 16; k += blockDim.x) {
        const uint4 q = __ldg(row + k);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            for (unsigned m = __vcmpleu4(gg::comp_of(q, j), r4) & 0x01010101u; m; m &= m - 1u) {
                const int v = k * 16 + j * 4 + (__ffs((int)m) - 1) / 8;
                if (v >= N) continue;
                const unsigned b = __ldg(rows + (size_t)v * rw + rw - 2);
                atomicOr(s_ball + (b >> 5), 1u << (b & 31u));
            }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < words; k += blockDim.x) ball[(size_t)o * words + k] = s_ball[k];
}

// A candidate's state: how it is scored, and the change of its number of pairs at each
// distance (kDeltaInf: unreached).
enum { kByChange = 0, kSearch = 1 };
struct DeltaCand {
    int mode;
    int count;                     // rows followed
    int edited;                    // distinct edited orbits
    int orbit[4];                  // they, or -1
    int hist[gg::kDeltaLevels];
};

// `rows` sources of a candidate's list, from `first` on.
struct DeltaUnit {
    int cand, first, rows;
};

struct DeltaArgs {
    LiftAxes ax;
    int N, M, d, g, K;
    const int32_t *table;          // base table, diffs in [0, n)
    const gg_lift_edit *ed;
    const uint16_t *rows;          // base adjacency rows
    int rw;
    const uint16_t *diffs;         // part: base diffs, dp a row
    int dp;
    gg::FastDiv div_m;             // division by M
    const uint8_t *dist;
    int pitch;
    const uint32_t *ball;
    int words;                     // words of a bit per orbit
    DeltaCand *cand;
    uint32_t *near;                // [K][words]: P
    uint16_t *lists;               // [K][M]
    uint3 *changes;                // [K][4 g]
    uint16_t *patch;               // part: [K][4][dp] diff rows of the edited orbits; else [K][4][g][rw]
    DeltaUnit *units;
    int *ctr;                      // [0] units made, [1] units taken
    int unit_rows;
    uint32_t *spill;               // [blocks of lift_delta][3][kDeltaSpill]
};

// One block a candidate: whether its edit keeps the lift symmetric, P from the edited
// orbits' balls, the work units, the changed pull entries and the edited rows.
__global__ void __launch_bounds__(128) lift_select(const DeltaArgs a) {
    __shared__ int s_mode, s_ne, s_orb[4], s_cnt, s_u0;
    const int k = blockIdx.x, tid = threadIdx.x;
    const gg_lift_edit &e = a.ed[k];
    const int ne_max = e.count;
    if (tid == 0) {
        int mode = kByChange, ne = 0;
        const int32_t *old[4], *add[4];
        for (int j = 0; j < ne_max; ++j) {
            old[j] = a.table + ((size_t)e.row[j] * a.d + e.slot[j]) * a.ax.axes;
            add[j] = e.diff[j];
            for (int i = 0; i < j; ++i)
                if (e.row[i] == e.row[j] && e.slot[i] == e.slot[j]) mode = kSearch;   // a slot edited twice
            bool seen = false;
            for (int i = 0; i < ne; ++i) seen |= s_orb[i] == e.row[j];
            if (!seen) s_orb[ne++] = e.row[j];
        }
        // the removed entries, and the added ones, hold each entry as often as its reverse
        for (int t = 0; t < 2; ++t)
            for (int j = 0; j < ne_max; ++j) {
                const int32_t *const *df = t ? add : old;
                const int q = a.ax.orbit_at(e.row[j], df[j]);
                int here = 0, back = 0;
                for (int i = 0; i < ne_max; ++i) {
                    here += e.row[i] == e.row[j] && a.ax.same(df[i], df[j]);
                    back += e.row[i] == q && a.ax.reverse(df[i], df[j]);
                }
                if (here != back) mode = kSearch;
            }
        s_mode = mode;
        s_ne = ne;
        s_cnt = 0;
        DeltaCand &c = a.cand[k];
        c.mode = mode;
        c.edited = ne;
        for (int i = 0; i < 4; ++i) c.orbit[i] = i < ne ? s_orb[i] : -1;
    }
    if (tid < gg::kDeltaLevels) a.cand[k].hist[tid] = 0;
    __syncthreads();
    if (s_mode != kByChange) {
        if (tid == 0) a.cand[k].count = 0;
        return;
    }
    const int ne = s_ne;
    uint16_t *lst = a.lists + (size_t)k * a.M;
    for (int w = tid; w < a.words; w += blockDim.x) {
        uint32_t p = 0u;
        for (int i = 0; i < ne; ++i) p |= __ldg(a.ball + (size_t)s_orb[i] * a.words + w);
        a.near[(size_t)k * a.words + w] = p;
        if (p) {
            int at = atomicAdd(&s_cnt, __popc(p));
            for (; p; p &= p - 1u) lst[at++] = (uint16_t)(w * 32 + __ffs((int)p) - 1);
        }
    }
    for (int q = tid; q < ne_max * a.g; q += blockDim.x) {
        const int j = q / a.g, c = q % a.g;
        const int r = a.ax.vertex(e.row[j], c);
        a.changes[(size_t)k * 4 * a.g + q] = make_uint3((unsigned)r, __ldg(a.rows + (size_t)r * a.rw + e.slot[j]),
                                                        (unsigned)a.ax.move(r, e.diff[j]));
    }
    if (a.ax.axes == 1) {
        for (int q = tid; q < ne * a.dp; q += blockDim.x) {
            const int i = q / a.dp, x = q % a.dp;
            int v = __ldg(a.diffs + (size_t)s_orb[i] * a.dp + x);
            for (int j = 0; j < ne_max; ++j)
                if (e.row[j] == s_orb[i] && e.slot[j] == x) v = e.diff[j][0];
            a.patch[(size_t)k * 4 * a.dp + q] = (uint16_t)v;
        }
    } else {
        for (int q = tid; q < ne * a.g; q += blockDim.x) {
            const int i = q / a.g, c = q % a.g;
            const int v = a.ax.vertex(s_orb[i], c);
            uint16_t *out = a.patch + ((size_t)(k * 4 + i) * a.g + c) * a.rw;
            for (int x = 0; x < a.rw; ++x) out[x] = __ldg(a.rows + (size_t)v * a.rw + x);
            for (int j = 0; j < ne_max; ++j)
                if (e.row[j] == s_orb[i]) out[e.slot[j]] = (uint16_t)a.ax.move(v, e.diff[j]);
        }
    }
    __syncthreads();
    const int cnt = s_cnt, nu = (cnt + a.unit_rows - 1) / a.unit_rows;
    if (tid == 0) {
        a.cand[k].count = cnt;
        s_u0 = nu ? atomicAdd(a.ctr, nu) : 0;
    }
    __syncthreads();
    for (int u = tid; u < nu; u += blockDim.x)
        a.units[s_u0 + u] = DeltaUnit{k, u * a.unit_rows, min(a.unit_rows, cnt - u * a.unit_rows)};
}

// A candidate's graph: base rows of RW words, the edited orbits' rows from its patch.
template <int RW>
struct LiftGraph {
    const uint16_t *rows, *patch;
    unsigned o0, o1, o2, o3, g, rw;
    __device__ __forceinline__ unsigned width() const { return RW > 0 ? (unsigned)RW : rw; }
    __device__ __forceinline__ unsigned slots() const { return width() - 2u; }
    __device__ __forceinline__ const uint16_t *row(const unsigned v, const unsigned place) const {
        const unsigned o = place & 0xffffu, c = place >> 16;
        if (o == o0 || o == o1 || o == o2 || o == o3)
            return patch + ((o == o0 ? 0u : o == o1 ? 1u : o == o2 ? 2u : 3u) * g + c) * width();
        return rows + (size_t)v * width();
    }
    __device__ __forceinline__ unsigned place(const unsigned v) const {   // orbit | copy << 16
        return __ldg(reinterpret_cast<const unsigned *>(rows + (size_t)v * width()) + width() / 2u - 1u);
    }
    __device__ __forceinline__ unsigned orbit(const unsigned v) const { return place(v) & 0xffffu; }
    // (the base row and the vertex's place are loaded together, the patch only if need be)
    __device__ __forceinline__ unsigned at(const unsigned v, const unsigned i) const {
        const uint16_t *own = rows + (size_t)v * width();
        unsigned u = __ldg(own + i);
        const uint16_t *r = row(v, place(v));
        if (r != own) u = __ldg(r + i);
        return u;
    }
    template <class F>
    __device__ __forceinline__ void each(const unsigned v, F f) const {
        const uint16_t *own = rows + (size_t)v * width();
        const unsigned nq = width() / 8u;
        constexpr unsigned Q = RW > 0 ? RW / 8u : 1u;
        uint4 q[Q];
#pragma unroll
        for (unsigned k = 0; k < Q; ++k) q[k] = __ldg(reinterpret_cast<const uint4 *>(own) + k);
        const uint16_t *r = row(v, RW > 0 ? q[Q - 1u].w : place(v));
        if (RW == 0 || r != own) {
#pragma unroll
            for (unsigned k = 0; k < Q; ++k) q[k] = __ldg(reinterpret_cast<const uint4 *>(r) + k);
        }
        for (unsigned k0 = 0;; k0 += Q) {
#pragma unroll
            for (unsigned k = 0; k < Q; ++k) {
                f(q[k].x & 0xffffu); f(q[k].x >> 16); f(q[k].y & 0xffffu); f(q[k].y >> 16);
                f(q[k].z & 0xffffu); f(q[k].z >> 16);
                if (k0 + k + 1u < nq) { f(q[k].w & 0xffffu); f(q[k].w >> 16); }
            }
            if (RW > 0 || k0 + 1u >= nq) break;
            q[0] = __ldg(reinterpret_cast<const uint4 *>(r) + k0 + 1u);
        }
    }
};

// The same for a part, from its diffs: vertex v of orbit v mod M has the neighbours
// v + diff mod N.  The table (24 KB at m = 1024, d = 12) stays in the L1, where the
// expanded rows (1 MB at N = 32768) do not: a row costs 40 cycles instead of 300, and the
// steps of lift_delta are chains of a few such loads.  DP diffs a row, padded with 0 (0: a
// run-time multiple of 4).
template <int DP>
struct PartGraph {
    const uint16_t *diffs, *patch;
    unsigned o0, o1, o2, o3, N, dp;
    gg::FastDiv div_m;
    __device__ __forceinline__ unsigned slots() const { return DP > 0 ? (unsigned)DP : dp; }
    __device__ __forceinline__ unsigned orbit(const unsigned v) const { return v - div_m.div(v) * div_m.d; }
    __device__ __forceinline__ const uint16_t *row(const unsigned o) const {
        if (o == o0 || o == o1 || o == o2 || o == o3)
            return patch + (o == o0 ? 0u : o == o1 ? 1u : o == o2 ? 2u : 3u) * slots();
        return diffs + o * slots();
    }
    __device__ __forceinline__ unsigned step(const unsigned v, const unsigned df) const {
        const unsigned u = v + df;
        return u - (u >= N ? N : 0u);
    }
    __device__ __forceinline__ unsigned at(const unsigned v, const unsigned i) const {
        return step(v, __ldg(row(orbit(v)) + i));
    }
    template <class F>
    __device__ __forceinline__ void each(const unsigned v, F f) const {
        const uint2 *p = reinterpret_cast<const uint2 *>(row(orbit(v)));
#pragma unroll
        for (unsigned k = 0; k < (DP > 0 ? DP / 4u : dp / 4u); ++k) {
            const uint2 q = __ldg(p + k);
            f(step(v, q.x & 0xffffu)); f(step(v, q.x >> 16)); f(step(v, q.y & 0xffffu)); f(step(v, q.y >> 16));
        }
    }
};

constexpr int kDeltaBlock = 128;

// Follows every listed row of every candidate, a work unit (as many rows as the block's
// shared memory holds) a block at a time: the lookups are random bytes of those rows and
// never leave the SM.  Bound by the latency of the steps (waves and sweeps of a handful of
// entries a row, a block barrier each); blocks a SM hide some of it.
// make_graph(a, cand): the candidate's graph.
template <class Make>
__device__ __forceinline__ void lift_delta_run(const DeltaArgs &a, Make make_graph) {
    extern __shared__ uint4 sm_rows[];
    __shared__ gg::DeltaShared s;
    __shared__ int s_unit;
    const int n_units = a.ctr[0];
    const gg::DeltaBlock b{&s, a.spill + (size_t)blockIdx.x * 3 * gg::kDeltaSpill,
                           (unsigned)__cvta_generic_to_shared(sm_rows), (unsigned)a.pitch};
    const unsigned q = (unsigned)a.pitch / 16u;
    int taken = 0;
    if (threadIdx.x == 0u) taken = atomicAdd(a.ctr + 1, 1);
    for (;;) {
        if (threadIdx.x == 0u) s_unit = taken;
        __syncthreads();
        const int u = s_unit;
        if (u >= n_units) break;
        if (threadIdx.x == 0u) taken = atomicAdd(a.ctr + 1, 1);   // the next one, on the way meanwhile
        const DeltaUnit un = a.units[u];
        const DeltaCand &c = a.cand[un.cand];
        const uint16_t *lst = a.lists + (size_t)un.cand * a.M + un.first;
        for (int slot = 0; slot < un.rows; ++slot) {
            const uint8_t *src = a.dist + (size_t)__ldg(lst + slot) * a.pitch;
            const unsigned dst = b.row((unsigned)slot);
            for (unsigned k = threadIdx.x; k < q; k += kDeltaBlock) gg::delta_cp16(dst + k * 16u, src + k * 16u);
        }
        const auto G = make_graph(c, un.cand);
        const uint3 *ch = a.changes + (size_t)un.cand * 4 * a.g;
        gg::delta_cp_wait();
        gg::delta_rows(G, b, (unsigned)un.rows, (unsigned)(a.ed[un.cand].count * a.g),
                       [&](const unsigned j) { return ch[j]; });
        if (s.overflow) {
            if (threadIdx.x == 0u) a.cand[un.cand].mode = kSearch;
        } else {
            int h = 0;
            const uint32_t *near = a.near + (size_t)un.cand * a.words;
            gg::delta_count(b, [&](const unsigned v) {
                const unsigned o = G.orbit(v);
                return 2u - ((__ldg(near + (o >> 5)) >> (o & 31u)) & 1u);
            }, h);
            if (h) atomicAdd(&a.cand[un.cand].hist[threadIdx.x & 31u], h);
        }
        __syncthreads();   // the next unit overwrites the rows and the list
    }
}

template <int RW>
__global__ void __launch_bounds__(kDeltaBlock) lift_delta(const DeltaArgs a) {
    lift_delta_run(a, [&](const DeltaCand &c, const int k) {
        return LiftGraph<RW>{a.rows, a.patch + (size_t)k * 4 * a.g * a.rw, (unsigned)c.orbit[0], (unsigned)c.orbit[1],
                             (unsigned)c.orbit[2], (unsigned)c.orbit[3], (unsigned)a.g, (unsigned)a.rw};
    });
}

template <int DP>
__global__ void __launch_bounds__(kDeltaBlock) part_delta(const DeltaArgs a) {
    lift_delta_run(a, [&](const DeltaCand &c, const int k) {
        return PartGraph<DP>{a.diffs, a.patch + (size_t)k * 4 * a.dp, (unsigned)c.orbit[0], (unsigned)c.orbit[1],
                             (unsigned)c.orbit[2], (unsigned)c.orbit[3], (unsigned)a.N, (unsigned)a.dp, a.div_m};
    });
}

void *lift_delta_for(int axes, int dp, int rw) {
    if (axes == 1) switch (dp) {
        case 4: return (void *)part_delta<4>;
        case 8: return (void *)part_delta<8>;
        case 12: return (void *)part_delta<12>;
        case 16: return (void *)part_delta<16>;
        default: return (void *)part_delta<0>;
    }
    switch (rw) {
        case 8: return (void *)lift_delta<8>;
        case 16: return (void *)lift_delta<16>;
        default: return (void *)lift_delta<0>;
    }
}

template <bool EXPL>
void *lift_kernel_for_t(int d) {
    switch (d) {
        case 3: return (void *)lift_kernel<3, EXPL>;
        case 4: return (void *)lift_kernel<4, EXPL>;
        case 5: return (void *)lift_kernel<5, EXPL>;
        case 6: return (void *)lift_kernel<6, EXPL>;
        case 8: return (void *)lift_kernel<8, EXPL>;
        case 10: return (void *)lift_kernel<10, EXPL>;
        case 12: return (void *)lift_kernel<12, EXPL>;
        case 16: return (void *)lift_kernel<16, EXPL>;
        default: return (void *)lift_kernel<0, EXPL>;
    }
}
void *lift_kernel_for(int d, bool expl) { return expl ? lift_kernel_for_t<true>(d) : lift_kernel_for_t<false>(d); }

gg_status lfail(gg_status s, const std::string &m) {
    (void)cudaGetLastError();
    gg::set_last_error(m.c_str());
    return s;
}

#define GL_CK(call)                                                                          \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess)                                                               \
            return lfail(e_ == cudaErrorMemoryAllocation ? GG_OUT_OF_MEMORY : GG_CUDA_ERROR, \
                         std::string(#call) + ": " + cudaGetErrorString(e_));                \
    } while (0)

}  // namespace

struct gg_lift {
    int N = 0, M = 0, d = 0, device = 0;
    int axes = 1;                                    // 1 part, 2 piece, 3 box
    int n[3] = {1, 1, 1}, m[3] = {1, 1, 1};          // lifted and orbit size of each axis
    int32_t *d_inv = nullptr;                        // piece / box: [N] representative index or -1
    int32_t *d_adj = nullptr;                        // piece / box: [cap][N][d] candidate adjacency
    int cpc = 0, g_auto = 1, g_max = 0, group = 0;   // group 0: automatic
    int sms = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    int32_t *d_base = nullptr, *d_tab = nullptr;
    gg_lift_edit *d_ed = nullptr, *h_ed = nullptr;
    int cap = 0;                                     // candidates the buffers hold
    uint4 *V = nullptr, *F0 = nullptr, *F1 = nullptr;
    unsigned long long *d_counts = nullptr, *h_counts = nullptr;
    size_t counts_cap = 0;                           // entries
    gg::Ctl *d_ctl = nullptr, *h_ctl = nullptr;
    unsigned long long *d_level_ns = nullptr, *h_level_ns = nullptr;
    int level_ns_n = 0;                              // entries the buffers hold
    int grid = 0;                                    // blocks of the cooperative launch
    int half_ppm = 850000;
    long long wait_ns = 10ll * 1000 * 1000 * 1000;
    bool base_set = false;
    float last_ms = 0.f;
    // moves by change
    bool delta_on = false;                           // the lift is within the limits and the buffers are there
    bool delta_always = false;                       // whatever delta_pays says (GG_LIFT_SEARCH=0)
    int delta_wait = 0;                              // evaluations until it is tried again
    int base_state = 0;                              // distances of the base: 0 not computed, 1 usable, -1 not usable
    long long base_cands = 0;                        // candidates of this base that would have gone by change with them
    int rw = 0, pitch = 0, words = 0, unit_rows = 1, delta_grid = 0;
    unsigned char *d_arena = nullptr, *d_each = nullptr;   // what the pointers below lie in (d_each: per candidate)
    uint4 *d_planes = nullptr;                       // [4][N][cpc]
    uint8_t *d_dist = nullptr;                       // [M][pitch]
    uint16_t *d_rows = nullptr;                      // [N][rw]
    uint16_t *d_diffs = nullptr;                     // part: [M][dp]
    int dp = 0;
    uint32_t *d_ball = nullptr, *d_spill = nullptr;
    int *d_ctr = nullptr;                            // [3]: units made, taken; asymmetric base
    int delta_cap = 0;                               // candidates the next buffers hold
    DeltaCand *d_cand = nullptr, *h_cand = nullptr;
    uint32_t *d_near = nullptr;
    uint16_t *d_lists = nullptr, *d_patch = nullptr;
    uint3 *d_changes = nullptr;
    DeltaUnit *d_units = nullptr;
    unsigned long long base_hist[gg::kDeltaLevels] = {};
};

namespace {

void lift_free(gg_lift *h) {
    if (!h) return;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    cudaFree(h->d_base); cudaFree(h->d_tab); cudaFree(h->d_ed); cudaFreeHost(h->h_ed);
    cudaFree(h->d_inv); cudaFree(h->d_adj);
    cudaFree(h->V); cudaFree(h->F0); cudaFree(h->F1);
    cudaFree(h->d_counts); cudaFreeHost(h->h_counts);
    cudaFree(h->d_level_ns); cudaFreeHost(h->h_level_ns);
    cudaFree(h->d_ctl); cudaFreeHost(h->h_ctl);
    cudaFree(h->d_arena); cudaFree(h->d_each); cudaFreeHost(h->h_cand);
    if (h->ev0) cudaEventDestroy(h->ev0);
    if (h->ev1) cudaEventDestroy(h->ev1);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

gg_status ensure_cand(gg_lift *h, int n) {
    if (n <= h->cap) return GG_OK;
    int cap = std::max(n, 2 * h->cap);
    cudaFree(h->d_tab); cudaFree(h->d_ed); cudaFreeHost(h->h_ed); cudaFree(h->d_adj);
    h->d_tab = nullptr; h->d_ed = nullptr; h->h_ed = nullptr; h->d_adj = nullptr; h->cap = 0;
    GL_CK(cudaMalloc(&h->d_tab, (size_t)cap * h->M * h->d * h->axes * sizeof(int32_t)));
    if (h->axes > 1) GL_CK(cudaMalloc(&h->d_adj, (size_t)cap * h->N * h->d * sizeof(int32_t)));
    GL_CK(cudaMalloc(&h->d_ed, (size_t)cap * sizeof(gg_lift_edit)));
    GL_CK(cudaMallocHost(&h->h_ed, (size_t)cap * sizeof(gg_lift_edit)));
    h->cap = cap;
    return GG_OK;
}

gg_status ensure_counts(gg_lift *h, size_t entries) {
    if (entries <= h->counts_cap) return GG_OK;
    const size_t cap = std::max(entries, 2 * h->counts_cap);
    cudaFree(h->d_counts); cudaFreeHost(h->h_counts);
    h->d_counts = nullptr; h->h_counts = nullptr; h->counts_cap = 0;
    GL_CK(cudaMalloc(&h->d_counts, cap * sizeof(unsigned long long)));
    GL_CK(cudaMallocHost(&h->h_counts, cap * sizeof(unsigned long long)));
    h->counts_cap = cap;
    return GG_OK;
}

std::string lift_tune_key(const gg_lift *h) {
    return gg::tune_key(h->device, "lift", {h->axes, h->n[0], h->n[1], h->n[2], h->m[0], h->m[1], h->m[2], h->d});
}

gg_status alloc_group(gg_lift *h, int groups) {
    cudaFree(h->V); cudaFree(h->F0); cudaFree(h->F1);
    h->V = h->F0 = h->F1 = nullptr;
    h->g_max = 0;
    const size_t bits = (size_t)h->N * h->cpc * groups * sizeof(uint4);
    GL_CK(cudaMalloc(&h->V, bits));
    GL_CK(cudaMalloc(&h->F0, bits));
    GL_CK(cudaMalloc(&h->F1, bits));
    h->g_max = groups;
    return GG_OK;
}

}  // namespace

namespace {

// Moves by change: 16-bit vertex and orbit ids, a distance row within a block's shared
// memory (at 64 KB three blocks a SM), and 1 GiB of distance rows.  The row of an edited
// orbit loses one of its d subtrees, about N / d vertices and more when few others reach
// them as soon; past a size that outgrows the lists (kDeltaList + kDeltaSpill) in nearly every
// candidate, which is then searched as well.  128 candidates, N / (d - 2), by change / searched:
// m = 1000, g = 18, d = 6, 4500: 2739 / 1918 us (125 of 128 searched); m = 1022, g = 22, d = 7, 4497:
// 3884 / 2976; m = 1022, g = 32, d = 10, 4088: 1563 / 3048 (14); m = 1000, g = 24, d = 8, 4000: 1216 /
// 2300 (7); m = 1022, g = 48, d = 12, 4906: 2248 / 4708 (17), g = 52, 5314: 6634 / 4993.  (Which side of
// the line a lift near it falls turns on its diameter, too: gg_lift_eval looks.)
constexpr size_t kDeltaRowBytes = 24 * 1024;   // rows of a block, when one is smaller
constexpr size_t kDeltaMostBytes = 64 * 1024;  // one row of the largest lift
constexpr int delta_most(int d) { return (d >= 12 ? 5000 : 4300) * (d - 2); }   // vertices
bool delta_fits(const gg_lift *h) {
    const size_t pitch = ((size_t)h->N + 15) / 16 * 16;
    return h->N <= 65536 && h->M <= 65535 && h->N / h->M <= 65535 && pitch * h->M <= (1ull << 30) &&
           (h->delta_always || h->N <= delta_most(std::min(h->d, 64)));
}

// Whether a population of n goes by change.  Microseconds, fits over 90 lifts (N = 268 to
// 31062, d = 4 to 12): a searched candidate takes `each`, one by change about a third of that; by
// change a population takes `more` longer before its first candidate (its waves are chains,
// longer at small degrees and with many copies edited at once); the distances of a new base
// take 135 and three searched candidates.  They are worth it once the candidates seen on the
// base would have paid for them: 32 candidates on a new base are searched at m = 500, g = 12, d
// = 6 (148 us, 314 by change) and go by change at m = 1024, g = 32, d = 12 (849 / 529).  Where
// both ways take as long, by this and measured: m = 992, g = 12, d = 6: 38 and 50 candidates;
// 752, 19, 7: 45, 47; 584, 6, 11: 98, 86; 558, 5, 6: 111, 126; 956, 32, 12: 21, 13; with the
// distances there 12, 10; 17, 12; 17, 8 at most; 20, 15; 7, 8 at most.
bool delta_pays(gg_lift *h, const int n) {
    if (h->delta_always) return true;
    const double each = 1.0 + 88e-6 * (double)h->N * h->cpc, k = h->d - 2;
    const double more = 40.0 + 0.012 * std::max(h->N / h->M - 4, 0) * h->N / (k * k);
    const double next = 1.5 + more / each;
    if (n < next) return false;
    h->base_cands += n;
    return h->base_state == 1 || (double)h->base_cands >= next + 4.0 + 190.0 / each;
}

// Buffers of the moves by change.  Without them candidates are searched.
void delta_open(gg_lift *h) {
    const size_t pitch = ((size_t)h->N + 15) / 16 * 16;
    h->pitch = (int)pitch;
    h->rw = (h->d + 2 + 7) / 8 * 8;
    h->dp = (h->d + 3) / 4 * 4;
    h->words = (h->M + 31) / 32;
    const size_t smem = std::max(kDeltaRowBytes, pitch);
    h->unit_rows = (int)std::min<size_t>(gg::kDeltaRows, smem / pitch);
    int per_sm = 0;
    void *k = lift_delta_for(h->axes, h->dp, h->rw);
    // (the limit belongs to the kernel, which handles of other sizes launch too)
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDeltaMostBytes);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kDeltaBlock, smem);
    h->delta_grid = per_sm * h->sms;
    if (e == cudaSuccess && per_sm < 1) e = cudaErrorInvalidConfiguration;
    // one allocation for all of them
    size_t at = 0;
    auto part = [&](size_t bytes) {
        const size_t o = at;
        at += (bytes + 255) / 256 * 256;
        return o;
    };
    const size_t o_planes = part(4 * (size_t)h->N * h->cpc * sizeof(uint4)), o_dist = part(pitch * h->M),
                 o_rows = part((size_t)h->N * h->rw * sizeof(uint16_t)),
                 o_diffs = part((size_t)h->M * h->dp * sizeof(uint16_t)),
                 o_ball = part((size_t)h->M * h->words * sizeof(uint32_t)),
                 o_spill = part((size_t)h->delta_grid * 3 * gg::kDeltaSpill * sizeof(uint32_t)), o_ctr = part(3 * sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc(&h->d_arena, at);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return;
    }
    h->d_planes = reinterpret_cast<uint4 *>(h->d_arena + o_planes);
    h->d_dist = h->d_arena + o_dist;
    h->d_rows = reinterpret_cast<uint16_t *>(h->d_arena + o_rows);
    h->d_diffs = reinterpret_cast<uint16_t *>(h->d_arena + o_diffs);
    h->d_ball = reinterpret_cast<uint32_t *>(h->d_arena + o_ball);
    h->d_spill = reinterpret_cast<uint32_t *>(h->d_arena + o_spill);
    h->d_ctr = reinterpret_cast<int *>(h->d_arena + o_ctr);
    h->delta_on = true;
}

// Per-candidate buffers of the moves by change; false: not enough memory.
bool delta_ensure(gg_lift *h, int n) {
    if (n <= h->delta_cap) return true;
    const size_t cap = (size_t)std::max(n, 2 * h->delta_cap), g = (size_t)h->N / h->M;
    const size_t units = (size_t)(h->M + h->unit_rows - 1) / h->unit_rows;
    cudaFree(h->d_each); cudaFreeHost(h->h_cand);
    h->d_each = nullptr;
    h->h_cand = nullptr;
    h->delta_cap = 0;
    size_t at = 0;
    auto part = [&](size_t bytes) {
        const size_t o = at;
        at += (bytes + 255) / 256 * 256;
        return o;
    };
    const size_t o_cand = part(cap * sizeof(DeltaCand)), o_near = part(cap * h->words * sizeof(uint32_t)),
                 o_lists = part(cap * h->M * sizeof(uint16_t)),
                 o_patch = part(cap * 4 * (h->axes == 1 ? h->dp : g * h->rw) * sizeof(uint16_t)),
                 o_changes = part(cap * 4 * g * sizeof(uint3)), o_units = part(cap * units * sizeof(DeltaUnit));
    cudaError_t e = cudaMalloc(&h->d_each, at);
    if (e == cudaSuccess) e = cudaMallocHost(&h->h_cand, cap * sizeof(DeltaCand));
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    h->d_cand = reinterpret_cast<DeltaCand *>(h->d_each + o_cand);
    h->d_near = reinterpret_cast<uint32_t *>(h->d_each + o_near);
    h->d_lists = reinterpret_cast<uint16_t *>(h->d_each + o_lists);
    h->d_patch = reinterpret_cast<uint16_t *>(h->d_each + o_patch);
    h->d_changes = reinterpret_cast<uint3 *>(h->d_each + o_changes);
    h->d_units = reinterpret_cast<DeltaUnit *>(h->d_each + o_units);
    h->delta_cap = (int)cap;
    return true;
}

// A handle for a lift of `axes` axes: lifted sizes n, orbit sizes m.
gg_status lift_open(int axes, const int n_in[3], const int m_in[3], int degree, int device, gg_lift **out) {
    if (!out) return lfail(GG_BAD_ARG, "null argument");
    *out = nullptr;
    long long N = 1, M = 1;
    for (int j = 0; j < axes; ++j) {
        if (m_in[j] < 1 || n_in[j] < 1 || m_in[j] > n_in[j] || n_in[j] % m_in[j] != 0)
            return lfail(GG_BAD_ARG, "every lifted size must be a positive multiple of its orbit size");
        N *= n_in[j];
        M *= m_in[j];
    }
    if (N < 2 || N >= (1ll << 30) || degree < 1 || degree > 4096)
        return lfail(GG_BAD_ARG, "need 2 <= N < 2^30 vertices and 1 <= degree <= 4096");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
        return lfail(GG_NO_DEVICE, "no such CUDA device");
    gg_lift *h = new gg_lift();
    h->axes = axes;
    for (int j = 0; j < axes; ++j) { h->n[j] = n_in[j]; h->m[j] = m_in[j]; }
    h->N = (int)N; h->M = (int)M; h->d = degree; h->device = device;
    h->cpc = (h->M + 127) / 128;
    auto fail = [&](gg_status s) { lift_free(h); return s; };
    if (cudaSetDevice(device) != cudaSuccess) return fail(lfail(GG_NO_DEVICE, "cudaSetDevice failed"));
    int l2 = 0, coop = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lift_kernel_for(degree, axes > 1), kLiftBlock, 0) !=
            cudaSuccess)
        return fail(lfail(GG_CUDA_ERROR, "device query failed"));
    if (!coop || per_sm < 1) return fail(lfail(GG_CUDA_ERROR, "cooperative launch unavailable"));
    h->grid = per_sm * h->sms;
    // one candidate's round share: three bitsets of N * cpc uint4
    // (half the L2: lines gathered from both dies' SMs are held in both halves;
    // at m=1024, g=32, d=12 a sweep of 2-8 candidates per round put the optimum at 5)
    const double per_cand = 3.0 * h->N * h->cpc * 16.0;
    const int fit = (int)std::max(1.0, 0.5 * l2 / per_cand);
    // items N * W must stay below 2^31
    const long long by_items = std::max(1ll, (1ll << 31) / ((long long)h->N * h->cpc));
    h->g_auto = (int)std::min<long long>({(long long)fit, (long long)kMaxGroup, by_items});
    {
        // a group recorded by gg_lift_autotune for this lift shape on this kind of GPU
        std::vector<int> tuned;
        if (gg::tune_get(lift_tune_key(h), &tuned) && !tuned.empty() && tuned[0] >= 1 &&
            tuned[0] <= kMaxGroup && tuned[0] <= by_items)
            h->g_auto = tuned[0];
    }
    cudaError_t e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreate(&h->ev0);
    if (e == cudaSuccess) e = cudaEventCreate(&h->ev1);
    if (e == cudaSuccess) e = cudaMalloc(&h->d_base, (size_t)h->M * degree * axes * sizeof(int32_t));
    if (e == cudaSuccess) e = cudaMalloc(&h->d_ctl, sizeof(gg::Ctl));
    if (e == cudaSuccess) e = cudaMallocHost(&h->h_ctl, sizeof(gg::Ctl));
    if (e == cudaSuccess && axes > 1) {
        // representatives: the corner tile, numbered like the table's rows
        // (cpuASPLpiece.cpp:199-200, cpuASPLbox.cpp:133-134)
        std::vector<int32_t> inv((size_t)h->N, -1);
        const int nz = h->n[2], ny = h->n[1];
        for (int x = 0; x < h->m[0]; ++x)
            for (int y = 0; y < h->m[1]; ++y)
                for (int z = 0; z < h->m[2]; ++z)
                    inv[((size_t)x * ny + y) * nz + z] = (x * h->m[1] + y) * h->m[2] + z;
        e = cudaMalloc(&h->d_inv, inv.size() * sizeof(int32_t));
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(h->d_inv, inv.data(), inv.size() * sizeof(int32_t), cudaMemcpyHostToDevice, h->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    }
    if (e != cudaSuccess)
        return fail(lfail(e == cudaErrorMemoryAllocation ? GG_OUT_OF_MEMORY : GG_CUDA_ERROR,
                          cudaGetErrorString(e)));
    // bitsets for the automatic group (a larger group set later reallocates)
    const gg_status s = alloc_group(h, h->g_auto);
    if (s != GG_OK) return fail(s);
    const char *search = std::getenv("GG_LIFT_SEARCH");   // 1: search every candidate, 0: none that can go by change
    h->delta_always = search && std::atoi(search) == 0;
    if (!(search && !h->delta_always) && delta_fits(h)) delta_open(h);
    *out = h;
    return GG_OK;
}

// Searches the candidates whose edits are in h->h_ed[0 .. n_cand); with `planes`, n_cand is
// 1 and the distance planes are written too.
gg_status lift_search(gg_lift *h, int n_cand, int max_levels, gg_cand_result *out, uint4 *planes = nullptr) {
    gg_status s;
    // Count rows for the first kFirstLevels levels; a population where some candidate
    // still finds pairs there (a lift of very large diameter) runs again with rows
    // for the full cap, so the buffers stay small for the usual diameters.
    const int ml_full = max_levels > 0 ? std::min(max_levels, h->N) : h->N;
    for (int ml = std::min(ml_full, kFirstLevels);; ml = ml_full) {
        s = ensure_counts(h, (size_t)(ml + 1) * n_cand);
        if (s != GG_OK) return s;
        if (ml + 1 > h->level_ns_n) {
            cudaFree(h->d_level_ns); cudaFreeHost(h->h_level_ns);
            h->d_level_ns = nullptr; h->h_level_ns = nullptr; h->level_ns_n = 0;
            GL_CK(cudaMalloc(&h->d_level_ns, (size_t)(ml + 1) * sizeof(unsigned long long)));
            GL_CK(cudaMallocHost(&h->h_level_ns, (size_t)(ml + 1) * sizeof(unsigned long long)));
            h->level_ns_n = ml + 1;
        }
        const int G = std::min(h->group ? h->group : h->g_auto, n_cand);
        const cudaStream_t st = h->stream;
        GL_CK(cudaMemcpyAsync(h->d_ed, h->h_ed, (size_t)n_cand * sizeof(gg_lift_edit), cudaMemcpyHostToDevice, st));
        GL_CK(cudaMemsetAsync(h->d_ctl, 0, sizeof(gg::Ctl), st));
        GL_CK(cudaMemsetAsync(h->d_counts, 0, (size_t)std::min(ml + 1, 2) * n_cand * sizeof(unsigned long long), st));
        GL_CK(cudaEventRecord(h->ev0, st));
        const long long tab_n = (long long)n_cand * h->M * h->d;
        lift_tables<<<(int)std::min<long long>((tab_n + 255) / 256, (long long)h->sms * 16), 256, 0, st>>>(
            h->d_base, h->d_ed, n_cand, h->M, h->d, h->axes, h->d_tab);
        GL_CK(cudaGetLastError());
        if (h->axes > 1) {
            const long long rows_n = (long long)n_cand * h->N;
            lift_expand<<<(int)std::min<long long>((rows_n + 255) / 256, (long long)h->sms * 16), 256, 0, st>>>(
                h->d_tab, n_cand, h->M, h->d, h->axes, h->n[0], h->n[1], h->n[2], h->m[0], h->m[1], h->m[2], h->d_adj);
            GL_CK(cudaGetLastError());
        }
        LiftArgs a{};
        a.tab = h->d_tab;
        a.adj = h->d_adj;
        a.inv = h->d_inv;
        a.N = h->N; a.M = h->M; a.d = h->d; a.K = n_cand; a.G = G; a.cpc = h->cpc; a.W = G * h->cpc;
        a.V = h->V; a.F0 = h->F0; a.F1 = h->F1;
        a.counts = h->d_counts;
        a.max_levels = ml;
        const unsigned threads = (unsigned)h->grid * kLiftBlock;
        if ((unsigned)a.W > threads) return lfail(GG_BAD_ARG, "more chunk columns than threads: lower the group");
        a.cols_threads = threads / (unsigned)a.W * (unsigned)a.W;
        a.vstep = a.cols_threads / (unsigned)a.W;
        a.half_ppm = h->half_ppm;
        a.level_ns = h->d_level_ns;
        a.ctl = h->d_ctl;
        a.wait_ns = h->wait_ns;
        a.planes = planes;
        a.expected = (unsigned)h->grid;
        GL_CK(cudaMemsetAsync(h->d_level_ns, 0, (size_t)(ml + 1) * sizeof(unsigned long long), st));
        void *args[] = {&a};
        GL_CK(cudaLaunchCooperativeKernel(lift_kernel_for(h->d, h->axes > 1), dim3(h->grid), dim3(kLiftBlock), args, 0,
                                          st));
        GL_CK(cudaEventRecord(h->ev1, st));
        GL_CK(cudaMemcpyAsync(h->h_ctl, h->d_ctl, sizeof(gg::Ctl), cudaMemcpyDeviceToHost, st));
        GL_CK(cudaStreamSynchronize(st));
        if (h->h_ctl->err) return lfail(GG_TIMEOUT, "grid barrier wait exceeded the limit");
        const int lr = std::min(h->h_ctl->levels_run, ml);
        GL_CK(cudaMemcpyAsync(h->h_counts, h->d_counts, (size_t)(lr + 1) * n_cand * sizeof(unsigned long long),
                              cudaMemcpyDeviceToHost, st));
        GL_CK(cudaMemcpyAsync(h->h_level_ns, h->d_level_ns, (size_t)(lr + 1) * sizeof(unsigned long long),
                              cudaMemcpyDeviceToHost, st));
        GL_CK(cudaStreamSynchronize(st));
        GL_CK(cudaEventElapsedTime(&h->last_ms, h->ev0, h->ev1));
        const unsigned long long all = (unsigned long long)h->M * (unsigned long long)h->N;
        for (int k = 0; k < n_cand; ++k) {
            unsigned long long tot = 0, reach = (unsigned long long)h->M;
            int lev = 0;
            for (int L = 1; L <= lr; ++L) {
                const unsigned long long c = h->h_counts[(size_t)L * n_cand + k];
                if (!c) continue;
                tot += (unsigned long long)L * c;
                reach += c;
                lev = L;
            }
            const bool capped = lev == ml && reach < all;
            out[k] = gg_cand_result{tot, reach, lev, (!capped && reach == all) ? 1 : 0};
        }
        bool again = false;
        for (int k = 0; k < n_cand && ml < ml_full; ++k)
            again |= out[k].levels == ml && out[k].reached < all;
        if (!again) break;
    }
    return GG_OK;
}


// The base's distances, rows and balls.  base_state = 1 when candidates can be scored by
// change: a symmetric, connected base of diameter at most 15.
gg_status delta_base(gg_lift *h) {
    h->base_state = -1;
    const cudaStream_t st = h->stream;
    LiftAxes ax{h->axes, {h->n[0], h->n[1], h->n[2]}, {h->m[0], h->m[1], h->m[2]}};
    const int blocks = h->sms * 8;
    GL_CK(cudaMemsetAsync(h->d_planes, 0, 4 * (size_t)h->N * h->cpc * sizeof(uint4), st));
    GL_CK(cudaMemsetAsync(h->d_ctr, 0, 3 * sizeof(int), st));
    delta_symmetry<<<std::min(blocks, (h->M * h->d + 255) / 256), 256, 0, st>>>(h->d_base, ax, h->M, h->d, h->d_ctr + 2);
    delta_rows_kernel<<<std::min(blocks, (h->N + 127) / 128), 128, 0, st>>>(h->d_base, ax, h->N, h->d, h->rw, h->d_rows);
    if (h->axes == 1)
        delta_diffs_kernel<<<std::min(blocks, (h->M * h->dp + 255) / 256), 256, 0, st>>>(h->d_base, h->M, h->d, h->dp, h->d_diffs);
    GL_CK(cudaGetLastError());
    h->h_ed[0] = gg_lift_edit{};   // the base itself
    gg_cand_result r{};
    gg_status s = lift_search(h, 1, 16, &r, h->d_planes);
    if (s != GG_OK) return s;
    int asym = 0;
    GL_CK(cudaMemcpyAsync(&asym, h->d_ctr + 2, sizeof(int), cudaMemcpyDeviceToHost, st));
    GL_CK(cudaStreamSynchronize(st));
    if (asym || !r.connected || r.levels > 15 || r.levels < 1) return GG_OK;
    for (int L = 0; L < gg::kDeltaLevels; ++L)
        h->base_hist[L] = L == 0 ? (unsigned long long)h->M : L <= r.levels ? h->h_counts[L] : 0ull;
    delta_bytes<<<dim3((unsigned)((h->N + 127) / 128), (unsigned)h->cpc), 128, 0, st>>>(h->d_planes, h->N, h->M, h->cpc,
                                                                                h->d_dist, h->pitch);
    delta_balls<<<h->M, 256, (size_t)h->words * 4, st>>>(h->d_dist, h->pitch, h->N, h->d_rows, h->rw, h->words,
                                                         (unsigned)(r.levels - 1) / 2u, h->d_ball);
    GL_CK(cudaGetLastError());
    h->base_state = 1;
    return GG_OK;
}

// Scores the candidates in h->h_ed[0 .. n_cand) by change; `left` gets the ones that have
// to be searched.
gg_status delta_eval(gg_lift *h, int n_cand, int max_levels, gg_cand_result *out, std::vector<int> &left) {
    const cudaStream_t st = h->stream;
    DeltaArgs a{};
    a.ax = LiftAxes{h->axes, {h->n[0], h->n[1], h->n[2]}, {h->m[0], h->m[1], h->m[2]}};
    a.N = h->N; a.M = h->M; a.d = h->d; a.g = h->N / h->M; a.K = n_cand;
    a.table = h->d_base;
    a.ed = h->d_ed;
    a.rows = h->d_rows; a.rw = h->rw;
    a.diffs = h->d_diffs; a.dp = h->dp;
    a.div_m = gg::FastDiv((uint32_t)h->M);
    a.dist = h->d_dist; a.pitch = h->pitch;
    a.ball = h->d_ball; a.words = h->words;
    a.cand = h->d_cand;
    a.near = h->d_near;
    a.lists = h->d_lists;
    a.changes = h->d_changes;
    a.patch = h->d_patch;
    a.units = h->d_units;
    a.ctr = h->d_ctr;
    a.unit_rows = h->unit_rows;
    a.spill = h->d_spill;
    GL_CK(cudaMemcpyAsync(h->d_ed, h->h_ed, (size_t)n_cand * sizeof(gg_lift_edit), cudaMemcpyHostToDevice, st));
    GL_CK(cudaMemsetAsync(h->d_ctr, 0, 2 * sizeof(int), st));
    GL_CK(cudaEventRecord(h->ev0, st));
    lift_select<<<n_cand, 128, 0, st>>>(a);
    GL_CK(cudaGetLastError());
    void *args[] = {&a};
    GL_CK(cudaLaunchKernel(lift_delta_for(h->axes, h->dp, h->rw), dim3(h->delta_grid), dim3(kDeltaBlock), args,
                           std::max(kDeltaRowBytes, (size_t)h->pitch), st));
    GL_CK(cudaEventRecord(h->ev1, st));
    GL_CK(cudaMemcpyAsync(h->h_cand, h->d_cand, (size_t)n_cand * sizeof(DeltaCand), cudaMemcpyDeviceToHost, st));
    GL_CK(cudaStreamSynchronize(st));
    GL_CK(cudaEventElapsedTime(&h->last_ms, h->ev0, h->ev1));
    if (h->h_ctl) h->h_ctl->levels_run = 0;   // no level times of this evaluation
    const unsigned long long all = (unsigned long long)h->M * (unsigned long long)h->N;
    const int cap = max_levels > 0 ? max_levels : h->N;
    for (int k = 0; k < n_cand; ++k) {
        const DeltaCand &c = h->h_cand[k];
        if (c.mode != kByChange) {
            left.push_back(k);
            continue;
        }
        unsigned long long tot = 0, reach = 0;
        int lev = 0;
        for (int L = 0; L < (int)gg::kDeltaInf && L <= cap; ++L) {
            const unsigned long long n = h->base_hist[L] + (unsigned long long)(long long)c.hist[L];
            tot += (unsigned long long)L * n;
            reach += n;
            if (n) lev = L;
        }
        out[k] = gg_cand_result{tot, reach, lev, reach == all ? 1 : 0};
    }
    return GG_OK;
}

}  // namespace

extern "C" {

gg_status gg_lift_create(int N, int M, int degree, int device, gg_lift **out) {
    const int n[3] = {N, 1, 1}, m[3] = {M, 1, 1};
    return lift_open(1, n, m, degree, device, out);
}

gg_status gg_lift_create_piece(int Nx, int Ny, int Mx, int My, int degree, int device, gg_lift **out) {
    const int n[3] = {Nx, Ny, 1}, m[3] = {Mx, My, 1};
    return lift_open(2, n, m, degree, device, out);
}

gg_status gg_lift_create_box(int Nx, int Ny, int Nz, int Mx, int My, int Mz, int degree, int device,
                             gg_lift **out) {
    const int n[3] = {Nx, Ny, Nz}, m[3] = {Mx, My, Mz};
    return lift_open(3, n, m, degree, device, out);
}

gg_status gg_lift_set_base(gg_lift *h, const int32_t *table) {
    if (!h || !table) return lfail(GG_BAD_ARG, "null argument");
    std::vector<int32_t> nd((size_t)h->M * h->d * h->axes);
    for (size_t k = 0; k < nd.size(); ++k) {
        const long long n = h->n[k % h->axes];
        nd[k] = (int32_t)((((long long)table[k] % n) + n) % n);
    }
    GL_CK(cudaSetDevice(h->device));
    GL_CK(cudaMemcpyAsync(h->d_base, nd.data(), nd.size() * sizeof(int32_t), cudaMemcpyHostToDevice, h->stream));
    GL_CK(cudaStreamSynchronize(h->stream));
    h->base_set = true;
    h->base_state = 0;
    h->base_cands = 0;
    return GG_OK;
}

gg_status gg_lift_set_group(gg_lift *h, int group) {
    if (!h || group < 0 || group > kMaxGroup) return lfail(GG_BAD_ARG, "group must be in [0, 32]");
    if (group > 0 && (long long)h->N * h->cpc * group >= (1ll << 31))
        return lfail(GG_BAD_ARG, "group too large for this lift");
    const int need = group ? group : h->g_auto;
    if (need > h->g_max) {
        GL_CK(cudaSetDevice(h->device));
        GL_CK(cudaStreamSynchronize(h->stream));
        const gg_status s = alloc_group(h, need);
        if (s != GG_OK) return s;
    }
    h->group = group;
    return GG_OK;
}

gg_status gg_lift_autotune(gg_lift *h, int n_cand, const gg_lift_edit *edits, int max_levels, int trials,
                           int *best_group, double *best_ms) {
    if (!h || n_cand < 1 || !edits || trials < 1 || max_levels < 0) return lfail(GG_BAD_ARG, "bad arguments");
    if (!h->base_set) return lfail(GG_BAD_ARG, "no base table set");
    std::vector<gg_cand_result> out((size_t)n_cand);
    const int keep = h->group;
    int best = 0;
    double best_t = 1e300;
    const long long by_items = std::max(1ll, (1ll << 31) / ((long long)h->N * h->cpc));
    for (int G = 1; G <= std::min<long long>({(long long)kMaxGroup, by_items, (long long)n_cand}); ++G) {
        if (G > 12 && G != 16 && G != 24 && G != 32) continue;
        gg_status s = gg_lift_set_group(h, G);
        if (s == GG_OUT_OF_MEMORY) { (void)cudaGetLastError(); break; }
        if (s != GG_OK) return s;
        s = gg_lift_eval(h, n_cand, edits, max_levels, out.data());  // warm
        if (s == GG_BAD_ARG) break;  // more chunk columns than threads: larger groups fail too
        if (s != GG_OK) return s;
        double t = 1e300;
        for (int k = 0; k < trials; ++k) {
            s = gg_lift_eval(h, n_cand, edits, max_levels, out.data());
            if (s != GG_OK) return s;
            t = std::min(t, (double)h->last_ms);
        }
        if (t < best_t) { best_t = t; best = G; }
    }
    if (!best) {
        gg_lift_set_group(h, keep);
        return lfail(GG_OUT_OF_MEMORY, "no group fits");
    }
    gg::tune_put(lift_tune_key(h), {best});
    h->g_auto = best;
    gg_status s = gg_lift_set_group(h, 0);
    if (s != GG_OK) return s;
    if (best_group) *best_group = best;
    if (best_ms) *best_ms = best_t;
    return GG_OK;
}

gg_status gg_lift_group(gg_lift *h, int *group) {
    if (!h || !group) return lfail(GG_BAD_ARG, "null argument");
    *group = h->group ? h->group : h->g_auto;
    return GG_OK;
}

gg_status gg_lift_eval(gg_lift *h, int n_cand, const gg_lift_edit *edits, int max_levels,
                       gg_cand_result *out) {
    if (!h || n_cand < 0 || (n_cand && (!edits || !out)) || max_levels < 0)
        return lfail(GG_BAD_ARG, "bad arguments");
    if (!h->base_set) return lfail(GG_BAD_ARG, "no base table set");
    if (n_cand == 0) return GG_OK;
    if (h->g_max < 1) return lfail(GG_OUT_OF_MEMORY, "bitsets were not allocated");
    GL_CK(cudaSetDevice(h->device));
    gg_status s = ensure_cand(h, n_cand);
    if (s != GG_OK) return s;
    for (int k = 0; k < n_cand; ++k) {
        const gg_lift_edit &q = edits[k];
        if (q.count < 0 || q.count > 4) return lfail(GG_BAD_ARG, "edit count must be in [0, 4]");
        gg_lift_edit &o = h->h_ed[k];
        o = gg_lift_edit{};
        o.count = q.count;
        for (int j = 0; j < q.count; ++j) {
            if (q.row[j] < 0 || q.row[j] >= h->M || q.slot[j] < 0 || q.slot[j] >= h->d)
                return lfail(GG_BAD_ARG, "edit slot outside the table");
            o.row[j] = q.row[j];
            o.slot[j] = q.slot[j];
            for (int c = 0; c < h->axes; ++c) {
                const long long n = h->n[c];
                o.diff[j][c] = (int32_t)((((long long)q.diff[j][c] % n) + n) % n);
            }
        }
    }
    const bool can = h->delta_on && h->group == 0 && h->base_state >= 0;
    if (can && h->delta_wait > 0) {
        --h->delta_wait;
    } else if (can && delta_pays(h, n_cand) && delta_ensure(h, n_cand)) {
        if (h->base_state == 0) {
            const gg_lift_edit first = h->h_ed[0];
            s = delta_base(h);
            if (s != GG_OK) return s;
            h->h_ed[0] = first;
            if (h->base_state < 0 && !h->delta_always) h->delta_wait = 63;   // (the next bases are often like it)
        }
        if (h->base_state == 1) {
            std::vector<int> left;
            s = delta_eval(h, n_cand, max_levels, out, left);
            if (s != GG_OK || left.empty()) return s;
            // the rest is searched
            for (size_t i = 0; i < left.size(); ++i) h->h_ed[i] = h->h_ed[left[i]];
            std::vector<gg_cand_result> res(left.size());
            const float ms = h->last_ms;
            s = lift_search(h, (int)left.size(), max_levels, res.data());
            if (s != GG_OK) return s;
            // (a search: 80 us and a time a candidate; when they are an eighth or more and all of
            // them would have taken less, the next populations are searched)
            const float each = std::max(h->last_ms - 0.08f, 0.f) / (float)left.size();
            if (left.size() * 8 > (size_t)n_cand && ms + h->last_ms > 0.08f + each * (float)n_cand && !h->delta_always)
                h->delta_wait = 63;
            h->last_ms += ms;
            for (size_t i = 0; i < left.size(); ++i) out[left[i]] = res[i];
            return GG_OK;
        }
    }
    return lift_search(h, n_cand, max_levels, out);
}

gg_status gg_lift_set_half_ppm(gg_lift *h, int half_ppm) {
    if (!h || half_ppm < 0 || half_ppm > 1000000) return lfail(GG_BAD_ARG, "half_ppm must be in [0, 1e6]");
    h->half_ppm = half_ppm;
    return GG_OK;
}

gg_status gg_lift_last_level_ns(gg_lift *h, uint64_t *ns, int n) {
    if (!h || !ns || n < 0) return lfail(GG_BAD_ARG, "bad arguments");
    const int lr = h->h_ctl ? h->h_ctl->levels_run : 0;
    for (int i = 0; i < n; ++i) ns[i] = (i <= lr && i < h->level_ns_n && h->h_level_ns) ? h->h_level_ns[i] : 0;
    return GG_OK;
}

gg_status gg_lift_last_ms(gg_lift *h, double *ms) {
    if (!h || !ms) return lfail(GG_BAD_ARG, "null argument");
    *ms = h->last_ms;
    return GG_OK;
}

gg_status gg_lift_destroy(gg_lift *h) {
    lift_free(h);
    return GG_OK;
}

}  // extern "C"
