// gg_engine.cu -- host side of the engine and the C ABI declared in include/gg.h.
//
// One gg_engine owns every device and pinned buffer of one calculator, sized at
// construction from its form and dimensions, the way the reference calculators
// size theirs in their constructors (cudaASPLconv.cu:122-137,
// cudaASPLgraph.cu:114-127).  An evaluation is:
//   H2D of the packed table -> expand_kernel (lifted forms) -> direct_kernel (small
//   ones), balls and sweep_kernel (every vertex, or a lift's orbits), or the general
//   bfs_batch_kernel over every source batch -> one D2H of the level counters
//   -> exact host fold into gg_result -> the reference's return convention.
// There is no per-level host round trip: the level loop, its termination test
// and the connectivity test live on the device.
#include "gg.h"
#include "gg_kernels.cuh"
#include "gg_direct.cuh"
#include "gg_sweep.cuh"
#include "gg_internal.h"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

using gg::BfsArgs;
using gg::Ctl;
using gg::ExpandArgs;
using gg::FastDiv;

namespace {

thread_local std::string g_err;

gg_status fail(gg_status s, const std::string &msg) {
    g_err = msg;
    return s;
}

#define GG_CK(call)                                                                     \
    do {                                                                                \
        cudaError_t e_ = (call);                                                        \
        if (e_ != cudaSuccess) {                                                        \
            (void)cudaGetLastError();                                                   \
            return fail(e_ == cudaErrorMemoryAllocation ? GG_OUT_OF_MEMORY : GG_CUDA_ERROR, \
                        std::string(#call) + ": " + cudaGetErrorString(e_));            \
        }                                                                               \
    } while (0)

enum Form { FORM_GRAPH = 0, FORM_PART = 1, FORM_PIECE = 2, FORM_BOX = 3 };

constexpr int kBeamerRows = 1000000;   // cudaASPLbeamer.cu:10-12
constexpr int kBeamerLevels = 7;       // cudaASPLbeamer.cu:17
constexpr int kSentinel = 100000000;   // cudaASPLconv.cu:207

int env_int(const char *name, int dflt) {
    const char *s = std::getenv(name);
    return (s && *s) ? std::atoi(s) : dflt;
}

// Host-side fault injection for the failure-path tests (GG_FAULT_INJECT):
//   "barrier" -- the grid barrier waits for one block more than is launched, so
//                its bounded wait runs out and the call returns GG_TIMEOUT;
//   "alloc"   -- engine creation reports an allocation failure;
//   "launch"  -- the BFS launch reports a CUDA error before anything is enqueued;
//   "rows"    -- no memory for the rows of all batches (vall_room);
//   "more_rows" -- no memory for more of them once there are some.
// Nothing here faults, traps or hangs the GPU.
bool fault(const char *what) {
    const char *s = std::getenv("GG_FAULT_INJECT");
    return s && std::strcmp(s, what) == 0;
}

}  // namespace

namespace gg {
// Shared with the other translation units of the library (not exported).
__attribute__((visibility("hidden"))) void set_last_error(const char *msg) { g_err = msg; }
}  // namespace gg

// What a captured evaluation depends on (see run_eval).
struct EvalKey {
    const void *table, *status, *bitsets, *inv, *planes;
    int s0, ns, cap;
    bool wvc, want_ns, sweep;
    bool operator==(const EvalKey &o) const {
        return table == o.table && status == o.status && bitsets == o.bitsets && inv == o.inv &&
               planes == o.planes && s0 == o.s0 && ns == o.ns && cap == o.cap && wvc == o.wvc &&
               want_ns == o.want_ns && sweep == o.sweep;
    }
};

struct gg_engine {
    int form = FORM_PART;
    int device = 0;
    int N = 0, M = 0, d = 0, rows = 0;
    int dims[6] = {0, 0, 0, 0, 0, 0};    // Nx Ny Nz Mx My Mz
    uint64_t scale = 1;
    size_t table_elems = 0;
    std::vector<int32_t> reps;           // source vertex ids, in source order

    // plan
    int batch_bits = 0;                  // sources per batch (multiple of 128)
    int nC = 0;                          // uint4 chunks per row
    uint32_t items = 0;
    int grid = 0;
    int dense_w_ppm = 100;               // level-mode thresholds (see bfs_batch_kernel)
    int dense_r_ppm = 4000;
    int full_skip_ppm = 995000;
    int split_ppm = 850000;
    int push_ppm = 300;                  // push (top-down) levels below this frontier share
    int push_min_items = 1 << 20;        // ... on bitsets of at least this many chunks
    int adj_smem_rows = 0;               // shared-memory adjacency slice (rows per block)
    size_t smem_bytes = 0;
    int bps_cap = 0;                     // resident blocks per SM (0: as many as fit)
    int walk_pref = -1;                  // walk depth: -1 automatic, 0 off, K > 0 forced
    int walk_K = 0;                      // levels computed by the walk pass (0: off)
    bool walk_auto = true;               // ... chosen by walk_levels, not asked for
    int walk_vpull = 1;                  // levels after the walk pull visited sets (GG_VPULL=0: frontiers)
    int walk_own_skip = 1;               // dense ones skip own chunks on tables without one-way entries (GG_OWN_SKIP)
    int walk_third = 1;                  // after the walk of all batches, levels alternate V and F0 (GG_WALK_THIRD)
    int walk_rpg = 1;                    // rows per walk group
    unsigned walk_smem_off = 0;          // byte offset of the walk buffers in dynamic smem
    int32_t *d_h2 = nullptr;             // [rows][d*d] level-2 walk ends (walk_K >= 3)
    // walk index (walk_index_kernel): [rows][walk_cap] entries, [rows][walk_off_stride] bucket starts
    uint16_t *d_went = nullptr, *d_woff = nullptr;
    size_t went_elems = 0, woff_elems = 0;
    int walk_cap = 0, walk_off_stride = 0;
    long long wait_ns = 10ll * 1000 * 1000 * 1000;
    int cap_alloc = 0;                   // levels the counter arrays hold
    int nb_alloc = 0;                    // batches the counter arrays hold

    // device
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    int32_t *d_table = nullptr, *d_adj = nullptr;
    // Status block of an evaluation (one device allocation, mirrored in pinned
    // host memory, so that an evaluation needs one memset and one copy back):
    //   [0, 256) Ctl | bad, asym | levels_run[nb_alloc] | batch_ns[2 nb_alloc] |
    //   counts[nb][cap_req + 1]
    unsigned char *d_status = nullptr, *h_status = nullptr;
    size_t off_levels_run = 0, off_batch_ns = 0, off_counts = 0;
    int *d_bad = nullptr;                // the table failed its range check
    int *d_asym = nullptr;               // adjacency not symmetric: no push levels
    uint4 *d_V = nullptr, *d_F0 = nullptr, *d_F1 = nullptr;   // one allocation (rows_room)
    unsigned char *d_loop = nullptr;     // the level loop's other buffers lie in it (loop_room)
    uint32_t *d_fl0 = nullptr, *d_fl1 = nullptr;
    uint4 *d_P0 = nullptr, *d_P1 = nullptr;     // push-level frontier, all zero between launches
    uint32_t *d_pf0 = nullptr, *d_pf1 = nullptr;
    uint32_t *d_nf = nullptr;            // not-full bit per visited chunk
    uint32_t *d_nf2 = nullptr;           // its second copy (visited-set pull levels alternate)
    int *d_redo = nullptr, *h_redo = nullptr;   // sweep_kernel gave up: bfs_batch_kernel instead
    bool loop_only = false;              // every evaluation runs the level loop (graph_engine)
    bool sweep = true;                   // sweep_kernel where it applies (GG_SWEEP, and no level mode asked for)
    int sweep_wait = 0;                  // evaluations until it is tried again
    int sweep_nC = 0;                    // its chunks per row (0: never)
    bool width_asked = false;            // ... are those of the batch width asked for (gg_set_batch_sources)
    int sweep_K = 0;                     // levels before its dense ones
    int sweep_ends = 1;                  // most new vertices of a source's level below that
    bool sweep_list = false;             // the sources are a list (source_ball_kernel)
    bool ball_limits = false;            // the balls' kernels have their shared-memory limit
    uint4 *d_swA = nullptr, *d_swB = nullptr;   // its level buffers (one allocation), when wider than d_V
    size_t sw_chunks = 0;                // chunks each of them holds
    int *d_wasym = nullptr;              // one-way flag of the table (walk_index_kernel)
    unsigned long long *d_vtot = nullptr;   // [nb][3] level totals (dense visited-set pull without own chunks)
    // walk_all_kernel output: the level-K rows of every batch and their flag words
    uint4 *d_vall = nullptr;
    uint32_t *d_vall_fl = nullptr;
    size_t vall_chunks = 0;              // chunks d_vall holds
    long long walk_all_mb = 4096;        // budget for d_vall (GG_WALK_ALL_MB; 0: per-batch walk passes)
    bool p_dirty = true;                 // push buffers must be zeroed before the next launch
    unsigned long long *d_counts = nullptr;
    unsigned *d_masks = nullptr;
    unsigned long long *d_wcounts = nullptr, *h_wcounts = nullptr;   // pairs within the sources (on first use)
    size_t wcounts_n = 0;
    unsigned long long *d_level_ns = nullptr, *h_level_ns = nullptr;
    int *d_levels_run = nullptr, *h_levels_run = nullptr;                 // [nb_alloc]
    unsigned long long *d_batch_ns = nullptr, *h_batch_ns = nullptr;     // [2 * nb_alloc]
    int32_t *d_inv = nullptr;            // source index of each vertex, when the sources
    int src_first = 0;                   // are not the consecutive ids src_first, src_first+1, ...
    Ctl *d_ctl = nullptr;
    // pinned host
    int32_t *h_table = nullptr;
    unsigned long long *h_counts = nullptr;
    unsigned *h_masks = nullptr;
    Ctl *h_ctl = nullptr;
    int *h_bad = nullptr;

    bool use_graph = true;               // replay captured evaluations (GG_NO_GRAPH=1: never)
    cudaGraphExec_t graph_exec = nullptr;
    EvalKey graph_key{};

    // small graphs (direct_kernel)
    bool direct_allowed = false;         // no launch shape or level mode was asked for by the environment
    bool direct = false;                 // ... nor by a call
    int sms = 0, smem_optin = 0;
    int32_t *d_src = nullptr;            // the source list, when not consecutive
    unsigned char *d_dir = nullptr, *h_dir = nullptr;   // DirectCtl | counts[cap + 1] | masks[cap + 1]
    int dir_cap = 0;
    bool dir_dirty = true;               // d_dir's counters must be cleared before the next launch
    unsigned dir_seq = 0;                // launches of direct_kernel
    int dir_wait = 0;                    // evaluations until it walks again (after a table with one-way entries)
    int dir_orbits = 0;                  // sources whose rows hold one-way entries when any does (0: all rows do)
    uint16_t *d_pack = nullptr, *h_pack = nullptr;      // plain-graph table as 16-bit ids (on first use)
    bool table_stale = false;            // the last call's table went to h_pack, d_table is older

    double last_ms = 0.0;
    int last_launches = 0;
    int last_batches = 0;                // batches of the last evaluation
    uint64_t last_h2d = 0, last_d2h = 0;
};

namespace {

void free_batch_buffers(gg_engine *e) {
    cudaFree(e->d_vall); cudaFree(e->d_vall_fl);
    e->d_vall = nullptr;
    e->d_vall_fl = nullptr;
    e->vall_chunks = 0;
    cudaFree(e->d_swA);
    e->d_swA = e->d_swB = nullptr;
    e->sw_chunks = 0;
    cudaFree(e->d_V); cudaFree(e->d_loop);
    e->d_loop = nullptr;
    e->d_nf = e->d_nf2 = nullptr;
    e->d_V = e->d_F0 = e->d_F1 = nullptr;
    e->d_fl0 = e->d_fl1 = nullptr;
    e->d_P0 = e->d_P1 = nullptr;
    e->d_pf0 = e->d_pf1 = nullptr;
}

void free_counters(gg_engine *e) {
    cudaFree(e->d_status); cudaFree(e->d_masks); cudaFree(e->d_level_ns); cudaFree(e->d_vtot);
    cudaFreeHost(e->h_status); cudaFreeHost(e->h_masks);
    cudaFreeHost(e->h_level_ns);
    cudaFree(e->d_wcounts); cudaFreeHost(e->h_wcounts);
    e->d_wcounts = e->h_wcounts = nullptr;
    e->wcounts_n = 0;
    e->d_status = e->h_status = nullptr;
    e->d_bad = e->d_asym = e->d_wasym = e->h_bad = nullptr;
    e->d_vtot = nullptr;
    e->d_levels_run = e->h_levels_run = nullptr;
    e->d_batch_ns = e->h_batch_ns = nullptr;
    e->d_counts = nullptr; e->d_masks = nullptr; e->d_ctl = nullptr; e->d_level_ns = nullptr;
    e->h_counts = nullptr; e->h_masks = nullptr; e->h_ctl = nullptr; e->h_level_ns = nullptr;
    e->cap_alloc = e->nb_alloc = 0;
}

// A captured evaluation holds buffer addresses, the plan and the wait limit:
// drop it whenever one of them changes.
void invalidate_graph(gg_engine *e) {
    if (e->graph_exec) cudaGraphExecDestroy(e->graph_exec);
    e->graph_exec = nullptr;
}

void destroy_all(gg_engine *e) {
    if (!e) return;
    cudaSetDevice(e->device);
    if (e->stream) cudaStreamSynchronize(e->stream);
    free_batch_buffers(e);
    free_counters(e);
    if (e->d_adj != e->d_table) cudaFree(e->d_adj);  // the graph form aliases the two
    cudaFree(e->d_h2);
    cudaFree(e->d_went);
    cudaFree(e->d_woff);
    cudaFree(e->d_table); cudaFree(e->d_inv); cudaFree(e->d_src);
    cudaFree(e->d_dir); cudaFreeHost(e->h_dir); cudaFree(e->d_pack); cudaFreeHost(e->h_pack);
    cudaFreeHost(e->h_table);
    if (e->ev0) cudaEventDestroy(e->ev0);
    if (e->ev1) cudaEventDestroy(e->ev1);
    invalidate_graph(e);
    if (e->stream) cudaStreamDestroy(e->stream);
    delete e;
}

int kernel_degree_slot(int d) {
    switch (d) {
        case 3: case 4: case 6: case 8: case 12: case 16: return d;
        default: return 0;
    }
}

template <int MODE>
void *kernel_for_t(int d) {
    switch (kernel_degree_slot(d)) {
        case 3: return (void *)gg::bfs_batch_kernel<3, MODE>;
        case 4: return (void *)gg::bfs_batch_kernel<4, MODE>;
        case 6: return (void *)gg::bfs_batch_kernel<6, MODE>;
        case 8: return (void *)gg::bfs_batch_kernel<8, MODE>;
        case 12: return (void *)gg::bfs_batch_kernel<12, MODE>;
        case 16: return (void *)gg::bfs_batch_kernel<16, MODE>;
        default: return (void *)gg::bfs_batch_kernel<0, MODE>;
    }
}

// The BFS kernel for degree d; mode: see gg::kPlain.
void *kernel_for(int d, int mode = gg::kPlain) {
    return mode == gg::kPlanes ? kernel_for_t<gg::kPlanes>(d)
                               : mode == gg::kWithin ? kernel_for_t<gg::kWithin>(d) : kernel_for_t<gg::kPlain>(d);
}

// Walk ends per row up to depth K: d + d^2 + ... + d^K.
long long walk_cap_for(int d, int K) {
    long long sum = 0, p = 1;
    for (int k = 1; k <= K; ++k) { p *= d; sum += p; }
    return sum;
}

// Levels the walk pass computes for this plan: the largest K <= 4 whose walk ends
// per row stay within 600 (d = 8: 3 levels, 584 ends; d = 16: 2; d = 4: 4), within
// the index kernel's row buffer and bucket count (kIndexMaxCap ends, kIndexMaxKeys
// = batches * K buckets), with the level-2 table (rows * d^2 int32, K >= 3) within
// 64 MiB and the index (rows * (ends + buckets) uint16) within 1 GiB; off for
// evaluations of a single source batch.  GG_WALK_LEVELS overrides the depth (0 = off;
// still within the size limits).
int walk_levels(gg_engine *e) {
    const int env = env_int("GG_WALK_LEVELS", e->walk_pref);
    e->walk_auto = env < 0;
    const int d = e->d;
    if (d <= 0 || e->nC > gg::kWalkMaxNC || env == 0) return 0;
    int K = 0;
    for (int k = 1; k <= 4 && walk_cap_for(d, k) <= 600; ++k) K = k;
    const long long nb = ((long long)e->reps.size() + e->batch_bits - 1) / e->batch_bits;
    // The index costs one pass over every row's walk ends per evaluation; with a
    // single source batch the pass it saves is not worth it (n = 4096, d = 16: 0.070
    // against 0.060 ms; a lift with one batch: 0.135 against 0.097 ms).
    if (nb < 2) K = 0;
    if (env > 0) K = std::min(env, 4);
    for (; K > 0; --K) {
        const long long cap = walk_cap_for(d, K), keys = nb * K;
        const bool ok = cap <= gg::kIndexMaxCap && keys <= gg::kIndexMaxKeys &&
                        (K < 3 || (long long)e->rows * d * d * 4 <= (64ll << 20)) &&
                        (long long)e->rows * (cap + keys + 1) * 2 <= (1ll << 30);
        if (ok) break;
    }
    return K;
}

// Share of the pairs (ppm) below which a level's feeding frontier is left to the flag words
// of bfs_batch_kernel (n = 60000, d = 5, 0.5 % after the walk: 1561 us here, 3739 there; n =
// 40000, d = 4, 0.27 %: 1023 / 1463).
constexpr int kSweepThinPpm = 2000;

// Degrees 3 to 8 walk four steps, 9 to 16 three: at most 4096 walk ends a row.
constexpr int sweep_K(int d) { return d <= 8 ? 4 : 3; }
struct SweepKernels { void *ball, *source_ball, *wide, *narrow; };
template <int D = 3>
SweepKernels sweep_for(int d) {
    if constexpr (D > 16) {
        return {};
    } else {
        if (d == D)
            return {(void *)gg::ball_kernel<D, sweep_K(D)>, (void *)gg::source_ball_kernel<D>,
                    (void *)gg::sweep_kernel<D, true>, (void *)gg::sweep_kernel<D, false>};
        return sweep_for<D + 1>(d);
    }
}

// Pairs left (ppm) below which last_rows takes a level.  A share u of the pairs left
// becomes about u^(d-1) with the level, and a row's 4096 pairs must then rarely (one row
// in twenty) hold one that is still missing: those cost d^2 gathers.  Far from critical:
// a random graph's share falls from above a half to below a tenth in one level.
int sweep_last_ppm(int d) { return (int)(1e6 * std::min(0.2, std::pow(1.2e-5, 1.0 / (d - 1)))); }

// Room for the rows of every batch (walk_all_kernel, ball_kernel), grown as needed.
bool vall_room(gg_engine *e, size_t chunks) {
    if ((long long)((chunks * sizeof(uint4)) >> 20) > e->walk_all_mb) return false;
    if (chunks <= e->vall_chunks) return true;
    invalidate_graph(e);
    const bool had = e->vall_chunks > 0;
    cudaFree(e->d_vall); cudaFree(e->d_vall_fl);
    e->d_vall = nullptr;
    e->d_vall_fl = nullptr;
    e->vall_chunks = 0;
    if (fault("rows") || (had && fault("more_rows")) || cudaMalloc(&e->d_vall, chunks * sizeof(uint4)) != cudaSuccess ||
        cudaMalloc(&e->d_vall_fl, (chunks + 31) / 32 * sizeof(uint32_t)) != cudaSuccess) {
        cudaFree(e->d_vall); cudaFree(e->d_vall_fl);
        e->d_vall = nullptr;
        e->d_vall_fl = nullptr;
        (void)cudaGetLastError();
        return false;
    }
    e->vall_chunks = chunks;
    return true;
}

// The rows of every batch for sweep_kernel: d_F1 where one batch fits it, else d_vall.
bool sweep_in_f1(const gg_engine *e, int nb) { return nb == 1 && e->sweep_nC <= e->nC; }

// The shared-memory limit of the balls' kernels: the most sweep_width lets a block have (two
// blocks an SM).  It belongs to the kernel, which engines of other sizes launch too, in
// other threads perhaps: every engine sets the same, before its first use.
bool ball_limits(gg_engine *e) {
    if (e->ball_limits) return true;
    const SweepKernels k = sweep_for(e->d);
    if (cudaFuncSetAttribute(k.ball, cudaFuncAttributeMaxDynamicSharedMemorySize, e->smem_optin / 2) != cudaSuccess ||
        cudaFuncSetAttribute(k.source_ball, cudaFuncAttributeMaxDynamicSharedMemorySize, e->smem_optin / 2) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return e->ball_limits = true;
}

// An engine is created with the buffers of what its evaluations go to and takes others when
// one needs them: of direct_kernel, sweep_kernel and the level loop most engines only ever
// run one.  Creation and first call, with all of the level loop's at once and the others on
// the first call -> now: n = 9000, d = 4: 5.9 -> 3.7 ms; n = 30012, d = 6: 5.7 -> 4.7.

// The level-2 lists.
gg_status h2_room(gg_engine *e) {
    if (e->d_h2) return GG_OK;
    invalidate_graph(e);
    GG_CK(cudaMalloc(&e->d_h2, (size_t)e->rows * e->d * e->d * sizeof(int32_t)));
    return GG_OK;
}

// Three buffers of a batch's rows.
gg_status rows_room(gg_engine *e) {
    if (e->d_V) return GG_OK;
    invalidate_graph(e);
    const size_t n = ((size_t)e->items + 31) / 32 * 32;   // (512-byte boundaries)
    GG_CK(cudaMalloc(&e->d_V, 3 * n * sizeof(uint4)));
    e->d_F0 = e->d_V + n;
    e->d_F1 = e->d_F0 + n;
    return GG_OK;
}

// Everything the level loop (bfs_batch_kernel) needs for the present plan.
gg_status loop_room(gg_engine *e) {
    gg_status s = rows_room(e);
    if (s == GG_OK && e->walk_K >= 3) s = h2_room(e);
    if (s != GG_OK) return s;
    if (!e->d_loop) {
        const size_t n = ((size_t)e->items + 31) / 32 * 32, f = (n / 32 + 63) / 64 * 64;   // (256-byte boundaries)
        invalidate_graph(e);
        GG_CK(cudaMalloc(&e->d_loop, 2 * n * sizeof(uint4) + 6 * f * sizeof(uint32_t)));
        e->d_P0 = reinterpret_cast<uint4 *>(e->d_loop);
        e->d_P1 = e->d_P0 + n;
        uint32_t *w = reinterpret_cast<uint32_t *>(e->d_P1 + n);
        for (uint32_t **q : {&e->d_fl0, &e->d_fl1, &e->d_pf0, &e->d_pf1, &e->d_nf, &e->d_nf2}) {
            *q = w;
            w += f;
        }
        e->p_dirty = true;
    }
    const size_t went = (size_t)e->rows * e->walk_cap, woff = (size_t)e->rows * e->walk_off_stride;
    if (went != e->went_elems || woff != e->woff_elems) {
        invalidate_graph(e);
        cudaFree(e->d_went);
        cudaFree(e->d_woff);
        e->d_went = e->d_woff = nullptr;
        e->went_elems = e->woff_elems = 0;
        if (went) {
            GG_CK(cudaMalloc(&e->d_went, went * sizeof(uint16_t)));
            GG_CK(cudaMalloc(&e->d_woff, woff * sizeof(uint16_t)));
        }
        e->went_elems = went;
        e->woff_elems = woff;
    }
    return GG_OK;
}

// sweep_kernel's buffers: the level-2 lists or none, the rows of every batch, and two level
// buffers -- d_V and d_F0, or a wider pair of its own.  False: no memory for them.
bool sweep_room(gg_engine *e, int nb) {
    const size_t chunks = (size_t)e->rows * e->sweep_nC;
    if (!ball_limits(e)) return false;
    if ((!e->sweep_list && h2_room(e) != GG_OK) || (e->sweep_nC <= e->nC && rows_room(e) != GG_OK)) {
        (void)cudaGetLastError();
        return false;
    }
    if (!sweep_in_f1(e, nb) && !vall_room(e, nb * chunks)) return false;
    if (e->sweep_nC <= e->nC || chunks <= e->sw_chunks) return true;
    invalidate_graph(e);
    cudaFree(e->d_swA);
    e->d_swA = e->d_swB = nullptr;
    e->sw_chunks = 0;
    if (cudaMalloc(&e->d_swA, 2 * chunks * sizeof(uint4)) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    e->d_swB = e->d_swA + chunks;
    e->sw_chunks = chunks;
    return true;
}

int sweep_batches(const gg_engine *e) { return ((int)e->reps.size() + 128 * e->sweep_nC - 1) / (128 * e->sweep_nC); }

// Shared memory of a ball_kernel block.
size_t ball_smem(const gg_engine *e) {
    return (size_t)(gg::kBallBlock / 32) *
           gg::ball_warp_bytes(e->d, sweep_K(e->d), sweep_batches(e) * (e->sweep_nC / 32));
}

constexpr int kSrcBallWarps = gg::kSrcBallBlock / 32;

// sweep_kernel's chunks per row, or 0 where it never applies.  Every vertex a source, in
// order; batches of whole 4096-source parts; two ball_kernel blocks an SM; and the walk's
// last level not thin on a graph whose walks rarely meet (others find out at batch 0).
// Its batches are as wide as keeps a level's rows within 64 MB, and even: half a level's
// gathers then still hit L2, and there are fewer barriers and last_rows passes.  n = 65536,
// d = 8: 4096 wide 1322 us, 8192 1225, 12288 1441; n = 50000, d = 6: 923, 893, 978;
// n = 30012, d = 6: 4096 wide 452, 8192 408, 16384 386.
int sweep_width(gg_engine *e) {
    const int n_src = (int)e->reps.size();
    const bool all = n_src == e->rows && !e->d_inv && e->src_first == 0;
    e->sweep_list = !all;
    if (!e->sweep || e->d < 3 || e->d > 16 || n_src < 1) return 0;
    if (all ? e->rows < 4096 : (e->form == FORM_GRAPH || e->rows != e->N)) return 0;   // (rows past N: one-way)
    const int parts = (n_src + 4095) / 4096;
    const int most = std::max(1, (int)((64ll << 20) / ((long long)e->rows * 512)));
    const int nb = (parts + most - 1) / most;
    int nC = 32 * ((parts + nb - 1) / nb);
    if (!all && n_src <= 2048)
        for (nC = 1; 128 * nC < n_src;) nC *= 2;
    e->sweep_nC = e->width_asked ? e->nC : nC;
    if (e->sweep_nC % 32 != 0 && (all || (e->sweep_nC & (e->sweep_nC - 1)) != 0 || e->sweep_nC > 16)) return 0;
    if ((long long)e->rows * e->sweep_nC >= (1ll << 31)) return 0;
    if (all) {
        const int K = e->sweep_K = sweep_K(e->d);
        if (sweep_batches(e) * K > gg::kBallCounts || 2 * (ball_smem(e) + 4096) > (size_t)e->smem_optin) return 0;
        double last = e->d;
        for (int k = 1; k < K; ++k) last *= e->d - 1;
        return last * 1e6 >= (double)e->rows * kSweepThinPpm ? e->sweep_nC : 0;
    }
    // A list: another walked level as long as its reductions (41 a ns: 1024 sources, 32768
    // rows, d = 12, three levels 44 us) cost no more than a dense level (4 us and 13 TB/s of
    // gathers)
    const double dense_ns = 4000.0 + (double)e->rows * e->d * n_src / 8.0 / 13000.0;
    double last = e->d;
    int K = 1;
    e->sweep_ends = 1;
    // (a one-way table's level may be d times the one before)
    while (K + 1 < gg::kSrcBallLevels && e->sweep_ends * e->d <= gg::kSrcBallList &&
           last * (e->d - 1) * n_src / 41.0 <= dense_ns) {
        e->sweep_ends *= e->d;
        last *= e->d - 1;
        ++K;
    }
    e->sweep_K = K;
    if (2 * (kSrcBallWarps * (size_t)gg::source_ball_warp_bytes(e->rows, e->sweep_ends) + 2048) > (size_t)e->smem_optin) return 0;
    return e->sweep_nC;
}

// Whether an evaluation goes to sweep_kernel (asked once per evaluation), if direct_kernel
// does not take it and sweep_room has the memory.  A graph that it gave up on has paid for
// the attempt, and its engine leaves it out for a while.
bool sweep_turn(gg_engine *e, const gg_eval_opts *o) {
    const int cap = (o && o->max_levels > 0) ? o->max_levels : std::max(e->rows, 1);
    if (!e->sweep_nC || (o && (o->level_ns || o->want_wvc || o->src_begin || o->src_end)) || fault("barrier") ||
        e->sweep_K > cap)
        return false;
    if (e->sweep_wait > 0) {
        --e->sweep_wait;
        return false;
    }
    return true;
}

template <int D, bool ONE>
void *walk_all_of(int K) {
    return K == 1 ? (void *)gg::walk_all_kernel<D, 1, ONE> : K == 2 ? (void *)gg::walk_all_kernel<D, 2, ONE>
                                                                    : (void *)gg::walk_all_kernel<D, 3, ONE>;
}

// walk_all_kernel for an evaluation of nb batches, or nullptr (a walk pass per
// batch): visited-set pull levels, batches of a multiple of 4096 sources, degree 3, 4, 6
// or 8, K <= 3 (with the level-2 table, or 16-byte rows), and the level-K rows of all nb
// batches within the GG_WALK_ALL_MB budget.  Grows d_vall as needed (a failed allocation
// falls back to the per-batch pass).  Only where the level loop runs a graph at all: after
// sweep_kernel gave up, source ranges, per-level times (one-way n = 30011, d = 6, degree 6
// walked for all batches: 784 -> 680 us).
void *walk_all_for(gg_engine *e, int K, int nb) {
    if (!e->walk_vpull || e->nC % 32 != 0 || K < 1 || K > 3 || nb * (e->nC / 32) * K > gg::kIndexMaxKeys) return nullptr;
    if (e->d != 3 && e->d != 4 && e->d != 6 && e->d != 8) return nullptr;
    if (K < 3 && e->d % 4 != 0) return nullptr;
    if (!vall_room(e, (size_t)nb * e->items)) return nullptr;
    void *k = nullptr;
    if (e->nC == 32)
        k = e->d == 8 ? walk_all_of<8, true>(K) : e->d == 4 ? walk_all_of<4, true>(K)
          : e->d == 6 ? (void *)gg::walk_all_kernel<6, 3, true> : (void *)gg::walk_all_kernel<3, 3, true>;
    else
        k = e->d == 8 ? walk_all_of<8, false>(K) : e->d == 4 ? walk_all_of<4, false>(K)
          : e->d == 6 ? (void *)gg::walk_all_kernel<6, 3, false> : (void *)gg::walk_all_kernel<3, 3, false>;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, gg::walk_all_smem(K)) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    return k;
}

void *index_kernel_for(int d) {
    switch (kernel_degree_slot(d)) {
        case 3: return (void *)gg::walk_index_kernel<3>;
        case 4: return (void *)gg::walk_index_kernel<4>;
        case 6: return (void *)gg::walk_index_kernel<6>;
        case 8: return (void *)gg::walk_index_kernel<8>;
        case 12: return (void *)gg::walk_index_kernel<12>;
        case 16: return (void *)gg::walk_index_kernel<16>;
        default: return (void *)gg::walk_index_kernel<0>;
    }
}

// Source-batch plan: batch width, chunks per row, grid size.
// gg_autotune's choices (batch width, resident blocks per SM, walk depth) are
// kept in the tuning cache under (GPU, form, rows, degree, sources).
std::string engine_tune_key(const gg_engine *e) {
    return gg::tune_key(e->device, "graph", {e->form, e->rows, e->d, (long long)e->reps.size()});
}

gg_status plan(gg_engine *e, int want_bits) {
    invalidate_graph(e);
    const int n_src = (int)e->reps.size();
    int bits;
    if (want_bits > 0) {
        bits = want_bits;
    } else {
        const int env = env_int("GG_BATCH_SOURCES", 0);
        std::vector<int> tuned;
        if (env > 0) {
            bits = env;
        } else if (gg::tune_get(engine_tune_key(e), &tuned) && tuned.size() >= 3 && tuned[0] > 0) {
            bits = tuned[0];
            e->bps_cap = tuned[1];
            e->walk_pref = tuned[2];
        } else {
            // The widest batch whose three bitsets (3 * rows * bits / 8 bytes)
            // stay within 3/4 of the L2, so that the gathers hit L2 rather than
            // HBM; at least 4096 sources (one 512-byte row segment per vertex)
            // when there are that many.
            int l2 = 0;
            if (cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, e->device) != cudaSuccess || l2 <= 0) {
                (void)cudaGetLastError();
                l2 = 64 << 20;
            }
            const double per_bit = 3.0 * e->rows / 8.0;
            long long fit = (long long)(0.75 * l2 / per_bit);
            fit = std::max<long long>(fit, 4096);
            bits = (int)std::min<long long>(fit, n_src);
            if (bits > 4096) bits = (bits / 4096) * 4096;
        }
    }
    bits = std::max(128, ((std::min(bits, std::max(n_src, 1)) + 127) / 128) * 128);
    const long long items = (long long)e->rows * (bits / 128);
    if (items >= (1ll << 31)) return fail(GG_BAD_ARG, "rows x batch width exceeds 2^31 uint4 chunks");
    if (bits != e->batch_bits) {
        free_batch_buffers(e);
        e->batch_bits = bits;
        e->nC = bits / 128;
        e->items = (uint32_t)items;
    }
    // Walk pass: levels 1..K of each batch from the walk ends of every row.
    e->walk_K = walk_levels(e);
    e->walk_rpg = 1;
    size_t walk_bytes = 0;
    if (e->walk_K > 0) {
        int g = e->nC, b = 32;
        while (b) { const int t = g % b; g = b; b = t; }   // gcd(nC, 32)
        e->walk_rpg = 32 / g;
        walk_bytes = (size_t)(gg::kBlock / 32) * gg::walk_smem_per_warp(e->nC);
    }
    e->sweep_nC = sweep_width(e);
    // row stride of the index: the walk ends, rounded up to a multiple of 8 (rows start
    // 16-byte aligned: the index kernel writes them 16 bytes at a time)
    e->walk_cap = e->walk_K ? (int)((walk_cap_for(e->d, e->walk_K) + 7) & ~7ll) : 0;
    e->walk_off_stride = e->walk_K ? (int)(((long long)e->reps.size() + bits - 1) / bits) * e->walk_K + 1 : 0;
    int per_sm = 0, sms = 0;
    GG_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device));
    GG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel_for(e->d), gg::kBlock, walk_bytes));
    if (per_sm < 1) return fail(GG_CUDA_ERROR, "BFS kernel cannot be resident");
    const long long tiles = ((long long)e->items + 31) / 32;
    const long long want = (tiles + (gg::kBlock / 32) - 1) / (gg::kBlock / 32);
    // Resident blocks per SM: at most what fits; GG_BLOCKS_PER_SM, else the tuned cap.
    const int cap_per_sm = env_int("GG_BLOCKS_PER_SM", e->bps_cap);
    if (cap_per_sm > 0) per_sm = std::min(per_sm, cap_per_sm);
    e->grid = (int)std::max<long long>(1, std::min<long long>((long long)per_sm * sms, want));
    // Shared-memory adjacency slice: a block's contiguous tile range spans at most
    // ceil(tiles/grid)*32/nC + 2 vertices.  Cached when it fits a small budget and
    // does not lower the number of resident blocks.
    e->adj_smem_rows = 0;
    e->smem_bytes = walk_bytes;
    e->walk_smem_off = 0;
    if (env_int("GG_ADJ_SMEM", 1) && e->d > 0) {
        const long long per_block = (tiles + e->grid - 1) / e->grid;
        const long long rows = per_block * 32 / e->nC + 2;
        const long long bytes = (rows * e->d * 4 + 15) / 16 * 16;
        // within 32 KB, and within the 48 KB a launch gets without opting in
        if (bytes <= 32 * 1024 && bytes + (long long)walk_bytes <= 48 * 1024) {
            int per_sm2 = 0;
            GG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm2, kernel_for(e->d), gg::kBlock,
                                                                (size_t)bytes + walk_bytes));
            if (per_sm2 >= per_sm) {
                e->adj_smem_rows = (int)rows;
                e->walk_smem_off = (unsigned)bytes;
                e->smem_bytes = (size_t)bytes + walk_bytes;
            }
        }
    }
    return GG_OK;
}

gg_status ensure_counters(gg_engine *e, int cap, int nb) {
    if (cap <= e->cap_alloc && nb <= e->nb_alloc) return GG_OK;
    cap = std::max(cap, e->cap_alloc);
    nb = std::max(nb, e->nb_alloc);
    invalidate_graph(e);
    free_counters(e);
    const size_t n = (size_t)(cap + 1) * nb;
    e->off_levels_run = 512;
    e->off_batch_ns = e->off_levels_run + (((size_t)nb * sizeof(int) + 15) & ~size_t(15));
    e->off_counts = e->off_batch_ns + (size_t)nb * 2 * sizeof(unsigned long long);
    const size_t bytes = e->off_counts + n * sizeof(unsigned long long);
    GG_CK(cudaMalloc(&e->d_status, bytes));
    GG_CK(cudaMallocHost(&e->h_status, bytes));
    e->d_ctl = reinterpret_cast<Ctl *>(e->d_status);
    e->h_ctl = reinterpret_cast<Ctl *>(e->h_status);
    e->d_bad = reinterpret_cast<int *>(e->d_status + sizeof(Ctl));
    e->h_bad = reinterpret_cast<int *>(e->h_status + sizeof(Ctl));
    e->d_asym = e->d_bad + 1;
    e->d_wasym = e->d_bad + 2;
    e->d_redo = e->d_bad + 3;
    e->h_redo = e->h_bad + 3;
    GG_CK(cudaMalloc(&e->d_vtot, (size_t)nb * 3 * sizeof(unsigned long long)));
    e->d_levels_run = reinterpret_cast<int *>(e->d_status + e->off_levels_run);
    e->h_levels_run = reinterpret_cast<int *>(e->h_status + e->off_levels_run);
    e->d_batch_ns = reinterpret_cast<unsigned long long *>(e->d_status + e->off_batch_ns);
    e->h_batch_ns = reinterpret_cast<unsigned long long *>(e->h_status + e->off_batch_ns);
    e->d_counts = reinterpret_cast<unsigned long long *>(e->d_status + e->off_counts);
    e->h_counts = reinterpret_cast<unsigned long long *>(e->h_status + e->off_counts);
    GG_CK(cudaMalloc(&e->d_masks, n * sizeof(unsigned)));
    GG_CK(cudaMallocHost(&e->h_masks, n * sizeof(unsigned)));
    GG_CK(cudaMalloc(&e->d_level_ns, (size_t)(cap + 1) * sizeof(unsigned long long)));
    GG_CK(cudaMallocHost(&e->h_level_ns, (size_t)(cap + 1) * sizeof(unsigned long long)));
    e->cap_alloc = cap;
    e->nb_alloc = nb;
    return GG_OK;
}

void *direct_for(int W) {
    return W == 1 ? (void *)gg::direct_kernel<1> : W == 2 ? (void *)gg::direct_kernel<2> : (void *)gg::direct_kernel<4>;
}

// ---- small graphs: direct_kernel -------------------------------------------------

struct DirectPlan {
    int W = 0;            // 32-source words a vertex (0: not for this evaluation)
    bool adj_smem = false;
    size_t smem = 0;
    int grid = 0, block = 0;
};

constexpr double kSweepUsPerChunk = 0.064e-3, kLoopUsPerChunk = 0.12e-3;
constexpr int kDirectCheck = 32;   // look-ups of the one-way check, at most, a thread of direct_kernel

// Rows that an evaluation checks for one-way entries, to take its first levels from walks
// then, or 0: where the check is not a small part of a pass, and for a while after a table
// that had some.
int direct_check(const gg_engine *e, int grid, int block) {
    const int rows = e->dir_orbits ? e->dir_orbits : e->rows;
    const long long looks = ((long long)rows + grid - 1) / grid * e->d * e->d;
    return e->dir_wait > 0 || looks > (long long)kDirectCheck * block ? 0 : rows;
}

// The word width that makes the fewest rounds of blocks cheapest, or none: the visited
// sets of every width must fit a block's shared memory.  A random row of 4, 8 or 16 bytes
// per lane costs about 3.5, 6.2 and 10.4 shared-memory cycles a warp.
DirectPlan direct_plan(const gg_engine *e, int ns, bool wvc, bool sweep) {
    DirectPlan best;
    if (!e->direct || e->d < 1 || e->rows < 1 || e->rows > 65535 || ns < 1) return best;   // (d = 0: no walk ends)
    const size_t budget = (size_t)e->smem_optin - 1024;
    double cost = 1e300;
    for (int W : {1, 2, 4}) {
        const size_t set = ((size_t)e->rows * W + 3) / 4 * 16, adj = ((size_t)e->rows * e->d * 2 + 15) / 16 * 16;
        if (2 * set > budget) continue;
        const int grid = (ns + 32 * W - 1) / (32 * W);
        const bool in_smem = 2 * set + adj <= budget;
        const size_t smem = 2 * set + (in_smem ? adj : 0);
        const int block = e->rows >= 1024 ? gg::kDirectBlock : std::max(128, (e->rows + 31) / 32 * 32);
        const int per_sm = (int)std::max<size_t>(1, std::min<size_t>(1024 / block, budget / std::max<size_t>(smem + 1024, 1)));
        const double rounds = std::ceil((double)grid / (e->sms * per_sm));
        const double c = rounds * (W == 1 ? 3.5 : W == 2 ? 6.2 : 10.4) * per_sm;
        if (c < cost && (rounds == 1 || e->rows <= 20480)) {
            cost = c;
            best = DirectPlan{W, in_smem, smem, grid, block};
        }
    }
    // Against bfs_batch_kernel: microseconds of the two (fits of both sides over n = 64 to
    // 27000 and lifts of 20 to 4000 orbits).  A round of one-word groups takes 3.2 + 0.1 d
    // ns a row (a tenth more with the WVC masks), less certain for a single round; the level
    // loop 50 us and 0.12 ns a chunk of 128 sources.  Device times: n = 4096, d = 16: 25
    // against 67 us; 16000, 6: 239 / 372; lifts of 6000 vertices, 500 orbits: 29 / 59, of
    // 20000, 1000: 85 / 82, of 20000, 2000: 96 / 90.
    // Against sweep_kernel, whose levels take half of that a chunk (whole calls, direct
    // first): n = 8192, d = 4: 70 against 111 us, 8192, 16: 120 / 131, 9000, 7: 104 / 133,
    // 10000, 8: 169 / 126, 10000, 5: 150 / 129, 12000, 4: 144 / 145, 16384, 6: 302 / 187.
    // Degrees without a loop of their own cost more where no walk shortens the search (tables
    // with one-way entries, whole calls against bfs_batch_kernel: 16000, 10: 536 / 454; 20000,
    // 10: 828 / 567; 14000, 13: 443 / 392; 10000, 9: 250 / 276; 9000, 16: 174 / 241), and above 20
    // they need their rows in shared memory (4096, 24: 89 / 116; 9000, 24: 344 / 301; 3000, 40,
    // 120 KB short of room: 159 / 109), few of them (1000, 64: 136 / 107; 1000, 40: 59 / 88).
    if (best.W) {
        const bool one = best.grid <= e->sms;
        double direct_us = cost / 3.5 * e->rows * (3.2 + 0.1 * e->d) * 1e-3 * (wvc ? 1.1 : 1.0) * (one ? 1.12 : 1.0);
        if (!sweep && e->d >= 9 && e->d != 12 && !direct_check(e, best.grid, best.block)) direct_us *= std::min(1.3, 1.0 + 0.06 * (e->d - 7));
        const double chunks = (double)e->rows * ((ns + 127) / 128);
        if (e->d > 20 && (!best.adj_smem || (e->d > 48 && (long long)e->rows * e->d > 50000))) best.W = 0;
        if (direct_us > 50.0 + (sweep ? kSweepUsPerChunk : kLoopUsPerChunk) * chunks) best.W = 0;
    }
    return best;
}

gg_status create_common(gg_engine *e) {
    if (fault("alloc")) return fail(GG_OUT_OF_MEMORY, "injected allocation failure");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        (void)cudaGetLastError();
        return fail(GG_NO_DEVICE, "no CUDA device");
    }
    if (e->device < 0 || e->device >= ndev) return fail(GG_NO_DEVICE, "device index out of range");
    GG_CK(cudaSetDevice(e->device));
    GG_CK(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking));
    GG_CK(cudaEventCreate(&e->ev0));
    GG_CK(cudaEventCreate(&e->ev1));
    const size_t tb = std::max<size_t>(e->table_elems, 1) * sizeof(int32_t);
    GG_CK(cudaMalloc(&e->d_table, tb));
    GG_CK(cudaMallocHost(&e->h_table, tb));
    if (e->form == FORM_GRAPH) {
        e->d_adj = e->d_table;  // the graph table is the adjacency
    } else {
        GG_CK(cudaMalloc(&e->d_adj, std::max<size_t>((size_t)e->rows * e->d, 1) * sizeof(int32_t)));
    }
    // The kernel finds a chunk's source from its vertex: directly when the
    // sources are consecutive vertex ids, else through the inverse list.
    bool consecutive = true;
    for (size_t i = 0; i < e->reps.size() && consecutive; ++i)
        consecutive = e->reps[i] == e->reps[0] + (int32_t)i;
    e->src_first = e->reps.empty() ? 0 : e->reps[0];
    if (!consecutive) {
        std::vector<int32_t> inv((size_t)std::max(e->rows, 1), -1);
        for (size_t i = 0; i < e->reps.size(); ++i) {
            const int32_t v = e->reps[i];
            if (v < 0 || v >= e->rows || inv[(size_t)v] != -1)
                return fail(GG_BAD_ARG, "sources must be distinct vertices");
            inv[(size_t)v] = (int32_t)i;
        }
        GG_CK(cudaMalloc(&e->d_src, e->reps.size() * sizeof(int32_t)));
        GG_CK(cudaMemcpyAsync(e->d_src, e->reps.data(), e->reps.size() * sizeof(int32_t), cudaMemcpyHostToDevice, e->stream));
        GG_CK(cudaMalloc(&e->d_inv, inv.size() * sizeof(int32_t)));
        GG_CK(cudaMemcpyAsync(e->d_inv, inv.data(), inv.size() * sizeof(int32_t), cudaMemcpyHostToDevice, e->stream));
        GG_CK(cudaStreamSynchronize(e->stream));   // an evaluation may come on another stream
    }
    e->dense_w_ppm = env_int("GG_DENSE_W_PPM", e->dense_w_ppm);
    e->dense_r_ppm = env_int("GG_DENSE_R_PPM", e->dense_r_ppm);
    e->full_skip_ppm = env_int("GG_FULL_SKIP_PPM", e->full_skip_ppm);
    e->split_ppm = env_int("GG_SPLIT_PPM", e->split_ppm);
    e->walk_vpull = env_int("GG_VPULL", e->walk_vpull) != 0;
    e->walk_own_skip = env_int("GG_OWN_SKIP", e->walk_own_skip) != 0;
    e->walk_third = env_int("GG_WALK_THIRD", e->walk_third) != 0;
    e->walk_all_mb = env_int("GG_WALK_ALL_MB", (int)e->walk_all_mb);
    e->push_ppm = env_int("GG_PUSH_PPM", e->push_ppm);
    e->push_min_items = env_int("GG_PUSH_MIN_ITEMS", e->push_min_items);
    e->use_graph = env_int("GG_NO_GRAPH", 0) == 0;
    // direct_kernel unless a launch shape or level mode is asked for
    e->direct = true;
    for (const char *name : {"GG_BATCH_SOURCES", "GG_BLOCKS_PER_SM", "GG_WALK_LEVELS", "GG_DENSE_W_PPM", "GG_DENSE_R_PPM",
                             "GG_FULL_SKIP_PPM", "GG_SPLIT_PPM", "GG_VPULL", "GG_OWN_SKIP", "GG_WALK_THIRD",
                             "GG_WALK_ALL_MB", "GG_PUSH_PPM", "GG_PUSH_MIN_ITEMS", "GG_NO_GRAPH", "GG_ADJ_SMEM"})
        if (std::getenv(name)) e->direct = false;
    e->sweep = e->direct && env_int("GG_SWEEP", 1) != 0;
    if (env_int("GG_DIRECT", 1) == 0) e->direct = false;
    e->direct_allowed = e->direct;
    {
        // a lift whose sizes are multiples of its orbit's: a row is its orbit's, translated
        bool whole = e->form != FORM_GRAPH && e->rows == e->N;
        if (e->form == FORM_PART) whole = whole && e->N % e->M == 0;
        else
            for (int j = 0; j < 3 && whole; ++j) whole = e->dims[j] % e->dims[3 + j] == 0;
        e->dir_orbits = whole ? (int)e->reps.size() : 0;
    }
    GG_CK(cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, e->device));
    GG_CK(cudaDeviceGetAttribute(&e->smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, e->device));
    for (int W : {1, 2, 4})
        GG_CK(cudaFuncSetAttribute(direct_for(W), cudaFuncAttributeMaxDynamicSharedMemorySize, e->smem_optin - 1024));
    const int wait_ms = env_int("GG_WAIT_LIMIT_MS", 10000);
    e->wait_ns = (long long)std::max(wait_ms, 1) * 1000000ll;
    gg_status s = plan(e, 0);
    // the buffers of a whole evaluation
    const bool sweep = e->sweep_nC > 0;
    if (s == GG_OK && (e->loop_only || !direct_plan(e, (int)e->reps.size(), false, sweep).W) &&
        (e->loop_only || !sweep || !sweep_room(e, sweep_batches(e))))
        s = loop_room(e);
    if (s != GG_OK) return s;
    return ensure_counters(e, 128, 1);
}

gg_status finish_create(gg_engine *e, gg_engine **out) {
    gg_status s = create_common(e);
    if (s != GG_OK) {
        destroy_all(e);
        *out = nullptr;
        return s;
    }
    *out = e;
    return GG_OK;
}

gg_status graph_create(int N, int degree_max, int device, bool loop_only, gg_engine **out) {
    if (!out) return fail(GG_BAD_ARG, "null out");
    *out = nullptr;
    if (N < 1 || degree_max < 0) return fail(GG_BAD_ARG, "need N >= 1, degree_max >= 0");
    gg_engine *e = new gg_engine();
    e->loop_only = loop_only;
    e->form = FORM_GRAPH; e->device = device;
    e->N = N; e->M = N; e->d = degree_max; e->rows = N; e->scale = 1;
    e->table_elems = (size_t)N * degree_max;
    e->reps.resize(N);
    for (int i = 0; i < N; ++i) e->reps[i] = i;
    return finish_create(e, out);
}

// A lifted form's table (device memory) -> the pull adjacency d_adj.
void launch_expand(gg_engine *e, const int32_t *d_table, cudaStream_t st, const bool sweep = false) {
    const long long n = (long long)e->rows * e->d;
    ExpandArgs x{};
    x.table = d_table;
    x.adj = e->d_adj;
    x.form = (e->form == FORM_PART) ? 1 : (e->form == FORM_PIECE ? 2 : 3);
    x.rows = e->rows; x.d = e->d; x.N = e->N; x.M = e->M;
    x.Nx = e->dims[0]; x.Ny = e->dims[1]; x.Nz = e->dims[2];
    x.Mx = e->dims[3]; x.My = e->dims[4]; x.Mz = e->dims[5];
    if (sweep && e->sweep_list) {
        x.vall = sweep_in_f1(e, sweep_batches(e)) ? e->d_F1 : e->d_vall;
        x.chunks = (long long)sweep_batches(e) * e->rows * e->sweep_nC;
        x.nC = e->sweep_nC;
        x.ns_total = (int)e->reps.size();
    }
    gg::expand_kernel<<<(int)std::min<long long>((n + 255) / 256, 8192), 256, 0, st>>>(x);
}

gg_status ensure_direct(gg_engine *e, int cap) {
    if (e->d_dir && cap <= e->dir_cap) return GG_OK;
    cap = std::max(cap, 256);
    cudaFree(e->d_dir); cudaFreeHost(e->h_dir);
    e->d_dir = e->h_dir = nullptr;
    e->dir_cap = 0;
    const size_t n = (size_t)cap + 1, bytes = 64 + n * 12;
    GG_CK(cudaMalloc(&e->d_dir, bytes));
    GG_CK(cudaMallocHost(&e->h_dir, bytes));
    std::memset(e->h_dir, 0, 64);
    e->dir_cap = cap;
    e->dir_dirty = true;
    return GG_OK;
}

// One evaluation by direct_kernel.  `table`: the calculator table in device memory, or
// adj16: a plain graph's checked 16-bit ids (device or pinned host memory).
gg_status direct_eval(gg_engine *e, const DirectPlan &p, const int32_t *table, const uint16_t *adj16,
                      const gg_eval_opts *o, int s0, int ns, int cap, gg_result *r, cudaStream_t st) {
    gg_status s = ensure_direct(e, cap);
    if (s != GG_OK) return s;
    (void)cudaGetLastError();
    if (fault("launch")) return fail(GG_CUDA_ERROR, "injected launch failure");
    const bool wvc = o && o->want_wvc;
    const long long n = (long long)e->rows * e->d;
    int launches = 1;
    gg::DirectArgs a{};
    a.adj = e->d_adj;
    a.adj16 = adj16;
    if (adj16) {
        // read as it is
    } else if (e->form == FORM_GRAPH) {
        a.adj = table;
        if ((reinterpret_cast<uintptr_t>(table) & 15u) && n > 0) {   // 16-byte loads
            GG_CK(cudaMemcpyAsync(e->d_table, table, (size_t)n * 4, cudaMemcpyDeviceToDevice, st));
            a.adj = e->d_table;
        }
        if (!p.adj_smem && n > 0) {
            GG_CK(cudaMemsetAsync(e->d_bad, 0, sizeof(int), st));
            gg::check_table_kernel<<<(int)std::min<long long>((n + 255) / 256, 4096), 256, 0, st>>>(a.adj, n, e->rows,
                                                                                                 e->d_bad);
            GG_CK(cudaGetLastError());
            a.bad_table = e->d_bad;
            ++launches;
        }
    } else if (n > 0) {
        launch_expand(e, table, st);
        GG_CK(cudaGetLastError());
        ++launches;
    }
    a.src = e->d_src;
    a.src_first = e->src_first;
    a.src_begin = s0;
    a.ns_total = ns;
    a.rows = e->rows; a.d = e->d;
    a.max_levels = cap;
    a.adj_smem = p.adj_smem ? 1 : 0;
    const size_t off = 64 + ((size_t)e->dir_cap + 1) * 8;
    a.ctl = reinterpret_cast<gg::DirectCtl *>(e->d_dir);
    a.h_ctl = reinterpret_cast<gg::DirectCtl *>(e->h_dir);
    a.counts = reinterpret_cast<unsigned long long *>(e->d_dir + 64);
    a.h_counts = reinterpret_cast<unsigned long long *>(e->h_dir + 64);
    a.masks = wvc ? reinterpret_cast<unsigned *>(e->d_dir + off) : nullptr;
    a.h_masks = reinterpret_cast<unsigned *>(e->h_dir + off);
    a.batch_ns = e->h_batch_ns;
    a.check = direct_check(e, p.grid, p.block);
    a.check_src = e->dir_orbits > 0;
    if (e->dir_wait > 0) --e->dir_wait;
    void *k = direct_for(p.W);
    e->last_ms = 0.0;
    if (e->dir_dirty) {
        const size_t c = 64 + ((size_t)e->dir_cap + 1) * 8;
        GG_CK(cudaMemsetAsync(e->d_dir, 0, c, st));
        GG_CK(cudaMemsetAsync(e->d_dir + c, 0xff, ((size_t)e->dir_cap + 1) * 4, st));
    }
    for (;;) {
        e->dir_dirty = true;   // until the launch has handed its counters over
        a.seq = ++e->dir_seq;
        if (a.seq == 0) a.seq = ++e->dir_seq;   // 0: none yet
        void *args[] = {&a};
        GG_CK(cudaLaunchKernel(k, dim3((unsigned)p.grid), dim3((unsigned)p.block), args, p.smem, st));
        // The kernel's last block stores its number after the counters; a wait for the stream
        // takes a few microseconds longer to come back.  Not there within a few milliseconds:
        // wait for the stream (a long evaluation, or an error to report).
        {
            const volatile unsigned *seq = &a.h_ctl->seq;
            const auto t0 = std::chrono::steady_clock::now();
            unsigned it = 0;
            while (*seq != a.seq) {
                if ((++it & 1023u) == 0u && std::chrono::steady_clock::now() - t0 > std::chrono::milliseconds(5)) {
                    GG_CK(cudaStreamSynchronize(st));
                    if (*seq != a.seq) return fail(GG_CUDA_ERROR, "direct_kernel ended without handing its counters over");
                    break;
                }
            }
            std::atomic_thread_fence(std::memory_order_acquire);
        }
        e->dir_dirty = false;
        e->last_ms += (double)(e->h_batch_ns[1] - e->h_batch_ns[0]) * 1e-6;
        if (!a.check || !a.h_ctl->oneway || a.h_ctl->bad) break;
        // one-way entries: what the walks found are not the sources' levels
        a.check = 0;
        e->dir_wait = 63;
        ++launches;
    }
    e->last_launches = launches;
    e->last_batches = 1;
    e->last_d2h = sizeof(gg::DirectCtl) + ((size_t)a.h_ctl->levels_run + 1) * (wvc ? 12 : 8);
    if (a.h_ctl->bad) return fail(GG_BAD_ARG, "adjacency entry outside [0, N)");
    const int run = a.h_ctl->levels_run;
    gg_result R{};
    R.scale = e->scale;
    R.pairs = (uint64_t)ns * (uint64_t)e->rows;
    R.n_sources = ns;
    R.batches = 1;
    R.wvc = -1;
    for (int L = 0; L <= run; ++L) {
        R.reached += a.h_counts[L];
        R.total += (uint64_t)L * a.h_counts[L];
        if (L > 0 && a.h_counts[L]) R.levels = L;
    }
    R.level_steps = run;
    R.capped = run >= cap && a.h_counts[cap] ? 1 : 0;
    R.connected = (!R.capped && R.reached == R.pairs) ? 1 : 0;
    if (wvc) R.wvc = R.levels > 0 ? __builtin_popcount(a.h_masks[R.levels - 1] ^ a.h_masks[R.levels]) : 0;
    if (o && o->level_counts)
        for (int L = 0; L <= cap; ++L) o->level_counts[L] = L <= run ? a.h_counts[L] : 0ull;
    *r = R;
    return GG_OK;
}

// Core evaluation with the table already on the device (d_table_in) on `st`.
gg_status run_eval(gg_engine *e, const int32_t *d_table_in, const gg_eval_opts *o, gg_result *r,
                   cudaStream_t st, const gg::EvalExtra *x = nullptr, int sweep_asked = -1) {
    const int n_src_all = x && x->inv ? x->ns : (int)e->reps.size();
    int s0 = 0, s1 = n_src_all;
    if (x && x->inv && (n_src_all < 1 || n_src_all > e->rows)) return fail(GG_BAD_ARG, "bad source list");
    if (x && x->planes && (o && (o->src_begin || o->src_end))) return fail(GG_BAD_ARG, "planes need every source");
    if (o && (o->src_begin || o->src_end)) {
        s0 = o->src_begin;
        s1 = o->src_end;
        if (s0 < 0 || s1 > n_src_all || s0 >= s1) return fail(GG_BAD_ARG, "bad source range");
        if (o->want_wvc && (s0 % 32)) return fail(GG_BAD_ARG, "WVC needs a 32-aligned source range");
    }
    const int cap_req = (o && o->max_levels > 0) ? o->max_levels : std::max(e->rows, 1);
    const bool wvc = o && o->want_wvc;
    const bool want_ns = o && o->level_ns;
    const int ns_all = s1 - s0;
    bool sweep = !x && (sweep_asked < 0 ? sweep_turn(e, o) : sweep_asked != 0);
    if (!x && !want_ns && !fault("barrier")) {
        DirectPlan p = direct_plan(e, ns_all, wvc, sweep);
        if (!p.W && sweep && !sweep_room(e, sweep_batches(e))) {
            sweep = false;
            p = direct_plan(e, ns_all, wvc, false);
        }
        if (p.W) return direct_eval(e, p, d_table_in, nullptr, o, s0, ns_all, cap_req, r, st);
        if (e->dir_wait > 0) --e->dir_wait;
    }
    const int nb_plain = (ns_all + e->batch_bits - 1) / e->batch_bits;
    int nb = sweep ? sweep_batches(e) : nb_plain;
    const bool within = x && x->within;
    if (within && (!x->inv || wvc || x->planes || e->form != FORM_GRAPH)) return fail(GG_BAD_ARG, "pairs within the sources need a source list");
    // Row width.  A short source list fills one batch of narrower rows (1600 of 65536
    // sources: 13 chunks instead of 32).
    const int nC = within && nb == 1 ? (ns_all + 127) / 128 : e->nC;
    const uint32_t items = (uint32_t)((long long)e->rows * nC);
    gg_status s = ensure_counters(e, cap_req, std::max(nb, nb_plain));
    if (s != GG_OK) return s;
    if (within && (size_t)nb * (cap_req + 1) > e->wcounts_n) {
        cudaFree(e->d_wcounts); cudaFreeHost(e->h_wcounts);
        e->d_wcounts = e->h_wcounts = nullptr;
        e->wcounts_n = 0;
        GG_CK(cudaMalloc(&e->d_wcounts, (size_t)nb * (cap_req + 1) * sizeof(unsigned long long)));
        GG_CK(cudaMallocHost(&e->h_wcounts, (size_t)nb * (cap_req + 1) * sizeof(unsigned long long)));
        e->wcounts_n = (size_t)nb * (cap_req + 1);
    }
    const int stride = cap_req + 1;      // counts of batch b at [b * stride, (b + 1) * stride)

    (void)cudaGetLastError();  // launch checks below must not see an earlier, unrelated error
    if (fault("launch")) return fail(GG_CUDA_ERROR, "injected launch failure");
    const unsigned extra = fault("barrier") ? 1u : 0u;
    const size_t lv = (size_t)cap_req + 1;
    uint64_t d2h = e->off_counts + (size_t)std::max(nb, nb_plain) * stride * sizeof(unsigned long long);
    if (wvc) d2h += (size_t)nb * stride * sizeof(unsigned);
    if (want_ns) d2h += lv * sizeof(unsigned long long);
    // Walk pass for this evaluation: not with the WVC masks or the distance planes
    // (their per-level bookkeeping lives in the level loop), at most the level cap.
    // Not with sweep_kernel either, whose rows are where the walk of all batches would put its.
    int walk_K = 0, launches = e->sweep_list ? 3 : 4;
    void *wall = nullptr;
    // What the level loop needs before it is enqueued or replayed.
    auto loop_ready = [&]() -> gg_status {
        gg_status ls = loop_room(e);
        if (ls != GG_OK) return ls;
        if (e->p_dirty) {
            // New buffers, or a launch that stopped early: the push buffers are
            // zero again only after these four writes.
            const size_t vbytes = (size_t)e->items * sizeof(uint4), fbytes = (size_t)((e->items + 31) / 32) * 4;
            GG_CK(cudaMemsetAsync(e->d_P0, 0, vbytes, st));
            GG_CK(cudaMemsetAsync(e->d_P1, 0, vbytes, st));
            GG_CK(cudaMemsetAsync(e->d_pf0, 0, fbytes, st));
            GG_CK(cudaMemsetAsync(e->d_pf1, 0, fbytes, st));
        }
        e->p_dirty = true;  // until the launch is known to have finished cleanly
        walk_K = (wvc || (x && (x->planes || within))) ? 0 : std::min(e->walk_K, cap_req);
        // (one level less where the walk of all batches then covers them: a level costs less
        // than a walk pass per batch)
        if (walk_K == 4 && e->walk_auto && walk_all_for(e, 3, nb_plain)) walk_K = 3;
        launches = 1 + ((long long)e->rows * e->d > 0 ? 1 : 0) + (walk_K > 0 ? 1 : 0) + (walk_K >= 3 ? 1 : 0);
        wall = walk_K > 0 ? walk_all_for(e, walk_K, nb_plain) : nullptr;
        return GG_OK;
    };
    if (!sweep) {
        s = loop_ready();
        if (s != GG_OK) return s;
    }

    // Everything the GPU does for one evaluation, on `q`: status words zeroed,
    // table -> adjacency (checked), one cooperative launch for every source
    // batch, and one copy back of the status block.
    // The timing events are recorded here only when launching directly; a
    // replayed graph is timed by events recorded around its launch.
    auto enqueue = [&](cudaStream_t q, bool timed) -> gg_status {
        if (timed) GG_CK(cudaEventRecord(e->ev0, q));
        // control block, range-check and symmetry words
        // (and, when a walk adds into them before any grid barrier, the levels run and the counts)
        GG_CK(cudaMemsetAsync(e->d_status, 0,
                              sweep || walk_K > 0 ? e->off_counts + (size_t)nb * stride * sizeof(unsigned long long)
                                         : sizeof(Ctl) + 4 * sizeof(int), q));   // ctl, bad, asym, wasym, redo
        const long long n = (long long)e->rows * e->d;
        if (e->form == FORM_GRAPH && within) {
            // read in place
        } else if (e->form == FORM_GRAPH) {
            if (d_table_in != e->d_table)
                GG_CK(cudaMemcpyAsync(e->d_table, d_table_in, e->table_elems * 4, cudaMemcpyDeviceToDevice, q));
            if (n > 0) {
                gg::check_table_kernel<<<(int)std::min<long long>((n + 255) / 256, 4096), 256, 0, q>>>(
                    e->d_table, n, e->rows, e->d_bad);
                GG_CK(cudaGetLastError());
            }
        } else if (n > 0) {
            launch_expand(e, d_table_in, q, sweep);
            GG_CK(cudaGetLastError());
        }
        if (want_ns)
            GG_CK(cudaMemsetAsync(e->d_level_ns, 0, lv * sizeof(unsigned long long), q));
        if (sweep) {
            const int K = e->sweep_K;
            uint4 *vall = sweep_in_f1(e, nb) ? e->d_F1 : e->d_vall;
            const SweepKernels k = sweep_for(e->d);
            GG_CK(cudaMemsetAsync(e->d_vtot, 0, (size_t)nb * 3 * sizeof(unsigned long long), q));
            if (e->sweep_list) {
                gg::SourceBallArgs ba{};
                ba.adj = e->d_adj;
                ba.src = e->d_src;
                ba.src_first = e->src_first;
                ba.ns_total = ns_all;
                ba.vall = reinterpret_cast<unsigned *>(vall);
                ba.counts = e->d_counts;
                ba.stride = stride;
                ba.oneway = e->d_wasym;
                ba.rows = e->rows; ba.nC = e->sweep_nC; ba.K = K;
                ba.list = e->sweep_ends;
                ba.ball_blocks = (ns_all + kSrcBallWarps - 1) / kSrcBallWarps;
                const size_t bsmem = kSrcBallWarps * (size_t)gg::source_ball_warp_bytes(e->rows, e->sweep_ends);
                const int check = (int)std::min<long long>((n + gg::kSrcBallBlock - 1) / gg::kSrcBallBlock, 16 * e->sms);
                void *bargs[] = {&ba};
                GG_CK(cudaLaunchKernel(k.source_ball, dim3(ba.ball_blocks + check), dim3(gg::kSrcBallBlock), bargs, bsmem, q));
            } else {
                // the level-2 lists, and with them (whole neighbour rows in a warp) the one-way check
                const long long nh = n * e->d;
                const int qd = e->d / 4;
                const bool h2_checks = e->d % 4 == 0 && (qd & (qd - 1)) == 0 && (nh / 4) % 32 == 0;
                gg::h2_kernel<<<(int)std::min<long long>((nh + 255) / 256, 8192), 256, 0, q>>>(
                    e->d_adj, e->d_h2, e->rows, e->d, e->form == FORM_GRAPH ? e->d_bad : nullptr,
                    h2_checks ? e->d_wasym : nullptr);
                GG_CK(cudaGetLastError());
                if (!h2_checks) {
                    gg::walk_check_kernel<<<(int)std::min<long long>((n + 255) / 256, 8192), 256, 0, q>>>(
                        e->d_adj, e->rows, e->d, e->d_wasym, e->form == FORM_GRAPH ? e->d_bad : nullptr);
                    GG_CK(cudaGetLastError());
                }
                gg::BallArgs ba{};
                ba.adj = e->d_adj;
                ba.h2 = e->d_h2;
                ba.bad = e->form == FORM_GRAPH ? e->d_bad : nullptr;
                ba.oneway = e->d_wasym;
                ba.vall = vall;
                ba.counts = e->d_counts;
                ba.stride = stride;
                ba.rows = e->rows; ba.nC = e->sweep_nC; ba.nb = nb;
                const size_t bsmem = ball_smem(e);
                int per_sm = 0;
                GG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k.ball, gg::kBallBlock, bsmem));
                const int warps = gg::kBallBlock / 32;
                const int bgrid = std::min((e->rows + warps - 1) / warps, e->sms * std::max(per_sm, 1));
                void *bargs[] = {&ba};
                GG_CK(cudaLaunchKernel(k.ball, dim3(bgrid), dim3(gg::kBallBlock), bargs, bsmem, q));
            }
            gg::SweepArgs sa{};
            sa.adj = e->d_adj;
            sa.bad = e->form == FORM_GRAPH ? e->d_bad : nullptr;
            sa.oneway = e->d_wasym;
            sa.vall = vall;
            sa.A = e->sweep_nC > e->nC ? e->d_swA : e->d_V;
            sa.B = e->sweep_nC > e->nC ? e->d_swB : e->d_F0;
            sa.ctl = e->d_ctl;
            sa.expected = (unsigned)e->sms;
            sa.wait_ns = e->wait_ns;
            sa.counts = e->d_counts;
            sa.vtot = e->d_vtot;
            sa.stride = stride;
            sa.levels_run = e->d_levels_run;
            sa.batch_ns = e->d_batch_ns;
            sa.redo = e->d_redo;
            sa.rows = e->rows; sa.nC = e->sweep_nC; sa.nb = nb; sa.K = K;
            sa.max_levels = cap_req;
            sa.ns_total = ns_all;
            sa.all = e->sweep_list ? 0 : 1;
            while ((1 << sa.sh) < sa.nC) ++sa.sh;
            sa.thin_ppm = e->sweep_list ? 0 : kSweepThinPpm;
            sa.last_ppm = sweep_last_ppm(e->d);
            const bool wide = sa.nC % 32 == 0;
            const int rows_tile = wide ? 1 : 32 / sa.nC;
            const int per = ((e->rows + rows_tile - 1) / rows_tile + e->sms - 1) / e->sms * rows_tile;
            const size_t ssmem = (size_t)per * e->d * sizeof(int32_t);
            // two slices of the table a block: a level's and last_rows' (65536 rows of 8: 14 KB each)
            sa.adj_smem_rows = 2 * ssmem <= 38u << 10 ? per : 0;
            void *sargs[] = {&sa};
            GG_CK(cudaLaunchCooperativeKernel(wide ? k.wide : k.narrow, dim3(e->sms), dim3(gg::kSweepBlock), sargs,
                                              sa.adj_smem_rows ? 2 * ssmem : 0, q));
            if (timed) GG_CK(cudaEventRecord(e->ev1, q));
            GG_CK(cudaMemcpyAsync(e->h_status, e->d_status, e->off_counts + (size_t)nb * stride * 8,
                                  cudaMemcpyDeviceToHost, q));
            return GG_OK;
        }
        if (walk_K > 0) {
            GG_CK(cudaMemsetAsync(e->d_vtot, 0, (size_t)nb * 3 * sizeof(unsigned long long), q));
            // the walk of all batches needs the table's one-way flag first; h2_kernel
            // takes the check along when its warps see whole neighbour rows
            const long long nh = (long long)e->rows * e->d * e->d;
            const int qd = e->d / 4;
            const bool h2_checks = wall && walk_K >= 3 && e->d % 4 == 0 && (qd & (qd - 1)) == 0 && (nh / 4) % 32 == 0;
            if (walk_K >= 3) {
                gg::h2_kernel<<<(int)std::min<long long>((nh + 255) / 256, 8192), 256, 0, q>>>(
                    e->d_adj, e->d_h2, e->rows, e->d, e->form == FORM_GRAPH ? e->d_bad : nullptr,
                    h2_checks ? e->d_wasym : nullptr);
                GG_CK(cudaGetLastError());
            }
            // the walk index of this evaluation's sources and batches
            gg::WalkIndexArgs wi{};
            wi.adj = e->d_adj;
            wi.h2 = walk_K >= 3 ? e->d_h2 : nullptr;
            wi.inv = x && x->inv ? x->inv : e->d_inv;
            wi.src_first = x && x->inv ? 0 : e->src_first;
            wi.src_begin = s0;
            wi.ns_total = ns_all;
            const int sub = wall ? e->nC / 32 : 1;
            wi.S = wall ? 4096 : 128 * e->nC;
            wi.sub = sub;
            wi.div_S = FastDiv((uint32_t)wi.S);
            wi.nb = nb * sub;
            wi.K = walk_K;
            wi.rows = e->rows;
            wi.d = e->d;
            wi.cap = e->walk_cap;
            wi.ent = e->d_went;
            wi.off = e->d_woff;
            wi.off_stride = e->walk_off_stride;
            wi.bad = e->form == FORM_GRAPH ? e->d_bad : nullptr;
            wi.asym = e->walk_vpull && e->walk_own_skip ? e->d_wasym : nullptr;
            // one resident wave of blocks, each striding over the rows
            void *wk = wall ? wall : index_kernel_for(e->d);
            const size_t wsmem = wall ? (size_t)gg::walk_all_smem(walk_K) : 0;
            if (wall) {
                wi.vall = e->d_vall;
                wi.vall_fl = e->d_vall_fl;
                wi.counts = e->d_counts;
                wi.counts_stride = stride;
                // the table's one-way flag first: walk_all_kernel reads it to choose
                // how it counts, the level kernel whether dense levels read own chunks
                wi.asym = nullptr;
                wi.oneway = e->d_wasym;
                if (!h2_checks) {
                    const long long ne = (long long)e->rows * e->d;
                    gg::walk_check_kernel<<<(int)std::min<long long>((ne + 255) / 256, 8192), 256, 0, q>>>(
                        e->d_adj, e->rows, e->d, e->d_wasym, e->form == FORM_GRAPH ? e->d_bad : nullptr);
                    GG_CK(cudaGetLastError());
                }
            }
            int sms = 0, per_sm = 0;
            GG_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device));
            GG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, wk, gg::kIndexBlock, wsmem));
            const int wgrid = (int)std::max<long long>(1, std::min<long long>(((long long)e->rows + 7) / 8,
                                                                              (long long)sms * std::max(per_sm, 1)));
            void *wargs[] = {&wi};
            GG_CK(cudaLaunchKernel(wk, dim3(wgrid), dim3(gg::kIndexBlock), wargs, wsmem, q));
        }
        BfsArgs a{};
        a.adj = within ? d_table_in : e->d_adj;
        a.inv = x && x->inv ? x->inv : e->d_inv;
        a.src_first = x && x->inv ? 0 : e->src_first;
        if (x && x->planes) {
            a.planes = x->planes;
            a.nplanes = x->nplanes;
            a.plane_cols = (unsigned)(nb * e->nC);
            a.plane_stride = (unsigned long long)e->rows * a.plane_cols;
        }
        a.src_begin = s0;
        a.ns_total = ns_all;
        a.nb = nb;
        a.V = e->d_V; a.F0 = e->d_F0; a.F1 = e->d_F1;
        a.fl0 = e->d_fl0; a.fl1 = e->d_fl1;
        a.P0 = e->d_P0; a.P1 = e->d_P1; a.pf0 = e->d_pf0; a.pf1 = e->d_pf1;
        // Below ~1M chunks a pull level costs about one grid barrier anyway.
        a.push_ppm = (long long)items >= (long long)e->push_min_items ? e->push_ppm : 0;
        a.nf = e->d_nf;
        a.nf2 = e->d_nf2;
        a.asym = e->d_asym;
        a.counts = e->d_counts;
        a.masks = wvc ? e->d_masks : nullptr;
        a.stride = stride;
        a.levels_run = e->d_levels_run;
        a.level_ns = want_ns ? e->d_level_ns : nullptr;
        a.batch_ns = e->d_batch_ns;
        a.ctl = e->d_ctl;
        a.rows = e->rows; a.d = e->d; a.nC = nC; a.items = items;
        a.div_nc = FastDiv((uint32_t)nC);
        a.wcounts = within ? e->d_wcounts : nullptr;
        a.max_levels = cap_req;
        a.dense_w_ppm = e->dense_w_ppm;
        a.dense_r_ppm = e->dense_r_ppm;
        a.full_skip_ppm = e->full_skip_ppm;
        a.split_ppm = e->split_ppm;
        a.adj_smem_rows = e->adj_smem_rows;
        a.wait_ns = e->wait_ns;
        a.expected = (unsigned)e->grid + extra;
        a.bad = e->form == FORM_GRAPH ? e->d_bad : nullptr;
        a.walk_K = walk_K;
        a.walk_rpg = e->walk_rpg;
        a.walk_smem_off = e->walk_smem_off;
        a.walk_ent = e->d_went;
        a.walk_off = e->d_woff;
        a.walk_cap = e->walk_cap;
        a.walk_off_stride = e->walk_off_stride;
        a.walk_vpull = walk_K > 0 && !wvc ? e->walk_vpull : 0;
        a.walk_asym = a.walk_vpull && e->walk_own_skip ? e->d_wasym : nullptr;
        a.vtot = e->d_vtot;
        a.vall = wall ? e->d_vall : nullptr;
        a.vall_fl = wall ? e->d_vall_fl : nullptr;
        a.third = wall && e->walk_third ? e->d_F0 : nullptr;
        void *args[] = {&a};
        const int mode = a.planes ? gg::kPlanes : within ? gg::kWithin : gg::kPlain;
        GG_CK(cudaLaunchCooperativeKernel(kernel_for(e->d, mode), dim3(e->grid), dim3(gg::kBlock), args,
                                          wall ? (size_t)e->walk_smem_off : e->smem_bytes, q));
        if (timed) GG_CK(cudaEventRecord(e->ev1, q));
        // One copy back: control block, status words, per-batch levels and
        // times, and the counts of every batch (cap_req + 1 each).
        GG_CK(cudaMemcpyAsync(e->h_status, e->d_status, e->off_counts + (size_t)nb * stride * 8,
                              cudaMemcpyDeviceToHost, q));
        if (wvc)
            GG_CK(cudaMemcpyAsync(e->h_masks, e->d_masks, (size_t)nb * stride * sizeof(unsigned),
                                  cudaMemcpyDeviceToHost, q));
        if (within)
            GG_CK(cudaMemcpyAsync(e->h_wcounts, e->d_wcounts, (size_t)nb * stride * sizeof(unsigned long long),
                                  cudaMemcpyDeviceToHost, q));
        if (want_ns)
            GG_CK(cudaMemcpyAsync(e->h_level_ns, e->d_level_ns, lv * sizeof(unsigned long long),
                                  cudaMemcpyDeviceToHost, q));
        return GG_OK;
    };

    // Repeated evaluations of one shape replay a captured CUDA graph of the
    // same work (one launch call instead of about eight).  Anything that
    // changes the work -- the table pointer, the source range, the level cap,
    // the outputs asked for, reallocated buffers -- captures a new graph.
    const EvalKey key{d_table_in, e->d_status, e->d_V, x ? (const void *)x->inv : nullptr,
                      x ? (const void *)x->planes : nullptr, s0, ns_all, cap_req, wvc, want_ns, sweep};
    bool replayed = false;
    if (e->use_graph && !extra && !(x && x->no_graph)) {
        if (!e->graph_exec || !(key == e->graph_key)) {
            if (e->graph_exec) { cudaGraphExecDestroy(e->graph_exec); e->graph_exec = nullptr; }
            cudaGraph_t g = nullptr;
            gg_status cs = GG_CUDA_ERROR;
            if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
                cs = enqueue(st, false);
                const cudaError_t ce = cudaStreamEndCapture(st, &g);
                if (ce != cudaSuccess) cs = GG_CUDA_ERROR;
            }
            if (cs == GG_OK && g && cudaGraphInstantiate(&e->graph_exec, g, 0) == cudaSuccess) {
                e->graph_key = key;
            } else {
                e->graph_exec = nullptr;
                e->use_graph = false;   // this device or driver cannot capture it: launch directly
            }
            if (g) cudaGraphDestroy(g);
            (void)cudaGetLastError();
        }
        if (e->graph_exec) {
            GG_CK(cudaEventRecord(e->ev0, st));
            GG_CK(cudaGraphLaunch(e->graph_exec, st));
            GG_CK(cudaEventRecord(e->ev1, st));
            replayed = true;
        }
    }
    if (!replayed) {
        gg_status es = enqueue(st, true);
        if (es != GG_OK) return es;
    }
    e->last_d2h = d2h;
    GG_CK(cudaStreamSynchronize(st));
    float ms = 0.f;
    GG_CK(cudaEventElapsedTime(&ms, e->ev0, e->ev1));
    e->last_ms = ms;
    e->last_launches = launches;
    if (sweep && *e->h_redo && !*e->h_bad && !e->h_ctl->err) {
        sweep = false;
        e->sweep_wait = 63;
        const DirectPlan p = direct_plan(e, ns_all, wvc, false);
        if (p.W) {
            const double first_ms = e->last_ms;
            const int first_launches = e->last_launches;
            const gg_status ds = direct_eval(e, p, d_table_in, nullptr, o, s0, ns_all, cap_req, r, st);
            e->last_ms += first_ms;
            e->last_launches += first_launches;
            return ds;
        }
        nb = nb_plain;
        gg_status es = loop_ready();
        if (es == GG_OK) es = enqueue(st, true);
        if (es != GG_OK) return es;
        GG_CK(cudaStreamSynchronize(st));
        GG_CK(cudaEventElapsedTime(&ms, e->ev0, e->ev1));
        e->last_ms += ms;
        e->last_launches += launches;
    }
    e->last_batches = nb;

    if (e->form == FORM_GRAPH && !within && *e->h_bad)
        return fail(GG_BAD_ARG, "adjacency entry outside [0, N)");
    if (e->h_ctl->err)
        return fail(GG_TIMEOUT, "grid barrier wait exceeded its limit at level " +
                                    std::to_string(e->h_ctl->err_level));
    if (!sweep) e->p_dirty = false;

    // Exact fold of the per-batch level counters.
    gg_result R{};
    R.scale = e->scale;
    R.pairs = (uint64_t)ns_all * (uint64_t)e->rows;
    R.n_sources = ns_all;
    R.batches = nb;
    R.wvc = -1;
    std::vector<int> lev(nb, 0);
    std::vector<unsigned long long> agg(cap_req + 1, 0ull);
    for (int b = 0; b < nb; ++b) {
        const unsigned long long *c = e->h_counts + (size_t)b * stride;
        const int run = e->h_levels_run[b];
        int last = 0;
        // (sweep: a batch's own counts may be negative mod 2^64, their sums are not)
        for (int L = 0; L <= run && L <= cap_req; ++L) {
            R.reached += c[L];
            R.total += (uint64_t)L * c[L];
            agg[L] += c[L];
            if (L > 0 && c[L]) last = L;
        }
        lev[b] = last;
        R.level_steps += run;
        R.levels = std::max(R.levels, last);
        if (run >= cap_req && c[cap_req]) R.capped = 1;
    }
    R.connected = (!R.capped && R.reached == R.pairs) ? 1 : 0;
    if (within) {
        x->within[0] = x->within[1] = 0;
        for (int b = 0; b < nb; ++b)
            for (int L = 0; L <= e->h_levels_run[b] && L <= cap_req; ++L) {
                const unsigned long long c = e->h_wcounts[(size_t)b * stride + L];
                x->within[0] += (uint64_t)L * c;
                x->within[1] += c;
            }
    }
    if (wvc) {
        // Lane-aggregated completion masks across batches: a batch's mask stays
        // at its final value after its last level.
        auto mask_at = [&](int L) {
            unsigned m = 0xffffffffu;
            for (int b = 0; b < nb; ++b)
                m &= e->h_masks[(size_t)b * stride + std::min(L, lev[b])];
            return m;
        };
        const int E = R.levels;
        R.wvc = E > 0 ? __builtin_popcount(mask_at(E - 1) ^ mask_at(E)) : 0;
    }
    if (o && o->level_counts)
        std::memcpy(o->level_counts, agg.data(), (size_t)(cap_req + 1) * sizeof(uint64_t));
    if (want_ns)
        std::memcpy(o->level_ns, e->h_level_ns, (size_t)(cap_req + 1) * sizeof(uint64_t));
    *r = R;
    return GG_OK;
}

// A host table into the pinned staging buffer, split over a few threads when it is
// large (one thread's copy bounded a 2 MiB table at about 0.1 ms a call).
void copy_to_pinned(void *dst, const void *src, size_t bytes) {
    constexpr size_t kPart = 256u << 10;
    const int parts = (int)std::min<size_t>(8, bytes / kPart);
    if (parts <= 1) {
        std::memcpy(dst, src, bytes);
        return;
    }
#pragma omp parallel for num_threads(parts) schedule(static)
    for (int i = 0; i < parts; ++i) {
        const size_t lo = bytes * (size_t)i / (size_t)parts, hi = bytes * (size_t)(i + 1) / (size_t)parts;
        std::memcpy(static_cast<char *>(dst) + lo, static_cast<const char *>(src) + lo, hi - lo);
    }
}

// A plain graph's table as checked 16-bit ids in pinned memory, by a few threads when it is
// large; false: an entry outside [0, rows).
bool pack16(uint16_t *dst, const int32_t *src, size_t n, int rows) {
    constexpr size_t kPart = 16u << 10;
    const int parts = (int)std::min<size_t>(8, std::max<size_t>(1, n / kPart));
    unsigned bad = 0u;
    auto range = [&](size_t lo, size_t hi) {
        unsigned b = 0u;
        for (size_t k = lo; k < hi; ++k) {
            const unsigned x = (unsigned)src[k];
            b |= x >= (unsigned)rows ? 1u : 0u;
            dst[k] = (uint16_t)x;
        }
        return b;
    };
    if (parts <= 1) return range(0, n) == 0u;
#pragma omp parallel for num_threads(parts) schedule(static) reduction(| : bad)
    for (int i = 0; i < parts; ++i) bad |= range(n * (size_t)i / (size_t)parts, n * (size_t)(i + 1) / (size_t)parts);
    return bad == 0u;
}

// Host table of a plain graph small enough for direct_kernel with its rows in shared
// memory: half the bytes to copy, and none where the few blocks of a small graph read
// them over the bus at less than a copy command costs (n = 256, d = 4: 2 KB, 8 blocks).
constexpr size_t kZeroCopyTotal = 128u << 10;

gg_status direct_host(gg_engine *e, const DirectPlan &p, const int32_t *table, const gg_eval_opts *o, gg_result *r) {
    const size_t n = e->table_elems, bytes = (n * 2 + 15) / 16 * 16;
    if (!e->h_pack) {
        GG_CK(cudaMallocHost(&e->h_pack, std::max<size_t>(bytes, 16)));
        GG_CK(cudaMalloc(&e->d_pack, std::max<size_t>(bytes, 16)));
        std::memset(e->h_pack, 0, std::max<size_t>(bytes, 16));
    }
    e->table_stale = true;
    if (!pack16(e->h_pack, table, n, e->rows)) return fail(GG_BAD_ARG, "adjacency entry outside [0, N)");
    const uint16_t *from = e->h_pack;
    if (bytes * (size_t)p.grid > kZeroCopyTotal) {
        GG_CK(cudaMemcpyAsync(e->d_pack, e->h_pack, bytes, cudaMemcpyHostToDevice, e->stream));
        from = e->d_pack;
    }
    const int cap = (o && o->max_levels > 0) ? o->max_levels : std::max(e->rows, 1);
    gg_status s = direct_eval(e, p, nullptr, from, o, 0, (int)e->reps.size(), cap, r, e->stream);
    e->last_h2d = n * 2;
    return s;
}

gg_status eval_host(gg_engine *e, const int32_t *table, const gg_eval_opts *o, gg_result *r) {
    if (!e || !r) return fail(GG_BAD_ARG, "null engine or result");
    if (e->table_elems && !table) return fail(GG_BAD_ARG, "null table");
    GG_CK(cudaSetDevice(e->device));
    e->table_stale = false;
    int sweep = -1;
    if (e->form == FORM_GRAPH && e->table_elems && !(o && (o->level_ns || o->src_begin || o->src_end || o->want_wvc)) &&
        !fault("barrier")) {
        sweep = sweep_turn(e, o);
        const DirectPlan p = direct_plan(e, (int)e->reps.size(), false, sweep);
        if (p.W && p.adj_smem) return direct_host(e, p, table, o, r);
    }
    if (e->table_elems) {
        copy_to_pinned(e->h_table, table, e->table_elems * sizeof(int32_t));
        GG_CK(cudaMemcpyAsync(e->d_table, e->h_table, e->table_elems * sizeof(int32_t),
                              cudaMemcpyHostToDevice, e->stream));
    }
    gg_status s = run_eval(e, e->d_table, o, r, e->stream, nullptr, sweep);
    e->last_h2d = e->table_elems * sizeof(int32_t);
    return s;
}

double aspl_of(uint64_t total, uint64_t scale, int N) {
    // total *= N/M; double(total)/(int64_t(N)*(N-1))  (cudaASPLconv.cu:241-242)
    const int64_t t = (int64_t)(total * scale);
    return double(t) / (int64_t(N) * (N - 1));
}

// The level loop `for(step=1; step<100; ...)` of cudaASPLconv::diameterASPL and
// its piece/box twins (cudaASPLconv.cu:208-242, cudaASPLpiece.cu:181-215,
// cudaASPLbox.cu:191-225).
gg_status lifted_diameter_aspl(gg_engine *e, const int32_t *table, int *diameter, double *aspl) {
    if (!diameter || !aspl) return fail(GG_BAD_ARG, "null output");
    gg_eval_opts o{};
    o.max_levels = 99;
    gg_result r;
    gg_status s = eval_host(e, table, &o, &r);
    if (s != GG_OK) return s;
    if (r.capped) {  // step 99 still found pairs: loop ends, diameter stays 1e8
        *diameter = kSentinel;
        *aspl = aspl_of(r.total, r.scale, e->N);
    } else if (!r.connected) {
        *diameter = kSentinel;
        *aspl = 100000000.0;
    } else {
        *diameter = r.levels;
        *aspl = aspl_of(r.total, r.scale, e->N);
    }
    return GG_OK;
}

}  // namespace

namespace gg {
gg_status engine_eval(gg_engine *e, const int32_t *d_table, const gg_eval_opts *o, gg_result *r,
                      cudaStream_t st, const EvalExtra *x) {
    if (!e || !r || !d_table) return fail(GG_BAD_ARG, "null argument");
    GG_CK(cudaSetDevice(e->device));
    return run_eval(e, d_table, o, r, st ? st : e->stream, x);
}
gg_status graph_engine(int n, int d, int device, gg_engine **out) { return graph_create(n, d, device, true, out); }

int engine_plane_cols(const gg_engine *e) {
    const int n_src = (int)e->reps.size();
    return ((n_src + e->batch_bits - 1) / e->batch_bits) * e->nC;
}
}  // namespace gg

extern "C" {

int gg_abi_version(void) { return GG_ABI_VERSION; }

const char *gg_status_str(gg_status s) {
    switch (s) {
        case GG_OK: return "ok";
        case GG_BAD_ARG: return "bad argument";
        case GG_CUDA_ERROR: return "CUDA error";
        case GG_TIMEOUT: return "bounded wait timed out";
        case GG_OUT_OF_MEMORY: return "out of memory";
        case GG_NO_DEVICE: return "no device";
    }
    return "unknown status";
}

const char *gg_last_error(void) { return g_err.c_str(); }

gg_status gg_graph_create(int N, int degree_max, int device, gg_engine **out) {
    return graph_create(N, degree_max, device, false, out);
}

gg_status gg_conv_create(int N, int M, int degree, int device, gg_engine **out) {
    if (!out) return fail(GG_BAD_ARG, "null out");
    *out = nullptr;
    if (N < 1 || M < 1 || M > N || degree < 0) return fail(GG_BAD_ARG, "need 1 <= M <= N, degree >= 0");
    gg_engine *e = new gg_engine();
    e->form = FORM_PART; e->device = device;
    e->N = N; e->M = M; e->d = degree; e->rows = N; e->scale = (uint64_t)(N / M);
    e->table_elems = (size_t)M * degree;
    e->reps.resize(M);
    for (int i = 0; i < M; ++i) e->reps[i] = i;
    return finish_create(e, out);
}

gg_status gg_beamer_create(int N, int M, int degree, int device, gg_engine **out) {
    if (!out) return fail(GG_BAD_ARG, "null out");
    *out = nullptr;
    if (N < 1 || M < 1 || M > N || degree < 0 || N > kBeamerRows)
        return fail(GG_BAD_ARG, "need 1 <= M <= N <= 10^6, degree >= 0");
    gg_engine *e = new gg_engine();
    e->form = FORM_PART; e->device = device;
    e->N = N; e->M = M; e->d = degree; e->rows = kBeamerRows; e->scale = (uint64_t)(N / M);
    e->table_elems = (size_t)M * degree;
    e->reps.resize(M);
    for (int i = 0; i < M; ++i) e->reps[i] = i;
    return finish_create(e, out);
}

gg_status gg_piece_create(int Nx, int Ny, int Mx, int My, int degree, int device, gg_engine **out) {
    if (!out) return fail(GG_BAD_ARG, "null out");
    *out = nullptr;
    if (Nx < 1 || Ny < 1 || Mx < 1 || My < 1 || Mx > Nx || My > Ny || degree < 0 ||
        (long long)Nx * Ny >= (1ll << 31))
        return fail(GG_BAD_ARG, "need 1 <= Mx <= Nx, 1 <= My <= Ny, degree >= 0");
    gg_engine *e = new gg_engine();
    e->form = FORM_PIECE; e->device = device;
    e->dims[0] = Nx; e->dims[1] = Ny; e->dims[2] = 1; e->dims[3] = Mx; e->dims[4] = My; e->dims[5] = 1;
    e->N = Nx * Ny; e->M = Mx * My; e->d = degree; e->rows = e->N;
    e->scale = (uint64_t)(e->N / e->M);
    e->table_elems = (size_t)e->M * degree * 2;
    // representatives: corner tile, source index x*My+y (cudaASPLpiece.cu:23-29)
    for (int x = 0; x < Mx; ++x)
        for (int y = 0; y < My; ++y) e->reps.push_back(x * Ny + y);
    return finish_create(e, out);
}

gg_status gg_box_create(int Nx, int Ny, int Nz, int Mx, int My, int Mz, int degree, int device,
                        gg_engine **out) {
    if (!out) return fail(GG_BAD_ARG, "null out");
    *out = nullptr;
    if (Nx < 1 || Ny < 1 || Nz < 1 || Mx < 1 || My < 1 || Mz < 1 || Mx > Nx || My > Ny || Mz > Nz ||
        degree < 0 || (long long)Nx * Ny * Nz >= (1ll << 31))
        return fail(GG_BAD_ARG, "need 1 <= M* <= N*, degree >= 0");
    gg_engine *e = new gg_engine();
    e->form = FORM_BOX; e->device = device;
    e->dims[0] = Nx; e->dims[1] = Ny; e->dims[2] = Nz; e->dims[3] = Mx; e->dims[4] = My; e->dims[5] = Mz;
    e->N = Nx * Ny * Nz; e->M = Mx * My * Mz; e->d = degree; e->rows = e->N;
    e->scale = (uint64_t)(e->N / e->M);
    e->table_elems = (size_t)e->M * degree * 3;
    // representatives: corner tile, source index (x*My+y)*Mz+z (cudaASPLbox.cu:25-32)
    for (int x = 0; x < Mx; ++x)
        for (int y = 0; y < My; ++y)
            for (int z = 0; z < Mz; ++z) e->reps.push_back((x * Ny + y) * Nz + z);
    return finish_create(e, out);
}

gg_status gg_destroy(gg_engine *e) {
    destroy_all(e);
    return GG_OK;
}


gg_status gg_eval(gg_engine *e, const int32_t *table, const gg_eval_opts *opts, gg_result *out) {
    return eval_host(e, table, opts, out);
}

gg_status gg_eval_device(gg_engine *e, const int32_t *d_table, const gg_eval_opts *opts,
                         gg_result *out, void *stream) {
    if (!e || !out) return fail(GG_BAD_ARG, "null engine or result");
    if (e->table_elems && !d_table) return fail(GG_BAD_ARG, "null table");
    GG_CK(cudaSetDevice(e->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : e->stream;
    gg_status s = run_eval(e, d_table ? d_table : e->d_table, opts, out, st);
    e->last_h2d = 0;
    return s;
}

gg_status gg_last_transfer_bytes(gg_engine *e, uint64_t *h2d, uint64_t *d2h) {
    if (!e || !h2d || !d2h) return fail(GG_BAD_ARG, "null argument");
    *h2d = e->last_h2d;
    *d2h = e->last_d2h;
    return GG_OK;
}

gg_status gg_last_device_ms(gg_engine *e, double *ms) {
    if (!e || !ms) return fail(GG_BAD_ARG, "null argument");
    *ms = e->last_ms;
    return GG_OK;
}

gg_status gg_last_batch_ns(gg_engine *e, uint64_t *ns, int n) {
    if (!e || !ns || n < 0) return fail(GG_BAD_ARG, "bad arguments");
    for (int b = 0; b < n && b < e->last_batches; ++b) {
        ns[2 * b] = e->h_batch_ns[2 * b];
        ns[2 * b + 1] = e->h_batch_ns[2 * b + 1];
    }
    return GG_OK;
}

gg_status gg_last_launches(gg_engine *e, int *launches) {
    if (!e || !launches) return fail(GG_BAD_ARG, "null argument");
    *launches = e->last_launches;
    return GG_OK;
}

gg_status gg_set_batch_sources(gg_engine *e, int sources) {
    if (!e || sources < 0) return fail(GG_BAD_ARG, "bad batch width");
    GG_CK(cudaSetDevice(e->device));
    GG_CK(cudaStreamSynchronize(e->stream));
    e->direct = sources == 0 && e->direct_allowed;   // an explicit width runs the batches it asks for
    e->width_asked = sources > 0;
    const gg_status s = plan(e, sources);
    return s == GG_OK ? loop_room(e) : s;
}

gg_status gg_autotune(gg_engine *e, const int32_t *table, int trials, int *best_sources, double *best_ms) {
    if (!e || (e->table_elems && !table) || trials < 1) return fail(GG_BAD_ARG, "bad arguments");
    GG_CK(cudaSetDevice(e->device));
    GG_CK(cudaStreamSynchronize(e->stream));
    const int n_src = (int)e->reps.size();
    struct Planned {   // the shapes timed here are bfs_batch_kernel's
        gg_engine *e;
        bool direct, sweep;
        ~Planned() { e->direct = direct; e->sweep = sweep; }
    } planned{e, e->direct, e->sweep};
    e->direct = e->sweep = e->width_asked = false;
    // the L2-resident width the default plan picks, and its neighbours
    int base = 0, max_bps = 0;
    {
        const int keep = e->batch_bits, keep_bps = e->bps_cap, keep_walk = e->walk_pref;
        e->bps_cap = 0;
        e->walk_pref = -1;
        gg_status s = plan(e, 0);
        if (s != GG_OK) return s;
        base = e->batch_bits;
        GG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&max_bps, kernel_for(e->d), gg::kBlock,
                                                            e->smem_bytes));
        e->bps_cap = keep_bps;
        e->walk_pref = keep_walk;
        if (keep > 0) { s = plan(e, keep); if (s != GG_OK) return s; }
    }
    std::vector<int> widths;
    for (double f : {0.25, 0.5, 1.0, 2.0, 4.0}) {
        int w = (int)(base * f);
        w = std::max(128, std::min(((w + 127) / 128) * 128, ((n_src + 127) / 128) * 128));
        widths.push_back(w);
    }
    widths.push_back(((n_src + 127) / 128) * 128);
    std::sort(widths.begin(), widths.end());
    widths.erase(std::unique(widths.begin(), widths.end()), widths.end());
    std::vector<int> bps_opts;   // 0 = as many as fit, then one and two fewer
    bps_opts.push_back(0);
    for (int k = 1; k <= 2; ++k)
        if (max_bps - k >= 1) bps_opts.push_back(max_bps - k);
    if (e->table_elems) {
        copy_to_pinned(e->h_table, table, e->table_elems * sizeof(int32_t));
        GG_CK(cudaMemcpyAsync(e->d_table, e->h_table, e->table_elems * sizeof(int32_t),
                              cudaMemcpyHostToDevice, e->stream));
    }
    int best = 0, best_bps = 0, best_walk = -1;
    double best_t = 1e300;
    gg_result r;
    for (int w : widths) {
        if ((long long)e->rows * (w / 128) >= (1ll << 31)) continue;
        for (int bps : bps_opts) {
            bool auto_walks = true;
            for (int walk : {-1, 0}) {
                if (walk == 0 && !auto_walks) continue;   // the automatic plan has no walk already
                e->bps_cap = bps;
                e->walk_pref = walk;
                gg_status s = plan(e, w);
                if (s == GG_OK) s = loop_room(e);
                if (s == GG_OUT_OF_MEMORY) { (void)cudaGetLastError(); break; }  // too wide for this device
                if (s != GG_OK) return s;
                if (walk == -1) auto_walks = e->walk_K > 0;
                s = run_eval(e, e->d_table, nullptr, &r, e->stream);  // warm
                if (s != GG_OK) return s;
                double t = 1e300;
                for (int k = 0; k < trials; ++k) {
                    s = run_eval(e, e->d_table, nullptr, &r, e->stream);
                    if (s != GG_OK) return s;
                    t = std::min(t, e->last_ms);
                }
                if (t < best_t) { best_t = t; best = w; best_bps = bps; best_walk = walk; }
            }
        }
    }
    if (!best) return fail(GG_OUT_OF_MEMORY, "no batch width fits");
    e->bps_cap = best_bps;
    e->walk_pref = best_walk;
    e->sweep = planned.sweep;
    gg_status s = plan(e, best);
    if (s != GG_OK) return s;
    gg::tune_put(engine_tune_key(e), {best, best_bps, best_walk});
    if (best_sources) *best_sources = best;
    if (best_ms) *best_ms = best_t;
    return GG_OK;
}

gg_status gg_engine_plan(gg_engine *e, int *batch_sources, int *blocks_per_sm, int *walk_levels) {
    if (!e) return fail(GG_BAD_ARG, "null engine");
    if (batch_sources) *batch_sources = e->batch_bits;
    if (blocks_per_sm) *blocks_per_sm = e->grid;
    if (walk_levels) *walk_levels = e->walk_K;
    int sms = 0;
    if (blocks_per_sm && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device) == cudaSuccess &&
        sms > 0)
        *blocks_per_sm = (e->grid + sms - 1) / sms;
    else
        (void)cudaGetLastError();
    return GG_OK;
}

gg_status gg_set_wait_limit_ms(gg_engine *e, int ms) {
    if (!e || ms < 1) return fail(GG_BAD_ARG, "bad wait limit");
    e->wait_ns = (long long)ms * 1000000ll;
    invalidate_graph(e);
    return GG_OK;
}

// cudaASPLgraph::calc (cudaASPLgraph.cu:141-199)
gg_status gg_graph_calc(gg_engine *e, const int32_t *adj, int *diameter, int64_t *total) {
    if (!e || !diameter || !total) return fail(GG_BAD_ARG, "null argument");
    if (e->form != FORM_GRAPH) return fail(GG_BAD_ARG, "not a graph engine");
    gg_eval_opts o{};
    o.max_levels = 199;
    gg_result r;
    gg_status s = eval_host(e, adj, &o, &r);
    if (s != GG_OK) return s;
    if (!r.capped && r.connected) {
        *diameter = r.levels;
        *total = (int64_t)r.total;
        return GG_OK;
    }
    if (e->table_stale) {
        copy_to_pinned(e->h_table, adj, e->table_elems * sizeof(int32_t));
        GG_CK(cudaMemcpyAsync(e->d_table, e->h_table, e->table_elems * sizeof(int32_t), cudaMemcpyHostToDevice, e->stream));
        e->table_stale = false;
    }
    // Some source hits the 199-step limit or misses a vertex: the reference
    // answers for the first 1024-source chunk (in source order) that does
    // either, so resolve chunk by chunk with the table already on the device.
    for (int off = 0; off < e->N; off += 1024) {
        gg_eval_opts c{};
        c.max_levels = 199;
        c.src_begin = off;
        c.src_end = std::min(off + 1024, e->N);
        gg_result rc;
        s = run_eval(e, e->d_table, &c, &rc, e->stream);
        if (s != GG_OK) return s;
        if (rc.capped) { *diameter = -2; *total = -2; return GG_OK; }
        if (!rc.connected) { *diameter = -1; *total = -1; return GG_OK; }
    }
    return fail(GG_CUDA_ERROR, "inconsistent chunk resolution");
}

gg_status gg_conv_calc(gg_engine *e, const int32_t *diffs, double *aspl) {
    if (!e || !aspl) return fail(GG_BAD_ARG, "null argument");
    gg_eval_opts o{};
    o.max_levels = 99;
    gg_result r;
    gg_status s = eval_host(e, diffs, &o, &r);
    if (s != GG_OK) return s;
    if (!r.capped && !r.connected) *aspl = 1e9;  // cudaASPLconv.cu:182
    else *aspl = aspl_of(r.total, r.scale, e->N);
    return GG_OK;
}

gg_status gg_conv_diameter_aspl(gg_engine *e, const int32_t *diffs, int *diameter, double *aspl) {
    if (!e) return fail(GG_BAD_ARG, "null engine");
    if (e->form != FORM_PART) return fail(GG_BAD_ARG, "not a part engine");
    return lifted_diameter_aspl(e, diffs, diameter, aspl);
}

// cudaASPLconv::WVCdiameterASPL (cudaASPLconv.cu:244-308)
gg_status gg_conv_wvc_diameter_aspl(gg_engine *e, const int32_t *diffs, int *wvc, int *diameter,
                                    double *aspl) {
    if (!e || !wvc || !diameter || !aspl) return fail(GG_BAD_ARG, "null argument");
    if (e->form != FORM_PART) return fail(GG_BAD_ARG, "not a part engine");
    gg_eval_opts o{};
    o.max_levels = 100;
    o.want_wvc = 1;
    gg_result r;
    gg_status s = eval_host(e, diffs, &o, &r);
    if (s != GG_OK) return s;
    if (r.capped || !r.connected) {
        *wvc = kSentinel; *diameter = kSentinel; *aspl = 100000000.0;
    } else {
        *wvc = r.wvc; *diameter = r.levels; *aspl = aspl_of(r.total, r.scale, e->N);
    }
    return GG_OK;
}

gg_status gg_piece_diameter_aspl(gg_engine *e, const int32_t *vals, int *diameter, double *aspl) {
    if (!e) return fail(GG_BAD_ARG, "null engine");
    if (e->form != FORM_PIECE) return fail(GG_BAD_ARG, "not a piece engine");
    return lifted_diameter_aspl(e, vals, diameter, aspl);
}

gg_status gg_box_diameter_aspl(gg_engine *e, const int32_t *vals, int *diameter, double *aspl) {
    if (!e) return fail(GG_BAD_ARG, "null engine");
    if (e->form != FORM_BOX) return fail(GG_BAD_ARG, "not a box engine");
    return lifted_diameter_aspl(e, vals, diameter, aspl);
}

// cudaASPLbeamer::calc (cudaASPLbeamer.cu:71-84)
gg_status gg_beamer_calc(gg_engine *e, const int32_t *diffs, int regular, double *aspl) {
    if (!e || !aspl) return fail(GG_BAD_ARG, "null argument");
    if (e->form != FORM_PART || e->rows != kBeamerRows) return fail(GG_BAD_ARG, "not a beamer engine");
    if (!regular) { *aspl = 100000000; return GG_OK; }
    gg_eval_opts o{};
    o.max_levels = kBeamerLevels;
    gg_result r;
    gg_status s = eval_host(e, diffs, &o, &r);
    if (s != GG_OK) return s;
    *aspl = aspl_of(r.total, r.scale, e->N);
    return GG_OK;
}

}  // extern "C"
