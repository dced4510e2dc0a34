// gg_inc.cu -- incremental exact evaluation of 2-opt moves on one plain graph.
//
// A full evaluation of the current graph also writes its distance matrix as
// bit-planes (4 planes: distances up to 15).  A 2-opt move (remove (a,b), (c,d);
// add (a,p), (b,q)) changes the distances from source s only if
//   * a removed edge joins two consecutive BFS levels of s and its deeper end has
//     no other neighbour on the shallower level (else every vertex keeps a parent
//     one level up, and by induction over the levels no distance grows), or
//   * an added edge joins vertices whose distances from s differ by 2 or more
//     (else no path gets shorter).
// Of those sources, the ones within floor((diameter - 1) / 2) of an endpoint of the move
// are searched again on the new graph (T; gg_batch.cu states why they see every changed
// pair): with w = 1 for vertices of T and 2 for the others, the new total is the old one
// plus the sum over s in T and every v of w(v) (new - old distance).  The engine counts
// the pairs inside T apart; T's old sums come from per-source distance sums kept for the
// current graph (row reductions, gg_planes.cuh) and from the plane rows of T.  The new
// diameter is the larger of the largest new distance from T and the largest old distance
// between vertices outside T.  Exact whenever the current graph is symmetric and
// connected with diameter <= 15; otherwise a call evaluates the moved graph in full.
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "gg.h"
#include "gg_internal.h"
#include "gg_kernels.cuh"
#include "gg_planes.cuh"

namespace {

constexpr int kPlanes = 4;

struct IncStatus {
    unsigned long long old_sum;   // distance sums of T (current graph)
    unsigned long long tt_sum;    // distances within T (current graph)
    unsigned long long tops;      // pairs (T, any) at the current diameter (up to n^2)
    unsigned affected;            // affected sources
    unsigned count;               // |T|
    int found;                    // outside_at's answer
};

struct IncArgs {
    const uint32_t *planes;       // plane words (vertex x, sources 32w..): [k * ps + x * cw + w]
    size_t ps, cw;
    const int32_t *adj;           // the current graph
    int n, d;
    gg_swap sw;
    unsigned radius;
    const unsigned *rowsum, *ecc, *top;
    int32_t *inv;                 // [n]: place in T, or -1
    uint32_t *tbits;              // [cw]: bit v: v in T (zero past the last vertex)
    int32_t *list;                // T
    IncStatus *st;
};

// A block of four warps per 1024 sources, a warp per endpoint (edit_masks): T, its list,
// inverse list and bits, and the old sums.  26 us with one thread a source gathering the
// plane bits one by one (n = 65536, d = 8).
__global__ void __launch_bounds__(128) inc_select(const IncArgs a) {
    __shared__ uint32_t s_aff[4][32], s_near[4][32];
    const unsigned lane = threadIdx.x & 31u;
    const int i = (int)(threadIdx.x >> 5);
    const gg_swap &sw = a.sw;
    const unsigned words = ((unsigned)a.n + 31u) / 32u, w = blockIdx.x * 32u + lane;
    const bool in = w < words;
    const int r = i == 0 ? sw.a : i == 1 ? sw.b : i == 2 ? sw.c : sw.d;
    const int f = i == 0 ? sw.b : i == 1 ? sw.a : i == 2 ? sw.d : sw.c;
    const int t = i == 0 ? (sw.mode ? sw.d : sw.c) : i == 1 ? (sw.mode ? sw.c : sw.d)
                : i == 2 ? (sw.mode ? sw.b : sw.a) : (sw.mode ? sw.a : sw.b);
    edit_masks(a.planes, a.ps, a.cw, a.adj, a.d, r, f, t, in ? w : 0u, a.radius, s_aff[i][lane], s_near[i][lane]);
    __syncthreads();
    uint32_t aff = s_aff[0][lane] | s_aff[1][lane] | s_aff[2][lane] | s_aff[3][lane];
    if (!in) aff = 0u;
    else if (w == words - 1u && (a.n & 31)) aff &= (1u << (a.n & 31)) - 1u;
    const uint32_t go = aff & (s_near[0][lane] | s_near[1][lane] | s_near[2][lane] | s_near[3][lane]);
    const unsigned mine = __popc(go);
    unsigned incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += y;
    }
    __shared__ unsigned s_first;
    if (i == 0) {
        const unsigned cnt = __shfl_sync(0xffffffffu, incl, 31);
        const unsigned na = __reduce_add_sync(0xffffffffu, (unsigned)__popc(aff));
        if (in) a.tbits[w] = go;
        if (lane == 0) {
            s_first = cnt ? atomicAdd(&a.st->count, cnt) : 0u;
            if (na) atomicAdd(&a.st->affected, na);
        }
        unsigned long long sum = 0ull;
        unsigned tops = 0u;
        for (uint32_t m = go; m; m &= m - 1u) {
            const unsigned s = w * 32u + (unsigned)__ffs((int)m) - 1u;
            sum += __ldg(a.rowsum + s);
            tops += __ldg(a.top + s);
        }
        if (sum) atomicAdd(&a.st->old_sum, sum);
        tops = __reduce_add_sync(0xffffffffu, tops);
        if (lane == 0 && tops) atomicAdd(&a.st->tops, (unsigned long long)tops);
    }
    __syncthreads();
    // the places of the block's 1024 vertices, each warp the words of a quarter
    const unsigned first = s_first;
    for (int k = i * 8; k < i * 8 + 8; ++k) {
        const uint32_t g = __shfl_sync(0xffffffffu, go, k);
        const unsigned at = first + __shfl_sync(0xffffffffu, incl - mine, k) + __popc(g & ((1u << lane) - 1u));
        const unsigned v = (blockIdx.x * 32u + (unsigned)k) * 32u + lane;
        if (v >= (unsigned)a.n) continue;
        const bool hit = (g >> lane) & 1u;
        a.inv[v] = hit ? (int32_t)at : -1;
        if (hit) a.list[at] = (int32_t)v;
    }
}

// The current distances within T: the plane rows of T masked with T's bits, 16 bytes a
// lane, kWithinParts warps a row (1600 rows of 4 x 8 KB at n = 65536: 52 MB from HBM; a
// warp a row with 4-byte loads under a test of the mask took 80 us).
constexpr unsigned kWithinParts = 4;
__global__ void __launch_bounds__(256) inc_within(const IncArgs a) {
    const unsigned lane = threadIdx.x & 31u, quads = (unsigned)(a.cw / 4);   // uint4 of a row
    const unsigned total = a.st->count * kWithinParts, per = (quads + kWithinParts - 1u) / kWithinParts;
    const uint4 *planes = reinterpret_cast<const uint4 *>(a.planes);
    const uint4 *tb = reinterpret_cast<const uint4 *>(a.tbits);
    unsigned long long sum = 0ull;
    for (unsigned q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < total; q += (gridDim.x * blockDim.x) >> 5) {
        const unsigned lo = q % kWithinParts * per, hi = min(quads, lo + per);
        const uint4 *row = planes + (size_t)a.list[q / kWithinParts] * quads;
        unsigned part = 0u;
#pragma unroll 4
        for (unsigned k = lo + lane; k < hi; k += 32u) {
            const uint4 m = __ldg(tb + k);
#pragma unroll
            for (int p = 0; p < kPlanes; ++p) {
                const uint4 x = __ldg(row + (size_t)p * (a.ps / 4) + k);
                part += (unsigned)(__popc(x.x & m.x) + __popc(x.y & m.y) + __popc(x.z & m.z) + __popc(x.w & m.w)) << p;
            }
        }
        sum += __reduce_add_sync(0xffffffffu, part);
    }
    if (lane == 0 && sum) atomicAdd(&a.st->tt_sum, sum);
}

// st->found = 1 when two vertices outside T lie at distance `dist` (a warp per vertex
// whose eccentricity allows it).  Only run when the pairs that T touches may be all there
// are at the current diameter.
__global__ void __launch_bounds__(256) inc_outside_at(const IncArgs a, const unsigned dist) {
    const unsigned lane = threadIdx.x & 31u, words = ((unsigned)a.n + 31u) / 32u;
    for (unsigned v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < (unsigned)a.n;
         v += (gridDim.x * blockDim.x) >> 5) {
        if (a.ecc[v] < dist || a.inv[v] >= 0 || a.st->found) continue;
        bool hit = false;
        for (unsigned k = lane; k < words; k += 32u) {
            uint32_t live = ~a.tbits[k];
            if (k == words - 1u && (a.n & 31)) live &= (1u << (a.n & 31)) - 1u;
            hit |= (dist4_eq(dist4_load(a.planes, a.ps, (size_t)v * a.cw + k), dist4_const(dist)) & live) != 0u;
        }
        if (__any_sync(0xffffffffu, hit) && lane == 0) a.st->found = 1;
    }
}

// The candidate's adjacency `cand` from the one of the move before it: that move's rows
// back to the current graph's, then the four slots of this move replaced (first
// occurrence, as gg_swap specifies).
__global__ void edit_rows_kernel(int32_t *cand, const int32_t *adj, int d, gg_swap last, gg_swap sw) {
    if (last.a >= 0) {
        const int rows[4] = {last.a, last.b, last.c, last.d};
        for (int k = threadIdx.x; k < 4 * d; k += blockDim.x) {
            const size_t at = (size_t)rows[k / d] * d + k % d;
            cand[at] = adj[at];
        }
    }
    __syncthreads();
    const int i = threadIdx.x;
    if (i >= 4) return;
    const int rows[4] = {sw.a, sw.b, sw.c, sw.d};
    const int from[4] = {sw.b, sw.a, sw.d, sw.c};
    const int to0[4] = {sw.c, sw.d, sw.a, sw.b};
    const int to1[4] = {sw.d, sw.c, sw.b, sw.a};
    int32_t *row = cand + (size_t)rows[i] * d;
    for (int k = 0; k < d; ++k)
        if (row[k] == from[i]) { row[k] = sw.mode ? to1[i] : to0[i]; break; }
}

gg_status ifail(gg_status s, const std::string &m) {
    (void)cudaGetLastError();
    gg::set_last_error(m.c_str());
    return s;
}

#define GI_CK(call)                                                                      \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess)                                                           \
            return ifail(e_ == cudaErrorMemoryAllocation ? GG_OUT_OF_MEMORY : GG_CUDA_ERROR, \
                         std::string(#call) + ": " + cudaGetErrorString(e_));           \
    } while (0)

}  // namespace

struct gg_inc {
    int n = 0, d = 0, device = 0;
    gg_engine *eng = nullptr;         // full evaluations and searches from a source list
    cudaStream_t stream = nullptr;
    std::vector<int32_t> h_adj;       // current graph (host copy, validates moves)
    int32_t *d_adj = nullptr, *d_cand = nullptr, *d_inv = nullptr, *d_list = nullptr;
    gg_swap last{0, -1, -1, -1, -1, 0};   // the move d_cand holds (a < 0: none)
    uint32_t *d_tbits = nullptr;
    unsigned *d_stats = nullptr;      // [3][n]: distance sum, eccentricity, vertices at the diameter
    uint64_t at_top = 0;              // pairs at the diameter
    int sms = 0;
    int *d_asym = nullptr, *h_asym = nullptr;
    uint4 *d_planes = nullptr;
    unsigned cols = 0;                // plane columns (chunks of 128 sources)
    IncStatus *d_st = nullptr, *h_st = nullptr;
    bool planes_ok = false;           // symmetric, connected, diameter <= 15
    gg_result cur{};                  // current graph's exact counts
};

namespace {

void inc_free(gg_inc *h) {
    if (!h) return;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    if (h->eng) gg_destroy(h->eng);
    cudaFree(h->d_adj); cudaFree(h->d_cand); cudaFree(h->d_inv); cudaFree(h->d_stats);
    // (d_list and d_tbits lie behind d_inv)
    cudaFree(h->d_planes); cudaFree(h->d_st); cudaFreeHost(h->h_st);
    cudaFree(h->d_asym); cudaFreeHost(h->h_asym);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

// Full evaluation of the current graph, writing the distance planes.
gg_status inc_rebuild(gg_inc *h) {
    gg_eval_opts o{};
    o.max_levels = 199;               // cudaASPLgraph's cap (cudaASPLgraph.cu:190)
    gg::EvalExtra x;
    x.planes = h->d_planes;
    x.nplanes = kPlanes;
    x.no_graph = true;
    uint64_t counts[200] = {};
    o.level_counts = counts;
    h->planes_ok = false;
    h->last.a = -1;
    GI_CK(cudaMemcpyAsync(h->d_cand, h->d_adj, h->h_adj.size() * sizeof(int32_t), cudaMemcpyDeviceToDevice, h->stream));
    gg_status s = gg::engine_eval(h->eng, h->d_adj, &o, &h->cur, h->stream, &x);
    if (s != GG_OK) return s;

    if (!h->cur.connected || h->cur.levels >= (1 << kPlanes)) return GG_OK;
    // the table passed the engine's range check; the row reductions need a
    // symmetric distance matrix
    const cudaStream_t st = h->stream;
    const long long ent = (long long)h->n * h->d;
    GI_CK(cudaMemsetAsync(h->d_asym, 0, sizeof(int), st));
    table_symmetry<<<(int)((ent + 255) / 256), 256, 0, st>>>(h->d_adj, h->n, h->d, h->d_asym);
    GI_CK(cudaGetLastError());
    h->at_top = counts[h->cur.levels];
    plane_row_stats<kPlanes><<<plane_row_stats_grid(h->n, h->sms), 256, 0, st>>>(
        h->d_planes, (unsigned long long)h->n * h->cols, h->cols, h->n, h->d_stats, h->d_stats + h->n,
        h->d_stats + 2 * (size_t)h->n, (unsigned)h->cur.levels);
    GI_CK(cudaGetLastError());
    GI_CK(cudaMemcpyAsync(h->h_asym, h->d_asym, sizeof(int), cudaMemcpyDeviceToHost, st));
    GI_CK(cudaStreamSynchronize(st));
    h->planes_ok = *h->h_asym == 0;
    return GG_OK;
}

gg_status check_swap(const gg_inc *h, const gg_swap *sw) {
    const int v[4] = {sw->a, sw->b, sw->c, sw->d};
    for (int i = 0; i < 4; ++i)
        if (v[i] < 0 || v[i] >= h->n) return ifail(GG_BAD_ARG, "move vertex out of range");
    for (int i = 0; i < 4; ++i)
        for (int j = i + 1; j < 4; ++j)
            if (v[i] == v[j]) return ifail(GG_BAD_ARG, "move needs four distinct vertices");
    if (sw->mode != 0 && sw->mode != 1) return ifail(GG_BAD_ARG, "move mode must be 0 or 1");
    auto has = [&](int x, int y) {
        for (int k = 0; k < h->d; ++k)
            if (h->h_adj[(size_t)x * h->d + k] == y) return true;
        return false;
    };
    if (!has(sw->a, sw->b) || !has(sw->b, sw->a) || !has(sw->c, sw->d) || !has(sw->d, sw->c))
        return ifail(GG_BAD_ARG, "move removes an edge the graph does not have");
    return GG_OK;
}

void apply_host(std::vector<int32_t> &adj, int d, const gg_swap &sw) {
    const int rows[4] = {sw.a, sw.b, sw.c, sw.d};
    const int from[4] = {sw.b, sw.a, sw.d, sw.c};
    const int to0[4] = {sw.c, sw.d, sw.a, sw.b};
    const int to1[4] = {sw.d, sw.c, sw.b, sw.a};
    for (int i = 0; i < 4; ++i)
        for (int k = 0; k < d; ++k)
            if (adj[(size_t)rows[i] * d + k] == from[i]) {
                adj[(size_t)rows[i] * d + k] = sw.mode ? to1[i] : to0[i];
                break;
            }
}

}  // namespace

extern "C" {

gg_status gg_inc_create(int n, int degree, int device, gg_inc **out) {
    if (!out || n < 2 || degree < 1) return ifail(GG_BAD_ARG, "need n >= 2, degree >= 1");
    *out = nullptr;
    gg_inc *h = new gg_inc();
    h->n = n; h->d = degree; h->device = device;
    gg_status s = gg::graph_engine(n, degree, device, &h->eng);
    if (s != GG_OK) { inc_free(h); return s; }
    if (cudaSetDevice(device) != cudaSuccess) { inc_free(h); return ifail(GG_NO_DEVICE, "cudaSetDevice failed"); }
    h->cols = (unsigned)gg::engine_plane_cols(h->eng);
    const size_t adj_b = (size_t)n * degree * sizeof(int32_t);
    const size_t plane_b = (size_t)kPlanes * n * h->cols * sizeof(uint4);
    cudaError_t e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&h->d_adj, adj_b);
    if (e == cudaSuccess) e = cudaMalloc(&h->d_cand, adj_b);
    // inv, list and T's bits in one allocation
    const size_t ids = ((size_t)n * sizeof(int32_t) + 255) / 256 * 256;
    if (e == cudaSuccess) e = cudaMalloc(&h->d_inv, 2 * ids + (size_t)h->cols * sizeof(uint4));
    if (e == cudaSuccess) {
        h->d_list = h->d_inv + ids / sizeof(int32_t);
        h->d_tbits = reinterpret_cast<uint32_t *>(h->d_inv + 2 * (ids / sizeof(int32_t)));
        e = cudaMemsetAsync(h->d_tbits, 0, (size_t)h->cols * sizeof(uint4), h->stream);
    }
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaMalloc(&h->d_stats, 3 * (size_t)n * sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMalloc(&h->d_asym, sizeof(int));
    if (e == cudaSuccess) e = cudaMallocHost(&h->h_asym, sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc(&h->d_planes, plane_b);
    if (e == cudaSuccess) e = cudaMalloc(&h->d_st, sizeof(IncStatus));
    if (e == cudaSuccess) e = cudaMallocHost(&h->h_st, sizeof(IncStatus));
    if (e != cudaSuccess) {
        inc_free(h);
        return ifail(e == cudaErrorMemoryAllocation ? GG_OUT_OF_MEMORY : GG_CUDA_ERROR, cudaGetErrorString(e));
    }
    *out = h;
    return GG_OK;
}

gg_status gg_inc_set_graph(gg_inc *h, const int32_t *adj, gg_result *r) {
    if (!h || !adj) return ifail(GG_BAD_ARG, "null argument");
    GI_CK(cudaSetDevice(h->device));
    h->h_adj.assign(adj, adj + (size_t)h->n * h->d);
    GI_CK(cudaMemcpyAsync(h->d_adj, h->h_adj.data(), h->h_adj.size() * 4, cudaMemcpyHostToDevice, h->stream));
    gg_status s = inc_rebuild(h);
    if (s != GG_OK) return s;
    if (r) *r = h->cur;
    return GG_OK;
}

gg_status gg_inc_eval(gg_inc *h, const gg_swap *sw, gg_cand_result *out, int *affected) {
    if (!h || !sw || !out) return ifail(GG_BAD_ARG, "null argument");
    if (h->h_adj.empty()) return ifail(GG_BAD_ARG, "no graph set");
    gg_status s = check_swap(h, sw);
    if (s != GG_OK) return s;
    GI_CK(cudaSetDevice(h->device));
    const cudaStream_t st = h->stream;
    edit_rows_kernel<<<1, 128, 0, st>>>(h->d_cand, h->d_adj, h->d, h->last, *sw);
    GI_CK(cudaGetLastError());
    h->last = *sw;
    gg_eval_opts o{};
    o.max_levels = 199;
    gg_result r{};
    if (!h->planes_ok) {
        // distances of the current graph unknown: evaluate the moved graph in full
        gg::EvalExtra full;
        full.no_graph = true;
        s = gg::engine_eval(h->eng, h->d_cand, &o, &r, st, &full);
        if (s != GG_OK) return s;
        out->total = r.total; out->reached = r.reached; out->levels = r.levels; out->connected = r.connected;
        if (affected) *affected = h->n;
        return GG_OK;
    }
    GI_CK(cudaMemsetAsync(h->d_st, 0, sizeof(IncStatus), st));
    const size_t n = (size_t)h->n;
    IncArgs a{};
    a.planes = reinterpret_cast<const uint32_t *>(h->d_planes);
    a.ps = n * h->cols * 4;
    a.cw = (size_t)h->cols * 4;
    a.adj = h->d_adj;
    a.n = h->n; a.d = h->d;
    a.sw = *sw;
    a.radius = (unsigned)(std::max<int>(h->cur.levels, 1) - 1) / 2;
    a.rowsum = h->d_stats; a.ecc = h->d_stats + n; a.top = h->d_stats + 2 * n;
    a.inv = h->d_inv; a.tbits = h->d_tbits; a.list = h->d_list;
    a.st = h->d_st;
    inc_select<<<(h->n + 1023) / 1024, 128, 0, st>>>(a);
    inc_within<<<h->sms * 8, 256, 0, st>>>(a);
    GI_CK(cudaGetLastError());
    GI_CK(cudaMemcpyAsync(h->h_st, h->d_st, sizeof(IncStatus), cudaMemcpyDeviceToHost, st));
    GI_CK(cudaStreamSynchronize(st));
    const IncStatus is = *h->h_st;
    if (affected) *affected = (int)is.affected;
    // (the edited graph is symmetric when both ends list a removed edge equally often)
    auto times = [&](int v, int u) { return std::count(&h->h_adj[(size_t)v * h->d], &h->h_adj[(size_t)v * h->d] + h->d, u); };
    if (times(sw->a, sw->b) != times(sw->b, sw->a) || times(sw->c, sw->d) != times(sw->d, sw->c)) {
        gg::EvalExtra full;
        full.no_graph = true;
        s = gg::engine_eval(h->eng, h->d_cand, &o, &r, st, &full);
        if (s != GG_OK) return s;
        out->total = r.total; out->reached = r.reached; out->levels = r.levels; out->connected = r.connected;
        return GG_OK;
    }
    if (is.count == 0) {
        // no distance changes
        out->total = h->cur.total; out->reached = h->cur.reached;
        out->levels = h->cur.levels; out->connected = h->cur.connected;
        return GG_OK;
    }
    gg::EvalExtra x;
    uint64_t within[2] = {0, 0};
    x.inv = h->d_inv;
    x.ns = (int)is.count;
    x.no_graph = true;   // the source count changes from call to call
    x.within = within;
    s = gg::engine_eval(h->eng, h->d_cand, &o, &r, st, &x);
    if (s != GG_OK) return s;
    const uint64_t T = is.count;
    out->total = h->cur.total - (2 * is.old_sum - is.tt_sum) + (2 * r.total - within[0]);
    out->reached = h->cur.reached - (2 * T * n - T * T) + (2 * r.reached - within[1]);
    int top = h->cur.levels;   // the largest distance between vertices outside T
    if (h->at_top <= 2ull * is.tops) {
        for (; top > r.levels; --top) {
            GI_CK(cudaMemsetAsync(&h->d_st->found, 0, sizeof(int), st));
            inc_outside_at<<<h->sms * 8, 256, 0, st>>>(a, (unsigned)top);
            GI_CK(cudaGetLastError());
            GI_CK(cudaMemcpyAsync(h->h_st, h->d_st, sizeof(IncStatus), cudaMemcpyDeviceToHost, st));
            GI_CK(cudaStreamSynchronize(st));
            if (h->h_st->found) break;
        }
    }
    out->levels = std::max(top, r.levels);
    out->connected = out->reached == (uint64_t)h->n * h->n;
    return GG_OK;
}

gg_status gg_inc_commit(gg_inc *h, const gg_swap *sw, gg_result *r) {
    if (!h || !sw) return ifail(GG_BAD_ARG, "null argument");
    if (h->h_adj.empty()) return ifail(GG_BAD_ARG, "no graph set");
    gg_status s = check_swap(h, sw);
    if (s != GG_OK) return s;
    GI_CK(cudaSetDevice(h->device));
    apply_host(h->h_adj, h->d, *sw);
    GI_CK(cudaMemcpyAsync(h->d_adj, h->h_adj.data(), h->h_adj.size() * 4, cudaMemcpyHostToDevice, h->stream));
    s = inc_rebuild(h);
    if (s != GG_OK) return s;
    if (r) *r = h->cur;
    return GG_OK;
}

gg_status gg_inc_destroy(gg_inc *h) {
    inc_free(h);
    return GG_OK;
}

}  // extern "C"
