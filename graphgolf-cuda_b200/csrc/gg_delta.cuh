// gg_delta.cuh -- exact change of a source's distance row under a few edge edits.
//
// The base graph's distances are known (a byte row per source); a candidate graph
// differs from it in a few pull entries ("changes"): row r lists t in place of f.
// A move of a lift changes about 57 of the N distances of a source that it reaches at all
// (m = 1024, g = 32, d = 12), so the change is followed from the edits outwards instead
// of searching again.  For one source, with D the base distances:
//
//   1. raised set A, by waves: a vertex v joins when no neighbour u in the new graph with
//      D[u] < D[v] is outside A.  The first ones are the rows r whose removed neighbour f
//      was a parent (D[f] = D[r] - 1); then the neighbours above what joined (a vertex
//      whose last such neighbour joins is looked at again, so the order does not
//      matter).  By induction over the levels a vertex outside A is at most D away.
//   2. new distances: A starts unreached, every other vertex at D, and each vertex of A
//      takes 1 + the least of its neighbours.  A vertex that gets a value tells the
//      neighbours it can lower (a vertex outside the list then joins it), and those are
//      looked at again, until none is left.  All values are lengths of walks of the new
//      graph and no edge is violated at the end, so they are its distances.
//
// Everything that changed is in the list, each entry with its old distance, and the
// caller gets the change of the number of pairs at every distance.
//
// The candidate graph must be symmetric (a pull row is also the list of the vertices
// that pull from it).  Distances up to kDeltaMax are represented; past it the source
// reports an overflow and the caller searches the candidate in full.
//
// Which sources: a pair {s, v} whose distance changes has a shortest path, old or
// new, of length at most the old diameter through a changed edge, so one of the two
// lies within floor((diameter - 1) / 2) of an endpoint (in the base graph).  With P
// the vertices that do -- in a lift, the orbits of such vertices, followed from their
// representative -- and the distance matrix symmetric, the rows of P suffice: a changed
// pair (s, v) counts once when v is in P too (v's own row brings the other order) and
// twice when not.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace gg {

constexpr int kDeltaLevels = 32;                 // distance counters a candidate keeps
constexpr unsigned kDeltaInf = kDeltaLevels - 1;    // "unreached" in a row and in the counters
constexpr unsigned kDeltaMax = kDeltaInf - 1;       // largest distance represented
constexpr unsigned kDeltaTouched = 0x80u;        // row byte: the vertex is in the list
constexpr int kDeltaRows = 32;                   // most rows a block follows together
constexpr int kDeltaList = 768;                  // list entries kept in shared memory; the rest spill
constexpr int kDeltaQueue = 256;                 // queue entries kept in shared memory; the rest spill
constexpr int kDeltaSpill = 2048;                // spilled entries of each

// A list or queue entry: vertex (22 bits), row slot (5 bits), old distance (5 bits).
constexpr unsigned kDeltaMaxVertex = 1u << 22;
__device__ __forceinline__ uint32_t delta_entry(const unsigned v, const unsigned slot, const unsigned old) {
    return v | (slot << 22) | (old << 27);
}
__device__ __forceinline__ unsigned delta_vertex(const uint32_t x) { return x & (kDeltaMaxVertex - 1u); }
__device__ __forceinline__ unsigned delta_slot(const uint32_t x) { return (x >> 22) & 31u; }
__device__ __forceinline__ unsigned delta_old(const uint32_t x) { return x >> 27; }

__device__ __forceinline__ void delta_cp16(const unsigned smem_dst, const void *gmem_src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void delta_cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Row bytes by shared-memory address.  A row's bytes are changed by word atomics only
// (several threads change different bytes of a word), but for whole passes between
// barriers.
__device__ __forceinline__ unsigned delta_ld(const unsigned at) {
    unsigned v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(at));
    return v;
}
__device__ __forceinline__ void delta_st(const unsigned at, const unsigned v) {
    asm volatile("st.shared.u8 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}
// Sets `bits` of the byte at `at`; its old value.
__device__ __forceinline__ unsigned delta_or(const unsigned at, const unsigned bits) {
    unsigned old;
    const unsigned sh = (at & 3u) * 8u;
    asm volatile("atom.shared.or.b32 %0, [%1], %2;" : "=r"(old) : "r"(at & ~3u), "r"(bits << sh) : "memory");
    return (old >> sh) & 255u;
}
__device__ __forceinline__ void delta_xor(const unsigned at, const unsigned bits) {
    asm volatile("red.shared.xor.b32 [%0], %1;" ::"r"(at & ~3u), "r"(bits << ((at & 3u) * 8u)) : "memory");
}

// What the threads of a block share while they follow its rows.
struct DeltaShared {
    unsigned n;            // list entries
    unsigned qn[3];        // queue entries: of this sweep, of the next, zeroed for the one after
    int overflow;
    uint32_t list[kDeltaList];
    uint32_t queue[2][kDeltaQueue];
};

struct DeltaBlock {
    DeltaShared *s;
    uint32_t *spill;       // [3][kDeltaSpill]: past the shared list and queues, a buffer of the block
    unsigned rows;         // shared-memory address of the rows' bytes, [slots][pitch], 4-byte aligned
    unsigned pitch;
    __device__ __forceinline__ uint32_t get(const unsigned e) const {
        return e < (unsigned)kDeltaList ? s->list[e] : __ldcg(spill + (e - kDeltaList));
    }
    __device__ __forceinline__ uint32_t getq(const unsigned q, const unsigned e) const {
        return e < (unsigned)kDeltaQueue ? s->queue[q][e] : __ldcg(spill + (q + 1u) * kDeltaSpill + (e - kDeltaQueue));
    }
    __device__ __forceinline__ void put(const uint32_t x) const {
        const unsigned e = atomicAdd(&s->n, 1u);
        if (e < (unsigned)kDeltaList) s->list[e] = x;
        else if (e < (unsigned)(kDeltaList + kDeltaSpill)) __stcg(spill + (e - kDeltaList), x);
        else s->overflow = 1;
    }
    // into queue q, counted by qn[c]
    __device__ __forceinline__ void putq(const unsigned q, const unsigned c, const uint32_t x) const {
        const unsigned e = atomicAdd(&s->qn[c], 1u);
        if (e < (unsigned)kDeltaQueue) s->queue[q][e] = x;
        else if (e < (unsigned)(kDeltaQueue + kDeltaSpill)) __stcg(spill + (q + 1u) * kDeltaSpill + (e - kDeltaQueue), x);
        else s->overflow = 1;
    }
    __device__ __forceinline__ unsigned row(const unsigned slot) const { return rows + slot * pitch; }
};

// Follows the changes of `nrows` sources together, by all threads of the block: their
// base distances are in b's rows (overwritten).  Working on many sources at once keeps
// the lanes full: a source's list holds a handful of entries, the block's hundreds.
// change(j): change j < nch, as {r, f, t}: row r lists t in place of f.  G: the candidate
// graph --
//   G.slots()             pull slots a row (a padded slot holds the vertex itself)
//   G.at(v, i)            slot i of row v
//   G.each(v, f)          f(u) for every slot u of row v
// A row's byte: bits 0-4 the distance, bit 7 set when the vertex is in the list, bit 5 or
// 6 (alternating) set when it waits in the next sweep's queue.  On return the list holds
// every (row, vertex) whose distance changed (and some that did not), the bytes & 31
// the new distances.  b.s->overflow is set when a distance past kDeltaMax may be needed
// or the lists ran out of room.
template <class Graph, class Change>
__device__ __forceinline__ void delta_rows(const Graph &G, const DeltaBlock &b, const unsigned nrows,
                                           const unsigned nch, Change change) {
    const unsigned S = G.slots(), tid = threadIdx.x, nthr = blockDim.x;
    DeltaShared &s = *b.s;
    if (tid < 3u) s.qn[tid] = 0u;
    if (tid == 0u) {
        s.n = 0u;
        s.overflow = 0;
    }
    __syncthreads();
    // whether row v (at distance x) has no lower neighbour outside the list (listed ones
    // read as kDeltaTouched or more)
    auto alone = [&](const unsigned row, const unsigned v, const unsigned x) {
        unsigned m = 255u;
        G.each(v, [&](const unsigned u) { m = min(m, delta_ld(row + u)); });
        return m >= x;
    };
    // 1. raised vertices: rows that lost their last lower neighbour ...
    for (unsigned k = tid; k < nrows * nch; k += nthr) {
        const unsigned slot = k / nch, row = b.row(slot);
        const uint3 ch = change(k - slot * nch);
        const unsigned r = ch.x, f = ch.y, x = delta_ld(row + r);
        if ((delta_ld(row + f) & 31u) + 1u == x && alone(row, r, x) && !(delta_or(row + r, kDeltaTouched) & kDeltaTouched))
            b.put(delta_entry(r, slot, x));
    }
    __syncthreads();
    // ... and, wave by wave, the higher neighbours whose lower ones all joined
    unsigned hi = min(s.n, (unsigned)(kDeltaList + kDeltaSpill));
    for (unsigned lo = 0u; lo < hi;) {
        __syncthreads();   // everyone has read s.n
        for (unsigned it = lo * S + tid; it < hi * S; it += nthr) {
            const uint32_t e = b.get(it / S);
            const unsigned w = G.at(delta_vertex(e), it % S), row = b.row(delta_slot(e));
            const unsigned x = delta_ld(row + w);
            if (x < kDeltaTouched && x > delta_old(e) && alone(row, w, x) &&
                !(delta_or(row + w, kDeltaTouched) & kDeltaTouched))
                b.put(delta_entry(w, delta_slot(e), x));
        }
        __syncthreads();
        lo = hi;
        hi = min(s.n, (unsigned)(kDeltaList + kDeltaSpill));
    }
    for (unsigned k = tid; k < hi; k += nthr) {
        const uint32_t e = b.get(k);
        delta_st(b.row(delta_slot(e)) + delta_vertex(e), kDeltaTouched | kDeltaInf);
    }
    __syncthreads();
    // 2. new distances; first the added edges that lower a vertex outside the list
    for (unsigned k = tid; k < nrows * nch; k += nthr) {
        const unsigned slot = k / nch, row = b.row(slot);
        const uint3 ch = change(k - slot * nch);
        const unsigned r = ch.x, t = ch.z, x = delta_ld(row + r);
        if (x < kDeltaTouched && (delta_ld(row + t) & 31u) + 1u < x &&
            !(delta_or(row + r, kDeltaTouched) & kDeltaTouched))
            b.put(delta_entry(r, slot, x));
    }
    __syncthreads();
    // The first sweep takes the list, the later ones their queue.
    const unsigned n0 = min(s.n, (unsigned)(kDeltaList + kDeltaSpill));
    unsigned c = 0u;   // counters: this sweep's queue c, the next sweep's c + 1, zeroed c + 2 (mod 3)
    for (unsigned k = 0u;; ++k) {
        const unsigned cn = c == 2u ? 0u : c + 1u, cz = cn == 2u ? 0u : cn + 1u;
        const unsigned n = k == 0u ? n0 : min(s.qn[c], (unsigned)(kDeltaQueue + kDeltaSpill));
        if (n == 0u) break;
        if (k == 0u) __syncthreads();   // everyone has read s.n
        const unsigned q = k & 1u, mine = k == 0u ? 0u : (q ? 0x40u : 0x20u), next = q ? 0x20u : 0x40u;
        if (tid == 0u) s.qn[cz] = 0u;
        for (unsigned i = tid; i < n; i += nthr) {
            const uint32_t e = k == 0u ? b.get(i) : b.getq(q, i);
            const unsigned slot = delta_slot(e), v = delta_vertex(e), row = b.row(slot);
            unsigned m = 255u;
            G.each(v, [&](const unsigned u) { m = min(m, delta_ld(row + u) & 31u); });
            const unsigned d = delta_ld(row + v) & 31u;
            ++m;
            if (m < d) {
                delta_xor(row + v, (d ^ m) | mine);
                G.each(v, [&](const unsigned w) {
                    if ((delta_ld(row + w) & 31u) > m + 1u) {
                        const unsigned x = delta_or(row + w, kDeltaTouched | next);
                        if (!(x & kDeltaTouched)) b.put(delta_entry(w, slot, x & 31u));
                        if (!(x & next)) b.putq(q ^ 1u, cn, delta_entry(w, slot, 0u));
                    }
                });
            } else {
                if (mine) delta_xor(row + v, mine);
                if (d == kDeltaInf && m == kDeltaInf) s.overflow = 1;   // the neighbour at kDeltaMax is real
            }
        }
        __syncthreads();
        c = cn;
    }
}

// Adds the listed changes to counters of the calling warp: lane L holds the change of the
// number of ordered pairs at distance L (kDeltaInf: unreached).  weight(v): 1 when v's
// own row is followed too, else 2.
template <class Weight>
__device__ __forceinline__ void delta_count(const DeltaBlock &b, Weight weight, int &h) {
    const unsigned n = min(b.s->n, (unsigned)(kDeltaList + kDeltaSpill)), lane = threadIdx.x & 31u;
    for (unsigned e0 = threadIdx.x - lane; e0 < n; e0 += blockDim.x) {
        unsigned key = ~0u;
        if (e0 + lane < n) {
            const uint32_t e = b.get(e0 + lane);
            const unsigned v = delta_vertex(e), old = delta_old(e);
            const unsigned c = delta_ld(b.row(delta_slot(e)) + v) & 31u;
            if (c != old) key = c | (old << 8) | (weight(v) << 16);
        }
        for (unsigned mk = __ballot_sync(0xffffffffu, key != ~0u); mk;) {
            const unsigned k = __shfl_sync(0xffffffffu, key, __ffs((int)mk) - 1);
            const unsigned same = __ballot_sync(0xffffffffu, key == k);
            const int c = __popc(same) * (int)(k >> 16);
            if (lane == (k & 255u)) h += c;
            if (lane == ((k >> 8) & 255u)) h -= c;
            mk &= ~same;
        }
    }
}

}  // namespace gg
