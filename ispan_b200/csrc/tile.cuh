// tile.cuh -- the SCCs of small components in shared memory.
//
// A CTA takes a few components as one graph of 16-bit local ids, its
// out-lists in shared memory, and runs labelling rounds on it: every vertex
// carries the lowest label (local id) among its ancestors, f, and among its
// descendants, b, inside its class.  f is pushed along the out-list with
// atomicMin, b pulled by its owner, so the out-lists alone are enough; a
// label also jumps to the label of its holder, so a ring takes about
// log(length) passes.  Where f = b = p the vertex is in p's SCC; the others
// go on, classed by (f, b), their lists pruned to their class.  The local ids
// are the ranks of the original ids: where ids follow the edges, the lowest
// label among the descendants (or ancestors) is the SCC's own, and two rounds
// end what random labels split in half per round.
//
// That jump helps one direction: where ids ascend along a ring, the lowest
// descendant's label comes back one edge a pass.  So every vertex also keeps
// a link to a descendant and one to an ancestor (first the neighbour nearest by
// id), joins their labels and jumps to their links: after k passes a link
// spans 2^k edges and the label is the lowest along them.  A label that
// arrives later somewhere under a long link is missed by it, so the links
// start anew every kTileAgain passes.
//
// What bounds it: shared-memory accesses at random addresses (about fifteen a
// vertex and pass) and the passes' barriers: 8,192 vertices on 1,024 threads
// take about 6 us a pass.  Pieces of time-ordered DAGs of rings (2,000 to 7,500
// vertices): 75 to 1,280 passes without the links, up to 4 ms a tile; with
// them 17 to 28 passes, 50-230 us.
#pragma once
#include "common.cuh"

namespace ispan {

constexpr int kTileAgain = 10;  // passes after which the links start anew: 2^10 hops
constexpr int kRankRounds = 3;  // rounds with ranks as labels, here and in k_resolve

// A permutation of the BITS-bit numbers and its inverse: odd factors (of the
// golden ratio, as in multiplicative hashing) around an xor-shift by half the
// width, which undoes itself.  Rounds below kRankRounds: the identity.
template <int BITS>
struct LabelMix {
    static constexpr uint32_t kMask = BITS == 32 ? 0xffffffffu : (1u << (BITS & 31)) - 1u;
    static constexpr int kShift = (BITS + 1) / 2;
    uint32_t a, b, ia, ib;
    bool on;
    __device__ __forceinline__ explicit LabelMix(int round) : on(round >= kRankRounds) {
        a = (0x9e3779b1u * (2u * (uint32_t)round + 1u)) | 1u;
        b = ((0x9e3779b1u * (2u * (uint32_t)round + 2u)) >> 5) | 1u;
        ia = a;
        ib = b;
        for (int k = 0; k < 4; ++k) {  // (Newton: 3 bits are right at first, twice as many each time)
            ia *= 2u - a * ia;
            ib *= 2u - b * ib;
        }
    }
    __device__ __forceinline__ uint32_t label(uint32_t i) const {
        if (!on) return i;
        const uint32_t y = (i * a) & kMask;
        return ((y ^ (y >> kShift)) * b) & kMask;
    }
    __device__ __forceinline__ uint32_t holder(uint32_t l) const {
        if (!on) return l;
        const uint32_t y = (l * ib) & kMask;
        return ((y ^ (y >> kShift)) * ia) & kMask;
    }
};

template <int V_, int E_, int THREADS>
struct Tile {
    static constexpr int kV = V_, kE = E_, kThreads = THREADS, kPer = V_ / THREADS;
    static constexpr int kBits = 31 - __builtin_clz(V_);  // of a local id
    static_assert(V_ == 1 << kBits, "labels are mixed within the tile's ids");
    union {
        int32_t orig[V_];      // original ids; while solving:
        uint16_t link[2][V_];  // an ancestor, a descendant
    };
    int32_t f[V_], b[V_];
    uint16_t off[V_], len[V_];
    uint16_t adj[E_];
    uint32_t dead[V_ / 32];
    int32_t start, count, edges;
};

// Sort the tile's vertices by original id.  Before: f[i] the original id of
// the i-th vertex; after: orig[j] the original ids in order, b[j] the place i
// that each came from, f[i] the rank j of the i-th (padding left out).  A
// bitonic sort over the next power of two.
template <typename T>
__device__ __forceinline__ void tile_sort(T &t, int n) {
    int m = 32;
    while (m < n) m <<= 1;
    for (int i = threadIdx.x; i < m; i += T::kThreads) {
        if (i >= n) t.f[i] = 0x7fffffff;
        t.b[i] = i;
    }
    for (int k = 2; k <= m; k <<= 1)
        for (int j = k >> 1; j; j >>= 1) {
            __syncthreads();
            for (int q = threadIdx.x; q < m / 2; q += T::kThreads) {
                const int a = 2 * q - (q & (j - 1)), c = a + j;  // j apart, a's bit j clear
                const int x = t.f[a], y = t.f[c];
                if ((x > y) == ((a & k) == 0)) {
                    t.f[a] = y;
                    t.f[c] = x;
                    const int z = t.b[a];
                    t.b[a] = t.b[c];
                    t.b[c] = z;
                }
            }
        }
    __syncthreads();
    for (int j = threadIdx.x; j < n; j += T::kThreads) t.orig[j] = t.f[j];
    __syncthreads();
    for (int j = threadIdx.x; j < n; j += T::kThreads) t.f[t.b[j]] = j;
    __syncthreads();
}

// entry k of the tile's lists (checked builds: the position and the id)
template <typename T>
__device__ __forceinline__ int tile_adj(const T &t, int k) {
    if (!ICHK(k >= 0 && k < T::kE, 30, k)) return 0;
    const int w = t.adj[k];
    return ICHK(w < T::kV, 31, w) ? w : 0;
}

// i's links anew: the descendant nearest by id, and i as that one's ancestor
// (of several, any).
template <typename T>
__device__ __forceinline__ void tile_link(T &t, int i) {
    int near = 0xffff, at = i;
    for (int k = t.off[i], z = k + t.len[i]; k < z; ++k) {
        const int w = tile_adj(t, k), far = abs(w - i);
        if (far < near && far) { near = far; at = w; }
    }
    t.link[1][i] = (uint16_t)at;
    t.link[0][at] = (uint16_t)i;
}

// Solve the tile's n vertices (orig and the lists written, dead cleared; the
// caller's threads need not have met since): labels,
// classes, histogram entries; the thread's vertices and SCCs are added to
// done and sccs.  Ends with a barrier.
template <typename T, typename RunT>
__device__ __forceinline__ void tile_solve(T &t, int n, const RunT &r, int64_t &done, int64_t &sccs) {
    if (!ICHK(n >= 0 && n <= T::kV, 32, n)) return;
    constexpr int kPer = T::kPer;
    const int tid = threadIdx.x;
    unsigned mine = 0;  // my vertices not solved yet
#pragma unroll
    for (int u = 0; u < kPer; ++u) mine |= (u * T::kThreads + tid < n ? 1u : 0u) << u;
    int32_t orig[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) orig[u] = (mine >> u) & 1u ? t.orig[u * T::kThreads + tid] : 0;
    __syncthreads();  // the lists' builders are done with f and b, and orig is read
    for (int round = 0;; ++round) {
        if (round > n) {  // every round finds the SCC of each class's lowest label
            if (tid == 0) atomicCAS(r.err, 0, kErrOverflow);
            break;
        }
        const LabelMix<T::kBits> mix(round);
        // labels and links: the descendant nearest by id, and the reverse
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            if (!((mine >> u) & 1u)) continue;
            const int i = u * T::kThreads + tid;
            t.f[i] = t.b[i] = (int32_t)mix.label(i);
            t.link[0][i] = (uint16_t)i;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kPer; ++u)
            if ((mine >> u) & 1u) tile_link(t, u * T::kThreads + tid);
        // (the barrier of the first test: lists, labels and links are in place)
        // after k passes a label has come k edges far, so n passes are enough
        int pass = 0;
        for (int ch = 1; __syncthreads_or(ch); ++pass) {
            if (pass > n + 2) {
                if (tid == 0) atomicCAS(r.err, 0, kErrOverflow);
                break;
            }
            ch = 0;
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                if (!((mine >> u) & 1u)) continue;
                const int i = u * T::kThreads + tid;
                volatile int32_t *f = t.f, *b = t.b;
                const int32_t f0 = f[i], b0 = b[i];
                // the link's link before its label: that then covers all between them
                volatile uint16_t *anc = t.link[0], *des = t.link[1];
                const int la = anc[i], ld = des[i];
                const uint16_t la2 = anc[la], ld2 = des[ld];
                const int32_t fv = min(min(f0, f[mix.holder(f0)]), f[la]);
                int32_t bv = min(min(b0, b[mix.holder(b0)]), b[ld]);
                const int o = t.off[i], z = o + t.len[i];
                for (int k = o; k < z; ++k) {
                    const int w = tile_adj(t, k);
                    if (f[w] > fv) { atomicMin(&t.f[w], fv); ch = 1; }
                    bv = min(bv, b[w]);
                }
                if (fv < f0) { atomicMin(&t.f[i], fv); ch = 1; }
                if (bv < b0) { b[i] = bv; ch = 1; }
                if (pass % kTileAgain != kTileAgain - 1) {
                    anc[i] = la2;
                    des[i] = ld2;
                } else {
                    tile_link(t, i);
                }
            }
        }
        // solved: f = b = p's label.  A solved p gathers its SCC's lowest
        // original id in f[p] and its size in b[p] (its members keep
        // p's label in their own f)
        unsigned sol = 0;
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int i = u * T::kThreads + tid;
            if (((mine >> u) & 1u) && t.f[i] == t.b[i]) sol |= 1u << u;
        }
        unsigned roots = 0;
#pragma unroll
        for (int u = 0; u < kPer; ++u)
            if (((sol >> u) & 1u) && (int)mix.holder(t.f[u * T::kThreads + tid]) == u * T::kThreads + tid)
                roots |= 1u << u;
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int i = u * T::kThreads + tid;
            if ((sol >> u) & 1u) atomicOr(&t.dead[i >> 5], 1u << (i & 31));
            if ((roots >> u) & 1u) {
                t.f[i] = orig[u];
                t.b[i] = 1;
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int i = u * T::kThreads + tid;
            if (((sol & ~roots) >> u) & 1u) {
                const int p = (int)mix.holder(t.f[i]);
                atomicMin(&t.f[p], orig[u]);
                atomicAdd(&t.b[p], 1);
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int i = u * T::kThreads + tid;
            if (!((sol >> u) & 1u)) continue;
            const bool root = (roots >> u) & 1u;
            const int32_t lab = root ? t.f[i] : t.f[mix.holder(t.f[i])], ov = orig[u];
            if (!VOK(ov, 33)) continue;
            r.label[ov] = lab;
            r.cls[ov] = CLS_MICE;
            clear_bit(r.A, ov);
            ++done;
            if (root) {
                atomicAdd((unsigned long long *)(r.hist + t.b[i]), 1ull);  // a tile's vertices < kHistCap
                ++sccs;
            }
        }
        mine &= ~sol;
        // the others keep the entries of their own class (f, b)
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            if (!((mine >> u) & 1u)) continue;
            const int i = u * T::kThreads + tid;
            const int32_t fv = t.f[i], bv = t.b[i];
            const int o = t.off[i], z = o + t.len[i];
            int q = o;
            for (int k = o; k < z; ++k) {
                const int w = tile_adj(t, k);
                if (!((t.dead[w >> 5] >> (w & 31)) & 1u) && t.f[w] == fv && t.b[w] == bv) t.adj[q++] = (uint16_t)w;
            }
            t.len[i] = (uint16_t)(q - o);
        }
        if (!__syncthreads_or(mine != 0u)) break;
    }
}

// The CTA's sums of tile_solve's counts to the run's counters.
template <typename RunT>
__device__ __forceinline__ void tile_report(const RunT &r, int64_t done, int64_t sccs) {
    const int64_t wd = warp_sum64(done), ws = warp_sum64(sccs);
    if (lane_id() == 0 && wd) {
        atomicAdd(r.counters + C_MICE_V, (unsigned long long)wd);
        atomicAdd(r.counters + C_MICE_SCC, (unsigned long long)ws);
    }
}

}  // namespace ispan
