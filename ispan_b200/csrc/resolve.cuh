// resolve.cuh -- the SCCs of the large WCCs on their compact graph
// (compact.cuh), in place of the colouring rounds of k_color, which still
// take what has no compact graph.
//
// Classes.  SCCs never span classes; whenever classes were refined, the lists
// are pruned to edges inside a class, so no search needs a class check.
//   Splitting (k_split): each vertex collects a mask of the pivots that reach
//     it (forward, even rounds) or that it reaches (backward, odd rounds).
//     An SCC's members have equal masks.  K pivots in a line of SCCs make
//     K + 1 classes, where a colour (the lowest pivot that reaches) makes
//     about ln K: on a DAG of planted SCCs a few splitting rounds do what
//     ~20 colouring rounds did.  Pivots come 16 or 64 times denser from round
//     to round; two pivots on one bit or two classes on one hash only make a
//     class coarser.  Alternating directions: downstream of a large SCC every
//     mask is full, upstream every backward one.
//   Tiles (k_tiles): the weakly connected components of what the lists still
//     join are mostly single SCCs; those of up to kTileV vertices are solved
//     in shared memory.  Larger ones are split again, kResIts times in all.
//   Labelling (in a tile, and k_resolve for what is left): every vertex
//     carries the lowest label among its ancestors, f, and among its
//     descendants, b, inside its class (labels are the ids, from the fourth
//     round on mixed ones, see tile.cuh).  Where f = b =
//     the label of p, p reaches the vertex and is reached from it: the vertex
//     is in p's SCC, found without a separate backward search.  At least the
//     SCC of each class's lowest label is.  The others go on, classed by
//     (f, b).
// Values spread by pulling: in a dense pass each vertex joins its
// neighbours' values to its own, in place (gathers, one writer per vertex,
// no atomics), until few vertices change; those are listed and push on,
// level by level.
//
// What bounds it: random sectors of L2 while the gathered array stays there
// (2.1 M vertices: k_split reads 20 GB of sectors at 3.7 TB/s, levels included,
// for 1 GB of DRAM traffic; a dense pass over 48 M entries 0.28 ms); beyond
// about half of the L2 the gathers' DRAM traffic (with 64-bit masks on 21 M
// vertices, 168 MB, a pass took 1.3 ms, with 32-bit ones 0.53).  In the tails a
// level's latency counts.  Web-shaped graphs, colouring stage before and now, one
// B200: 7 M vertices (1.1 M here) 10.0 and 5.3 ms, 140 M vertices (21 M
// here) 244 and 85 ms.
#pragma once
#include "compact.cuh"
#include "tile.cuh"

namespace ispan {

constexpr int kResSplitShift = 8;      // at most one pivot in 256 vertices
constexpr int kResIts = 3;             // times k_split and k_tiles run
constexpr int64_t kResFew = 16;        // fewer vertices left than 1 / 16: no more splitting (a time takes ~1.5 ms even
                                       // for few; the labelling rounds of 18,000 vertices 0.5 ms)
// Width of the masks: 64 bits (three rounds) while their array stays in L2,
// 48 MB; beyond, 16 bits (four rounds): a gather is then a DRAM access more
// often than not, and a dense pass takes the time of its traffic.  (21 M
// vertices: 34 ms a first round with 64 bits, 19 with 32, 9-11 with 16.  42 M
// and 84 M, a call on a web graph: 347-382 and 826-914 ms with 64 bits, 297-350
// and 697-845 with 16.)
constexpr int64_t kResWideN = 6 << 20;
constexpr int64_t kResSparse = 16;     // a pass that changed at most 1 / 16 of the vertices ends the dense passes
                                       // (a listed vertex costs ~0.17 ns to push, a dense pass ~0.01-0.017 ns a vertex);
                                       // more listed ones than that begin them again
constexpr uint32_t kResHash = 0x07ffffffu;  // class word while splitting: 27 bits of hash, 5 bits of log2 |WCC|
constexpr uint32_t kResDead = 0xffffffffu;  // class word of a vertex whose SCC is known


struct ResBufs {
    // the lists of vertex v, [beg[v], end[v]) of adj: [0] in-, [1] out-lists,
    // pruned in place
    int32_t *beg[2], *end[2], *adj[2];
    const int32_t *old;     // original ids
    const int32_t *parent, *wsize;  // WCC root of an original id and, at roots, the WCC's size; read at the start only
    uint32_t *val[2];       // [2 n] forward and backward values (val[1] overlays parent)
    uint32_t *cls;          // [n] class words
    int32_t *mn, *size;     // [n] at a found SCC's p: its lowest original id and its size (mn overlays wsize)
    int32_t *list[2];       // [n] vertices left
    uint32_t *q[2];         // [cap_q] changed vertices, the direction in the top bit
    int64_t cap_q;
    int64_t cap_e;          // entries of each of adj
    int32_t *order;         // [n] vertices grouped by component (overlays q[1])
    int32_t *pos;           // [n] place of a vertex in order (overlays val[0])
};

// lowbias32, the 32-bit integer hash of C. Wellons' hash prospector
__device__ __forceinline__ uint32_t mix32(uint32_t h) {
    h ^= h >> 16;
    h *= 0x7feb352du;
    h ^= h >> 15;
    h *= 0x846ca68bu;
    h ^= h >> 16;
    return h;
}

// Entry k of one direction's lists, and of a list of vertices (checked
// builds: the position and the id)
template <bool CG = false>  // (CG: in L2, where entries move within a kernel or L1 gains nothing)
__device__ __forceinline__ int32_t res_adj(const ResBufs &m, const int32_t *adj, int32_t k) {
    if (!ICHK(k >= 0 && k < m.cap_e, 20, k)) return 0;
    const int32_t w = CG ? __ldcg(adj + k) : adj[k];
    return VOK(w, 21) ? w : 0;
}
__device__ __forceinline__ int32_t res_at(const int32_t *list, int64_t i) {
    if (!list) return (int32_t)i;
    if (!VOK(i, 22)) return 0;
    const int32_t v = list[i];
    return VOK(v, 23) ? v : 0;
}

// The vertex that a label belongs to
__device__ __forceinline__ uint32_t res_holder(const LabelMix<32> &mix, uint32_t l) {
    const uint32_t v = mix.holder(l);
    return VOK((long long)v, 29) ? v : 0u;
}

// The value of a vertex: a mask of pivots while splitting (OR, 16 or 64 bits
// wide), a 32-bit label while labelling (minimum).  The arrays hold 2 n words.
enum ResKind { R_MIN = 32, R_OR16 = 16, R_OR64 = 64 };
template <int K> struct ResVal;
template <> struct ResVal<R_MIN> { using T = uint32_t; };
template <> struct ResVal<R_OR16> { using T = unsigned short; };
template <> struct ResVal<R_OR64> { using T = unsigned long long; };
template <int K>
__device__ __forceinline__ typename ResVal<K>::T res_join(typename ResVal<K>::T a, typename ResVal<K>::T b) {
    return K == R_MIN ? min(a, b) : (typename ResVal<K>::T)(a | b);
}
// join x into *p, the old value back
template <int K>
__device__ __forceinline__ typename ResVal<K>::T res_atomic(typename ResVal<K>::T *p, typename ResVal<K>::T x) {
    if constexpr (K == R_MIN) return atomicMin(p, x);
    if constexpr (K == R_OR64) return atomicOr(p, x);
    if constexpr (K == R_OR16) {  // in the aligned word around it
        const uintptr_t a = reinterpret_cast<uintptr_t>(p);
        const int sh = (int)(a & 2) * 8;
        return (unsigned short)(atomicOr(reinterpret_cast<unsigned *>(a & ~(uintptr_t)3), (unsigned)x << sh) >> sh);
    }
}
template <int K>
__device__ __forceinline__ typename ResVal<K>::T res_warp_join(typename ResVal<K>::T x) {
#pragma unroll
    for (int o = 16; o; o >>= 1) x = res_join<K>(x, (typename ResVal<K>::T)__shfl_xor_sync(kFull, x, o));
    return x;
}

// The entry of v's list whose original id is nearest to its own (v if none).
__device__ __forceinline__ int32_t res_near(const ResBufs &m, int d, int32_t v) {
    const int32_t mine = m.old[v];
    int32_t at = v, near = 0x7fffffff;
    for (int32_t k = m.beg[d][v], e = m.end[d][v]; k < e; ++k) {
        const int32_t w = res_adj(m, m.adj[d], k), far = abs(m.old[w] - mine);
        if (far < near) { near = far; at = w; }
    }
    return at;
}

// One dense step of direction d for four vertices of a lane (v < 0: none):
// their list ranges, then their entries four by four, then the entries'
// values, each group of loads in flight together; a list's entries beyond
// kResLane are read by the whole warp.  Returns a bit per vertex whose value
// changed.
constexpr int kResU = 4;
constexpr int kResLane = 64;
template <int K>
__device__ __forceinline__ unsigned res_pull(const ResBufs &m, int d, const int32_t (&v)[kResU],
                                             const LabelMix<32> &mix) {
    using T = typename ResVal<K>::T;
    T *val = reinterpret_cast<T *>(m.val[d]);
    const int32_t *adj = m.adj[d];
    int32_t b[kResU], e[kResU];
    T own[kResU], nw[kResU];
#pragma unroll
    for (int u = 0; u < kResU; ++u) {
        b[u] = v[u] >= 0 ? m.beg[d][v[u]] : 0;
        e[u] = v[u] >= 0 ? m.end[d][v[u]] : 0;
        own[u] = v[u] >= 0 ? __ldcg(val + v[u]) : (T)0;
    }
    // a label jumps: the holder of my lowest label has ancestors of mine
#pragma unroll
    for (int u = 0; u < kResU; ++u) {
        nw[u] = own[u];
        if constexpr (K == R_MIN)
            if (v[u] >= 0) nw[u] = min(own[u], __ldcg(val + res_holder(mix, own[u])));
    }
    bool more = true;
    for (int step = 0; step < kResLane && more; step += 4) {
        more = false;
        int32_t w[kResU][4];
#pragma unroll
        for (int u = 0; u < kResU; ++u)
#pragma unroll
            for (int q = 0; q < 4; ++q) w[u][q] = b[u] + q < e[u] ? res_adj(m, adj, b[u] + q) : -1;
#pragma unroll
        for (int u = 0; u < kResU; ++u) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (w[u][q] >= 0) nw[u] = res_join<K>(nw[u], __ldcg(val + w[u][q]));
            b[u] = min(b[u] + 4, e[u]);
            more |= b[u] < e[u];
        }
    }
    if (__any_sync(kFull, more)) {
#pragma unroll
        for (int u = 0; u < kResU; ++u) {
            unsigned g = __ballot_sync(kFull, b[u] < e[u]);
            for (; g; g &= g - 1) {
                const int l = __ffs(g) - 1;
                const int32_t lb = __shfl_sync(kFull, b[u], l), le = __shfl_sync(kFull, e[u], l);
                T acc = (T)__shfl_sync(kFull, nw[u], l);
                for (int32_t k = lb + lane_id(); k < le; k += 32) acc = res_join<K>(acc, __ldcg(val + res_adj(m, adj, k)));
                acc = res_warp_join<K>(acc);
                if (lane_id() == l) nw[u] = acc;
            }
        }
    }
    unsigned ch = 0;
#pragma unroll
    for (int u = 0; u < kResU; ++u)
        if (nw[u] != own[u]) {
            __stcg(val + v[u], nw[u]);
            ch |= 1u << u;
        }
    return ch;
}

// The same for one vertex of a lane (v < 0: none), over its link too: the link
// then jumps to its target's, which is read before the target's value (that
// covers all between).  again: the link starts anew.
template <int K>
__device__ __forceinline__ bool res_pull_linked(const ResBufs &m, int d, int32_t v, uint32_t *link, bool again,
                                                const LabelMix<32> &mix) {
    using T = typename ResVal<K>::T;
    T *val = reinterpret_cast<T *>(m.val[d]);
    const int32_t *adj = m.adj[d];
    int32_t b = 0, e = 0;
    T own = 0, nw = 0;
    if (v >= 0) {
        b = m.beg[d][v];
        e = m.end[d][v];
        const uint32_t far = __ldcg(link + v), to = __ldcg(link + far);
        own = __ldcg(val + v);
        nw = res_join<K>(own, __ldcg(val + far));
        if constexpr (K == R_MIN) nw = min(nw, __ldcg(val + res_holder(mix, own)));
        __stcg(link + v, again ? (uint32_t)res_near(m, d, v) : to);
    }
    const int32_t c = min(e, b + kResLane);
    for (; b < c; b += 4) {
        int32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = b + q < c ? res_adj(m, adj, b + q) : v;
#pragma unroll
        for (int q = 0; q < 4; ++q) nw = res_join<K>(nw, __ldcg(val + w[q]));
    }
    b = min(b, e);
    for (unsigned g = __ballot_sync(kFull, b < e); g; g &= g - 1) {
        const int l = __ffs(g) - 1;
        const int32_t lb = __shfl_sync(kFull, b, l), le = __shfl_sync(kFull, e, l);
        T acc = (T)__shfl_sync(kFull, nw, l);
        for (int32_t k = lb + lane_id(); k < le; k += 32) acc = res_join<K>(acc, __ldcg(val + res_adj(m, adj, k)));
        acc = res_warp_join<K>(acc);
        if (lane_id() == l) nw = acc;
    }
    if (nw == own) return false;
    __stcg(val + v, nw);
    return true;
}

// The listed vertices of a warp (ent valid where have) push: a forward value
// along the out-list, a backward one along the in-list.  put(lanes' counts,
// then their entries) appends the vertices whose value that changed.
template <int K, typename Put>
__device__ __forceinline__ void res_push(const ResBufs &m, bool have, uint32_t ent, Put put) {
    using T = typename ResVal<K>::T;
    const int32_t v = (int32_t)(ent & 0x7fffffffu);
    const int d = (int)(ent >> 31);
    const int32_t *adj = m.adj[d ^ 1];
    T *val = reinterpret_cast<T *>(m.val[d]);
    int32_t b = have ? m.beg[d ^ 1][v] : 0;
    int32_t e = have ? m.end[d ^ 1][v] : 0;
    const T mv = have ? __ldcg(val + v) : (T)0;
    // a long list is spread over the warp first: every lane takes a part of it
    unsigned lng = __ballot_sync(kFull, e - b > kResLane);
    for (; lng; lng &= lng - 1) {
        const int l = __ffs(lng) - 1;
        const int32_t lb = __shfl_sync(kFull, b, l), le = __shfl_sync(kFull, e, l);
        const T lv = (T)__shfl_sync(kFull, mv, l);
        const uint32_t le_ent = __shfl_sync(kFull, ent, l);
        const int ld = (int)(le_ent >> 31);
        T *lval = reinterpret_cast<T *>(m.val[ld]);
        for (int32_t k = lb; k < le; k += 32) {
            const int32_t w = k + lane_id() < le ? res_adj<true>(m, m.adj[ld ^ 1], k + lane_id()) : -1;
            bool grew = false;
            if (w >= 0) {
                T x = __ldcg(lval + w);
                if (res_join<K>(x, lv) != x) {
                    x = res_atomic<K>(lval + w, lv);
                    grew = res_join<K>(x, lv) != x;
                }
            }
            const uint32_t en[4] = {(uint32_t)w | ((uint32_t)ld << 31), 0u, 0u, 0u};
            put(grew ? 1u : 0u, en);
        }
        if (lane_id() == l) e = b;
    }
    // four entries of the list at a time, their values, then the atomics of
    // those that grow, each in flight together
    while (__any_sync(kFull, b < e)) {
        int32_t w[4];
        T xv[4];
        unsigned grew = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = b + q < e ? res_adj<true>(m, adj, b + q) : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) xv[q] = w[q] >= 0 ? __ldcg(val + w[q]) : mv;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool go = w[q] >= 0 && res_join<K>(xv[q], mv) != xv[q];
            if (go) xv[q] = res_atomic<K>(val + w[q], mv);
            grew |= (go && res_join<K>(xv[q], mv) != xv[q] ? 1u : 0u) << q;
        }
        b = min(b + 4, e);
        const uint32_t en[4] = {(uint32_t)w[0] | ((uint32_t)d << 31), (uint32_t)w[1] | ((uint32_t)d << 31),
                                (uint32_t)w[2] | ((uint32_t)d << 31), (uint32_t)w[3] | ((uint32_t)d << 31)};
        put(grew, en);
    }
}

// Spread the values of the listed vertices (list null: all of [0, n)) to
// the fixpoint in the directions of `dirs` (bit 0 forward, bit 1 backward).
// s: the rotating counter slot; seeded: the vertices that hold a value are
// listed already (q[0], their number in the slot).  Returns 1; 0 if a grid barrier failed; 2 if
// it gave up, which only masks do, after about kResBudget levels or kResPasses
// dense passes: on long paths without shortcuts they come one edge far per
// level, where labels jump (after kResHops levels the labels take dense passes
// again).
//   dense passes while many vertices change;
//   levels of listed vertices over the whole grid, then,
//   while a level has at most kResTail of them, levels in CTA 0 alone,
//   separated by its own barriers (~3 us a level instead of ~9), the other
//   CTAs waiting at the grid barrier.
constexpr int kResTail = 1024;
constexpr int kResTailLevels = 256;  // levels in CTA 0 before the grid meets again
constexpr int kResBudget = 1024;
constexpr int kResPasses = 160;  // (web graphs: up to 40, rings of 300 with shuffled ids 140; grids both ways, one
                                 // SCC: 450, in each of up to 7 rounds.  400 x 400: 18-30 ms a call, so 4-5;
                                 // 1,000 x 1,000 with shuffled ids 27-29, so 18)
constexpr int kResHops = 64;
// Few vertices take dense passes to the end, over links too (see Tile): a pass
// costs what a level does, ~9 us, and the links end rings of a thousand hops
// in tens of passes.  (What 97 separate graphs left after the tiles, 44,000
// vertices: 4.5 ms of levels, 0.66 with links.)  Many vertices have no links:
// two more gathers in a pass of about three, measured 7.6 ms -> 10.7 on a web
// graph of 1.1 M vertices here.
constexpr int64_t kResLinkN = 1 << 18;
constexpr int kResAgain = 10;          // passes after which the links start anew: 2^10 hops
struct ResSmem {
    int64_t sum[kWarps];
    uint32_t q[2][2 * kResTail];
    int cnt[2];
};
template <int K>
__device__ __forceinline__ int res_spread(const Run<int32_t> &r, const ResBufs &m, unsigned long long *chg,
                                           unsigned long long *qc, const unsigned long long *x_large, const int32_t *list, int64_t n, int dirs, int &s,
                                           ResSmem &sm, bool seeded, const LabelMix<32> &mix) {
    const int64_t gt = (int64_t)blockIdx.x * kBlock + threadIdx.x;
    const int64_t nt = (int64_t)gridDim.x * kBlock;
    bool dense = true;
    int64_t prev = n * 2, nq = 0;
    int cur = 0, levels = 0, hops = 0, passes = 0;
    // few vertices: links, and dense passes to the end
    const bool linked = n <= kResLinkN;
    uint32_t *link[2] = {nullptr, nullptr};
    if (linked) {
        const int64_t all = (int64_t)__ldcg(x_large);
        for (int d = 0; d < 2; ++d) {
            if (!((dirs >> d) & 1)) continue;
            link[d] = K == R_MIN ? m.val[d] + all : m.val[d ^ 1];  // (masks spread one way at a time)
            for (int64_t i = gt; i < n; i += nt) {
                const int32_t v = res_at(list, i);
                link[d][v] = (uint32_t)res_near(m, d, v);
            }
        }
        if (!grid_sync(r.gsync, r.err)) return 0;
    }
    if (seeded) {
        nq = (int64_t)__ldcg(qc + s);
        s = s == 2 ? 0 : s + 1;
        dense = linked || nq > n / kResSparse || nq > m.cap_q;
    }
    for (int64_t guard = 0; guard <= 128 * (r.V + 2); ++guard) {  // every pass lowers a value or sets a bit
        const int s1 = s == 2 ? 0 : s + 1;
        if (blockIdx.x == 0 && threadIdx.x == 0) { chg[s1] = 0ull; qc[s1] = 0ull; }
        if (K != R_MIN && (levels > kResBudget || passes > kResPasses)) return 2;
        if (dense) {
            // few changes in the last pass: the vertices that change now are listed
            const bool listing = prev <= n / kResSparse && !linked;
            int changed = 0;
            if (linked)
                for (int64_t i = gt; i - threadIdx.x < n; i += nt) {
                    const int32_t v = i < n ? res_at(list, i) : -1;
                    for (int d = 0; d < 2; ++d)
                        if ((dirs >> d) & 1)
                            changed += res_pull_linked<K>(m, d, v, link[d], levels % kResAgain == kResAgain - 1, mix);
                }
            const int64_t gw = gt >> 5, nw = nt >> 5;
            for (int64_t i0 = gw * (32 * kResU); i0 < n && !linked; i0 += nw * (32 * kResU)) {
                int32_t v[kResU];
#pragma unroll
                for (int u = 0; u < kResU; ++u) {
                    const int64_t i = i0 + u * 32 + lane_id();
                    v[u] = i < n ? res_at(list, i) : -1;
                }
                for (int d = 0; d < 2; ++d) {
                    if (!((dirs >> d) & 1)) continue;
                    const unsigned ch = res_pull<K>(m, d, v, mix);
                    changed += __popc(ch);
                    if (!listing) continue;
                    unsigned g[kResU];
                    int tot = 0;
#pragma unroll
                    for (int u = 0; u < kResU; ++u) {
                        g[u] = __ballot_sync(kFull, (ch >> u) & 1u);
                        tot += __popc(g[u]);
                    }
                    if (!tot) continue;
                    unsigned long long at = 0;
                    if (lane_id() == 0) at = atomicAdd(qc + s, (unsigned long long)tot);
                    at = __shfl_sync(kFull, at, 0);
#pragma unroll
                    for (int u = 0; u < kResU; ++u) {
                        const unsigned long long to = at + __popc(g[u] & lanemask_lt());
                        if (((ch >> u) & 1u) && (int64_t)to < m.cap_q) m.q[0][to] = (uint32_t)v[u] | ((uint32_t)d << 31);
                        at += __popc(g[u]);
                    }
                }
            }
            const int64_t t = block_sum64(changed, sm.sum);
            if (threadIdx.x == 0 && t) atomicAdd(chg + s, (unsigned long long)t);
            if (!grid_sync(r.gsync, r.err)) return 0;
            prev = (int64_t)__ldcg(chg + s);
            nq = (int64_t)__ldcg(qc + s);
            s = s1;
            if (prev == 0) return 1;
            if (listing && nq <= m.cap_q) { dense = false; cur = hops = 0; }
            ++levels;
            ++passes;
            continue;
        }
        const uint32_t *qi = m.q[cur];
        uint32_t *qo = m.q[cur ^ 1];
        if (nq > kResTail) {
            unsigned long long *qn = qc + s;
            const int64_t cap = m.cap_q;
            for (int64_t i = gt; i - threadIdx.x < nq; i += nt)
                res_push<K>(m, i < nq, i < nq ? __ldcg(qi + i) : 0u, [&](unsigned grew, const uint32_t (&en)[4]) {
                    const int mine = __popc(grew);
                    if (!__any_sync(kFull, mine)) return;
                    int incl = mine;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(kFull, incl, o);
                        if (lane_id() >= o) incl += y;
                    }
                    unsigned long long at = 0;
                    if (lane_id() == 31) at = atomicAdd(qn, (unsigned long long)incl);
                    at = __shfl_sync(kFull, at, 31) + incl - mine;
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if ((grew >> q) & 1u) {
                            if ((int64_t)at < cap) qo[at] = en[q];
                            ++at;
                        }
                });
        } else if (blockIdx.x == 0) {
            int n0 = (int)nq, c = 0;
            for (int i = threadIdx.x; i < n0; i += kBlock) sm.q[0][i] = __ldcg(qi + i);
            if (threadIdx.x == 0) sm.cnt[0] = sm.cnt[1] = 0;
            __syncthreads();
            for (int lv = 0; n0 > 0 && n0 <= kResTail && lv < kResTailLevels; ++lv) {
                int *cn = &sm.cnt[c ^ 1];
                uint32_t *qn = sm.q[c ^ 1];
                for (int i = threadIdx.x; i - (int)threadIdx.x < n0; i += kBlock)
                    res_push<K>(m, i < n0, i < n0 ? sm.q[c][i] : 0u, [&](unsigned grew, const uint32_t (&en)[4]) {
                        if (!grew) return;
                        int at = atomicAdd(cn, __popc(grew));
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if ((grew >> q) & 1u) {
                                if (at < 2 * kResTail) qn[at] = en[q];
                                else if (at < m.cap_q) qo[at] = en[q];
                                ++at;
                            }
                    });
                __syncthreads();
                n0 = sm.cnt[c ^ 1];
                if (threadIdx.x == 0) sm.cnt[c] = 0;
                c ^= 1;
                __syncthreads();
            }
            // nothing left, a level for the grid again, or enough of them for now
            for (int i = threadIdx.x; i < min(n0, 2 * kResTail); i += kBlock) qo[i] = sm.q[c][i];
            if (threadIdx.x == 0) qc[s] = (unsigned long long)n0;
        }
        const int lv = nq > kResTail ? 1 : kResTailLevels;  // (at most, in CTA 0)
        levels += lv;
        hops += lv;
        if (!grid_sync(r.gsync, r.err)) return 0;
        nq = (int64_t)__ldcg(qc + s);
        s = s1;
        cur ^= 1;
        if (nq == 0) return 1;
        // a wide level, or entries that did not fit: dense passes again
        // (they see every vertex, so nothing unlisted is lost)
        if (nq > n / kResSparse || nq > m.cap_q || (K == R_MIN && hops > kResHops)) { dense = true; prev = n * 2; }
    }
    if (threadIdx.x == 0) atomicCAS(r.err, 0, kErrOverflow);
    return 0;
}

// Drop the list entries that lead out of their vertex's class (cls(v): its
// class, or what now tells it from the others of its old one).  A warp takes
// a group of 32 consecutive vertices, whose lists lie back to back (the
// build writes them so and pruning keeps it), reads the group's entries 32
// at a time, coalesced, and packs the kept ones to the group's front with
// one ballot per step; each lane counts what its vertex keeps.  (A thread
// per vertex storing its own kept entries took 6.6 ms for 2 x 65 M entries
// of 21 M vertices, this form 1.8 ms.)
template <typename Cls>
__device__ __forceinline__ void res_prune(const ResBufs &m, int d, int64_t v0, int64_t n, Cls cls) {
    const int lane = lane_id();
    const int64_t v = v0 + lane;
    const bool have = v < n;
    int32_t *adj = m.adj[d];
    const int32_t b0 = have ? m.beg[d][v] : 0, e0 = have ? m.end[d][v] : 0;
    const uint32_t c = have ? cls((int32_t)v) : kResDead;
    const int32_t len = e0 - b0;
    int32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
    }
    const int32_t total = __shfl_sync(kFull, incl, 31), base = __shfl_sync(kFull, b0, 0);
    const int32_t my0 = incl - len;  // my entries: [my0, incl) of the group's
    int32_t kept = 0, out = 0;
    for (int32_t k0 = 0; k0 < total; k0 += 32) {
        const int32_t k = k0 + lane;
        int o = 0;  // owner: the number of lanes whose inclusive prefix is <= k
#pragma unroll
        for (int st = 16; st; st >>= 1)
            if (__shfl_sync(kFull, incl, o + st - 1) <= k) o += st;
        const uint32_t co = __shfl_sync(kFull, c, o & 31);
        const int32_t w = k < total ? res_adj<true>(m, adj, base + k) : -1;
        const bool keep = w >= 0 && cls(w) == co;
        const unsigned g = __ballot_sync(kFull, keep);
        if (keep && ICHK(base + out >= 0 && base + out < m.cap_e, 24, base + out))
            __stcg(adj + base + out + __popc(g & lanemask_lt()), w);
        out += __popc(g);
        // the step's bits that are mine: entries [my0, incl) - k0, cut to [0, 32)
        const int32_t lo = max(0, my0 - k0), hi = min(32, incl - k0);
        if (lo < hi) kept += __popc(g & ((hi == 32 ? kFull : (1u << hi) - 1u) & ~((1u << lo) - 1u)));
    }
    int32_t nincl = kept;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(kFull, nincl, o);
        if (lane >= o) nincl += y;
    }
    if (have) {
        m.beg[d][v] = base + nincl - kept;
        m.end[d][v] = base + nincl;
    }
}

// The same for one vertex, where few of a group are left: its kept entries
// move to the front of its own list.
template <typename Cls>
__device__ __forceinline__ void res_prune_one(const ResBufs &m, int32_t v, Cls cls) {
    const uint32_t c = cls(v);
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        const int32_t b = m.beg[d][v], e = m.end[d][v];
        int32_t *adj = m.adj[d];
        int32_t p = b;
        for (int32_t k = b; k < e; k += 4) {
            int32_t u[4];
            uint32_t cu[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) u[q] = k + q < e ? res_adj<true>(m, adj, k + q) : -1;
#pragma unroll
            for (int q = 0; q < 4; ++q) cu[q] = u[q] >= 0 ? cls(u[q]) : ~c;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (cu[q] == c) {
                    if (p != k + q) __stcg(adj + p, u[q]);
                    ++p;
                }
        }
        if (p != e) m.end[d][v] = p;
    }
}

// Splitting rounds (forward and backward in turn) over all vertices (it = 0)
// or the ones the tiles before left (m.list), then the weakly connected components
// of what the lists still join: components of at most kTileV vertices get a
// run of m.order (those of at most kTileT back to back from the front, larger
// ones one by one from the back) for k_tiles, the vertices of larger ones go
// to the next list.
__global__ void __launch_bounds__(kBlock, 2) k_split(Run<int32_t> r, Ext<int32_t> x, ResBufs m, int it) {
    pdl_wait();  // predecessor done, its writes visible
    pdl_trigger();
    if (!__ldcg(x.ctl + K_CMP_OK)) return;
    __shared__ ResSmem sm;
    const int64_t n = (int64_t)__ldcg(x.ctl + K_LARGE);
    const int64_t nl = it ? (int64_t)__ldcg(x.ctl + K_RES_LEFT + it - 1) : n;
    if (nl == 0) return;
    const int32_t *list = it ? m.list[(it - 1) & 1] : nullptr;
    const int64_t gt = (int64_t)blockIdx.x * kBlock + threadIdx.x;
    const int64_t nt = (int64_t)gridDim.x * kBlock;
    const int lane = lane_id();
    unsigned long long *chg = x.ctl + K_RES_CHG, *qc = x.ctl + K_RES_Q;
    unsigned long long *work = x.ctl + K_RES_WORK + kResWork * it;
    int32_t *uf = reinterpret_cast<int32_t *>(m.cls);
    int32_t *cnt = m.mn, *base = m.size;
    // the labelling rounds take what is left if it is little, or if the last time
    // ended next to nothing: one SCC, on which masks are lost
    const int64_t before = it > 1 ? (int64_t)__ldcg(x.ctl + K_RES_LEFT + it - 2) : n;
    if (it && (nl < n / kResFew || 10 * nl > 9 * before || __ldcg(x.ctl + K_RES_STOP))) {
        for (int64_t i = gt; i < nl; i += nt) m.list[it & 1][i] = res_at(list, i);
        if (gt == 0) x.ctl[K_RES_LEFT + it] = (unsigned long long)nl;
        return;
    }
    // masks as wide as their array stays in L2 (gathers from both dies: about
    // half of its 126 MB): wider ones split more per round
    const bool wide = n <= kResWideN;
    const int bits = wide ? 6 : 4;  // log2 of the pivots per class aimed at
    // (what k_super left of the large WCCs has mostly fallen apart: its
    // components first)
    const int rounds_now = it ? 2 : __ldcg(x.ctl + K_SUP_LEFT) ? 0 : wide ? 3 : 4;
    if (gt < 3) { chg[gt] = 0ull; qc[gt] = 0ull; }
    for (int64_t i = gt; i < nl; i += nt) {
        int32_t root, size;
        const int32_t v = res_at(list, i);
        if (it == 0) {  // the WCCs
            root = m.parent[m.old[v]];
            size = m.wsize[root];
            m.end[0][v] = m.beg[0][v + 1];
            m.end[1][v] = m.beg[1][v + 1];
        } else {  // the components of the last time
            root = uf[v];
            size = cnt[root];
        }
        m.cls[v] = (mix32((uint32_t)root) & kResHash) | ((uint32_t)(31 - __clz(max(1, size))) << 27);
    }
    if (!grid_sync(r.gsync, r.err)) return;  // parent and wsize are read: their space is free
    int s = 0, rounds = it ? (int)__ldcg(r.counters + C_COLOR_ROUNDS) : 0;
    for (int k = 0; k < rounds_now; ++k) {
        const int d = k & 1;
        unsigned long long *v64 = reinterpret_cast<unsigned long long *>(m.val[d]);
        unsigned short *v16 = reinterpret_cast<unsigned short *>(m.val[d]);
        if (gt == 0) { chg[s == 2 ? 0 : s + 1] = 0ull; qc[s == 2 ? 0 : s + 1] = 0ull; }
        for (int64_t i = gt; i < nl; i += nt) {
            const int32_t v = res_at(list, i);
            const uint32_t h = mix32((uint32_t)v * 16u + (uint32_t)(4 * it + k) + 1u);
            const int shift = max(kResSplitShift, (int)(m.cls[v] >> 27) - bits * (it ? 1 : k + 1));
            const bool pivot = (h >> (32 - shift)) == 0u;
            if (wide) v64[v] = pivot ? 1ull << (mix32(h) & 63u) : 0ull;
            else v16[v] = pivot ? (unsigned short)(1u << (mix32(h) & 15u)) : (unsigned short)0;
            if (pivot) {
                const unsigned long long at = atomicAdd(qc + s, 1ull);
                if ((int64_t)at < m.cap_q) m.q[0][at] = (uint32_t)v | ((uint32_t)d << 31);
            }
        }
        if (!grid_sync(r.gsync, r.err)) return;
        const int ok = wide ? res_spread<R_OR64>(r, m, chg, qc, x.ctl + K_LARGE, list, nl, 1 << d, s, sm, true, LabelMix<32>(0))
                            : res_spread<R_OR16>(r, m, chg, qc, x.ctl + K_LARGE, list, nl, 1 << d, s, sm, true, LabelMix<32>(0));
        if (ok == 0) return;
        if (ok == 2) {  // these masks say nothing; the labelling rounds take what no tile does
            if (gt == 0) x.ctl[K_RES_STOP] = 1ull;
            break;
        }
        for (int64_t i = gt; i < nl; i += nt) {
            const int32_t v = res_at(list, i);
            const uint32_t c = m.cls[v];
            const unsigned long long y = wide ? __ldcg(v64 + v) : (unsigned long long)__ldcg(v16 + v);
            m.cls[v] = (mix32(c ^ mix32((uint32_t)y ^ mix32((uint32_t)(y >> 32)))) & kResHash) | (c & ~kResHash);
        }
        const auto prune = [&](auto cls) {
            if (4 * nl >= n)
                for (int64_t g = gt >> 5; g * 32 < n; g += nt >> 5) {
                    res_prune(m, 0, g * 32, n, cls);
                    res_prune(m, 1, g * 32, n, cls);
                }
            else
                for (int64_t i = gt; i < nl; i += nt) res_prune_one(m, res_at(list, i), cls);
        };
        // an entry led to the same class before, so 16-bit masks tell where it
        // leads now: half the words to gather (21 M vertices, 84 MB of class words: 1.4-1.9 ms a round)
        if (wide) {
            if (!grid_sync(r.gsync, r.err)) return;
            prune([&](int32_t w) { return __ldcg(m.cls + w); });
        } else {
            prune([&](int32_t w) { return (uint32_t)__ldcg(v16 + w); });
        }
        if (!grid_sync(r.gsync, r.err)) return;
        ++rounds;
    }
    // components: union-find over the class words (dead now), root = minimum
    int32_t *first = reinterpret_cast<int32_t *>(m.val[1]);  // [tiles]: start of the first component in each tile
    const int64_t tiles = nl / kTileT + 1;
    for (int64_t i = gt; i < nl; i += nt) {
        const int32_t v = res_at(list, i);
        uf[v] = v;
        cnt[v] = 0;
    }
    for (int64_t i = gt; i < tiles; i += nt) first[i] = 0x7fffffff;
    if (!grid_sync(r.gsync, r.err)) return;
    for (int64_t i = gt; i < nl; i += nt) {
        const int32_t v = res_at(list, i);
        for (int32_t k = m.beg[0][v], e = m.end[0][v]; k < e; ++k) uf_hook(uf, v, res_adj<true>(m, m.adj[0], k));
    }
    if (!grid_sync(r.gsync, r.err)) return;
    for (int64_t i = gt; i - threadIdx.x < nl; i += nt) {
        const int32_t v = i < nl ? res_at(list, i) : -1;
        const int32_t root = v >= 0 ? uf_root(uf, v) : -1;
        if (v >= 0) uf[v] = root;
        const unsigned grp = __match_any_sync(kFull, root);
        if (root >= 0 && lane == __ffs(grp) - 1) atomicAdd(cnt + root, __popc(grp));
    }
    if (!grid_sync(r.gsync, r.err)) return;
    for (int64_t i = gt; i - threadIdx.x < nl; i += nt) {  // a run of m.order for each component that fits a tile
        const int32_t v = i < nl ? res_at(list, i) : -1;
        const bool root = v >= 0 && uf[v] == v;
        const int32_t c = root ? __ldcg(cnt + v) : 0;
        const bool small = c > 0 && c <= kTileT, mid = c > kTileT && c <= kTileV;
        const int32_t cs = small ? c : 0;
        int32_t incl = cs;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
        }
        const int32_t tot = __shfl_sync(kFull, incl, 31);
        unsigned long long at = 0;
        if (lane == 31 && tot) at = atomicAdd(work + W_SMALL, (unsigned long long)tot);
        at = __shfl_sync(kFull, at, 31);
        int32_t b = -1;
        if (small) {
            b = (int32_t)at + incl - c;
            atomicMin(first + b / kTileT, b);
        } else if (mid) {
            b = (int32_t)(nl - (int64_t)atomicAdd(work + W_BACK, (unsigned long long)c)) - c;
            const unsigned long long q = atomicAdd(work + W_MID, 1ull);
            if (VOK((long long)(2 * q + 1), 28)) {  // (a mid component has over two vertices: q fits)
                m.q[0][2 * q] = (uint32_t)b;
                m.q[0][2 * q + 1] = (uint32_t)c;
            }
        }
        if (root) base[v] = b;
    }
    if (!grid_sync(r.gsync, r.err)) return;
    for (int64_t i = gt; i - threadIdx.x < nl; i += nt) {
        bool big = false;
        int32_t v = 0;
        if (i < nl) {
            v = res_at(list, i);
            const int32_t root = uf[v], b = base[root];
            big = b < 0;
            if (!big) {
                const int32_t at = b + atomicSub(cnt + root, 1) - 1;
                if (VOK(at, 25)) m.order[at] = v;
                m.pos[v] = at;
            }
        }
        wl_append(big, v, m.list[it & 1], x.ctl + K_RES_LEFT + it);
    }
    if (gt == 0) r.counters[C_COLOR_ROUNDS] = (unsigned long long)rounds;
}

// ---------------------------------------------------------------------------
// The components that start in kTileT consecutive entries of m.order, or one
// component of up to kTileV vertices, as a tile (tile.cuh) of a CTA.
constexpr int kTilePer = kTileV / kTileThreads;

__global__ void __launch_bounds__(kTileThreads, 1) k_tiles(Run<int32_t> r, Ext<int32_t> x, ResBufs m, int it) {
    pdl_wait();  // predecessor done, its writes visible
    pdl_trigger();
    if (!__ldcg(x.ctl + K_CMP_OK)) return;
    extern __shared__ __align__(16) unsigned char tile_raw[];
    TileSmem &t = *reinterpret_cast<TileSmem *>(tile_raw);
    const int tid = threadIdx.x, lane = tid & 31;
    unsigned long long *work = x.ctl + K_RES_WORK + kResWork * it;
    const int64_t n_small = (int64_t)__ldcg(work + W_SMALL), n_mid = (int64_t)__ldcg(work + W_MID);
    const int64_t tiles = (n_small + kTileT - 1) / kTileT;
    const int32_t *first = reinterpret_cast<const int32_t *>(m.val[1]);
    int64_t done = 0, sccs = 0;
    for (;;) {
        __syncthreads();  // the previous tile's readers are done
        if (tid == 0) {
            // larger pieces first
            const int64_t w = (int64_t)atomicAdd(work + W_TILE, 1ull);
            int64_t a = 0, z = -1;
            if (w < n_mid) {
                a = (int64_t)m.q[0][2 * w];
                z = a + (int64_t)m.q[0][2 * w + 1];
            } else if (w - n_mid < tiles) {
                const int64_t k = w - n_mid;
                a = first[k];
                z = n_small;
                for (int64_t j = k + 1; j < tiles; ++j)
                    if (first[j] != 0x7fffffff) { z = first[j]; break; }
                if (a > z) a = z;  // no component starts here
            }
            t.start = (int32_t)a;
            t.count = (int32_t)(z - a);  // -1: no more work
            t.edges = 0;
        }
        __syncthreads();
        const int n = t.count, start = t.start;
        if (n < 0) break;
        if (n == 0 || !ICHK(n <= kTileV && start >= 0, 27, ((long long)start << 32) | n)) continue;
        for (int i = tid; i < n; i += kTileThreads) t.f[i] = m.old[res_at(m.order, start + i)];
        for (int i = tid; i < kTileV / 32; i += kTileThreads) t.dead[i] = 0u;
        tile_sort(t, n);
        int32_t e0[kTilePer];  // the list of each of my vertices
        for (int u = 0; u < kTilePer && u * kTileThreads < n; ++u) {
            const int i = u * kTileThreads + tid;
            int32_t d = 0;
            if (i < n) {
                const int32_t v = m.order[start + t.b[i]];
                e0[u] = m.beg[1][v];
                d = m.end[1][v] - e0[u];
            }
            int32_t incl = d;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t y = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += y;
            }
            int32_t at = 0;
            if (lane == 31) at = atomicAdd(&t.edges, min(incl, kTileE + 1));  // (the sum of 32 lists stays far below 2^31)
            at = __shfl_sync(kFull, at, 31);
            if (i < n) {
                t.off[i] = (uint16_t)min(at + incl - d, 0xffff);
                t.len[i] = (uint16_t)min(d, 0xffff);
            }
        }
        __syncthreads();
        if (t.edges > kTileE) {  // too dense for a tile: the labelling rounds take it
            for (int i = tid; i - tid < n; i += kTileThreads)
                wl_append(i < n, i < n ? m.order[start + i] : 0, m.list[it & 1], x.ctl + K_RES_LEFT + it);
            continue;
        }
#pragma unroll
        for (int u = 0; u < kTilePer; ++u) {
            const int i = u * kTileThreads + tid;
            if (i >= n) break;
            const int d = t.len[i], o = t.off[i];
            for (int k = 0; k < d; k += 4) {
                int32_t w[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) w[q] = k + q < d ? res_adj<true>(m, m.adj[1], e0[u] + k + q) : -1;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (w[q] < 0) continue;
                    const int p = __ldcg(m.pos + w[q]) - start;
                    if (ICHK(p >= 0 && p < n && o + k + q < kTileE, 26, ((long long)p << 32) | (o + k + q)))
                        t.adj[o + k + q] = (uint16_t)t.f[p];
                }
            }
        }
        tile_solve(t, n, r, done, sccs);
    }
        tile_report(r, done, sccs);
}

// Labelling rounds of the vertices that no tile took, to the end.
__global__ void __launch_bounds__(kBlock, 2) k_resolve(Run<int32_t> r, Ext<int32_t> x, ResBufs m) {
    pdl_wait();  // predecessor done, its writes visible
    pdl_trigger();
    if (!__ldcg(x.ctl + K_CMP_OK)) return;
    __shared__ ResSmem sm;
    const int64_t gt = (int64_t)blockIdx.x * kBlock + threadIdx.x;
    const int64_t nt = (int64_t)gridDim.x * kBlock;
    unsigned long long *chg = x.ctl + K_RES_CHG, *qc = x.ctl + K_RES_Q, *left = x.ctl + K_RES_LEFT;
    int64_t nl = (int64_t)__ldcg(left + kResIts - 1);  // (the slots rotate from there)
    if (nl == 0) return;
    if (gt < 3) { chg[gt] = 0ull; qc[gt] = 0ull; }
    if (gt == 0) left[0] = 0ull;
    int s = 0, rounds = (int)__ldcg(r.counters + C_COLOR_ROUNDS);
    const int32_t *list = m.list[(kResIts - 1) & 1];
    for (int k = 0;; ++k) {
        int32_t *next = m.list[(kResIts + k) & 1];
        unsigned long long *n_next = left + k % 3;
        if (gt == 0) left[(k + 1) % 3] = 0ull;
        const LabelMix<32> mix(k);
        for (int64_t i = gt; i < nl; i += nt) {
            const int32_t v = res_at(list, i);
            m.val[0][v] = m.val[1][v] = mix.label((uint32_t)v);
            m.mn[v] = 0x7fffffff;
            m.size[v] = 0;
        }
        if (!grid_sync(r.gsync, r.err)) return;
        if (res_spread<R_MIN>(r, m, chg, qc, x.ctl + K_LARGE, list, nl, 3, s, sm, false, mix) != 1) return;
        for (int64_t i = gt; i < nl; i += nt) {
            const int32_t v = res_at(list, i);
            const uint32_t f = __ldcg(m.val[0] + v);
            if (f == __ldcg(m.val[1] + v)) {
                const uint32_t p = res_holder(mix, f);
                atomicMin(m.mn + p, m.old[v]);
                atomicAdd(m.size + p, 1);
            }
        }
        if (!grid_sync(r.gsync, r.err)) return;
        int64_t done = 0, roots = 0;
        for (int64_t i = gt; i - threadIdx.x < nl; i += nt) {
            bool keep = false;
            int32_t v = 0;
            if (i < nl) {
                v = res_at(list, i);
                const uint32_t f = __ldcg(m.val[0] + v), b = __ldcg(m.val[1] + v);
                keep = f != b;
                if (keep) {
                    m.cls[v] = mix32(f ^ mix32(b)) & 0x7fffffffu;
                } else {
                    const int32_t ov = m.old[v];
                    r.label[ov] = __ldcg(m.mn + res_holder(mix, f));
                    r.cls[ov] = CLS_MICE;
                    clear_bit(r.A, ov);
                    m.cls[v] = kResDead;
                    ++done;
                    if ((int32_t)mix.holder(f) == v) {  // one histogram entry per SCC
                        const int32_t sz = __ldcg(m.size + v);
                        if (sz < kHistCap) {
                            atomicAdd((unsigned long long *)(r.hist + sz), 1ull);
                        } else {
                            const unsigned long long at = atomicAdd(r.counters + C_BIG, 1ull);
                            if (at < kBigCap) r.hist[kHistCap + at] = sz;
                        }
                        ++roots;
                    }
                }
            }
            wl_append(keep, v, next, n_next);
        }
        const int64_t a = block_sum64(done, sm.sum), b = block_sum64(roots, sm.sum);
        if (threadIdx.x == 0) {
            if (a) atomicAdd(r.counters + C_MICE_V, (unsigned long long)a);
            if (b) atomicAdd(r.counters + C_MICE_SCC, (unsigned long long)b);
        }
        if (!grid_sync(r.gsync, r.err)) return;
        const int64_t nn = (int64_t)__ldcg(n_next);
        if (blockIdx.x == 0 && threadIdx.x == 0 && rounds < kTraceLevels) {  // diagnostics
            long long *t = r.trace + ((long long)2 * kTraceLevels + rounds) * 4;
            t[0] = rounds + 1;
            t[1] = nl;
            t[2] = nl - nn;
            t[3] = (long long)globaltimer();
        }
        ++rounds;
        if (nn == 0) break;
        if (nn >= nl) {  // every round finds the SCC of each class's lowest label
            if (threadIdx.x == 0) atomicCAS(r.err, 0, kErrOverflow);
            return;
        }
        list = next;
        nl = nn;
        for (int64_t i = gt; i < nl; i += nt) res_prune_one(m, res_at(list, i), [&](int32_t w) { return __ldcg(m.cls + w); });
        if (!grid_sync(r.gsync, r.err)) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) r.counters[C_COLOR_ROUNDS] = (unsigned long long)rounds;
}

}  // namespace ispan
