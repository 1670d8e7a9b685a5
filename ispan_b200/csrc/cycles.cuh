// cycles.cuh -- cycles along near ids, contracted before the WCC stage, and
// the peel of the contracted large WCCs.
//
// On a DAG of planted cycles (a batch of such graphs: half of its vertices)
// every search has to walk every ring, up to 1,000 hops one after the other,
// and classes split over ~20 rounds.  Where ids have locality -- each
// vertex's nearest in-neighbour by id is usually the one before it on a
// cycle -- the rings can be had directly:
//   k_cycles  every residual vertex points at its active in-neighbour of the
//             nearest id; a vertex whose pointer leads to a higher id walks
//             the pointers, and if it comes back to itself without meeting a
//             lower id, the walk is a cycle of the graph and the vertex its
//             minimum.  A cycle's vertices belong to one SCC whatever the
//             pointers were chosen by, so they are one node from here on (rep
//             = the minimum).  A ring with a chord, or whose closing edge is
//             not the nearest one, is left in pieces: then the nodes choose
//             again, a single vertex its nearest in-neighbour (a single one
//             if there is any), a node of several vertices the nearest single
//             one, and cycles of nodes are joined.
//   WCC stage starts its union-find from rep.
//   k_super   order the nodes of the large WCCs by id.  A cycle through
//             several nodes goes down somewhere between any two neighbours of
//             the nodes it spans, so a node that no descending edge's span
//             covers is an SCC: one pass over the edges and one scan over the
//             ids end every node of a DAG whose ids are a topological order
//             (rings in their order, time-ordered ids).  If most of it is
//             left, the nodes are peeled like the vertices of trim-1
//             (src/trim_1_gfq.h:365-458): a node without active in- or
//             out-edges to other nodes is an SCC.  What remains goes on to the
//             large-WCC path as single vertices.
// Whether ids have such locality is sampled first; without it (web-shaped
// graphs with permuted ids) both kernels return at once.
//
// A batch of 512 graphs (82 M vertices, 42 M residual), one B200: colouring
// 250 ms of a run's 298; k_cycles 3.0 ms (list reads 2.0, the rest latency of
// walks) and k_super 3.5 ms (one edge pass, a scan, the labels), a run 27-35 ms.
// With the peel alone instead of the spans 32 ms and 18 ms for what rings in
// pieces kept from it.
#pragma once
#include "stages.cuh"

namespace ispan {

constexpr int64_t kCycMin = 1 << 15;  // fewer residual vertices: most WCCs fit a tile, which takes less than these kernels
constexpr int kCycSample = 2048;    // residual vertices sampled
constexpr int kCycNear = 1024;      // an in-neighbour this near counts; a quarter of the sample must have one
constexpr int kCycMax = 1 << 12;    // longest walk, in runs of consecutive ids (later: in nodes)
constexpr int kCycSteps = 64;       // steps (32 consecutive ids, or a node) of a walk over nodes while ids are its priorities
constexpr int kCycTries = 2;        // times the nodes choose again, while single vertices are joined
constexpr int kSuperTail = 1024;    // a round of the peel of at most this many vertices: one CTA alone
constexpr int kSuperTailRounds = 256;

struct CycBufs {
    int32_t *par;     // [V] nearest in-neighbour; later, at a single vertex, the lowest id of the cycle it found
    int32_t *skip;    // [V] where the run of consecutive ids that the pointers follow from here ends; later, at a
                      // single vertex, the number of nodes of the cycle it found (0: none)
    int32_t *rep;     // [V] minimum of the vertex's node
    int32_t *size;    // [V] at a node's minimum: its vertices
    unsigned long long *key;  // [V] first: at a run's end, the walk through it (minimum, entry); then, at a node's
                              // minimum, its choice (other than single, distance, in-neighbour); in the peel, at a
                              // node's minimum, its place in order
    int32_t *order;   // [V] vertices by node (the peel)
    int32_t *single;  // [V] vertices on no cycle after the first walk (overlays q[0])
    int32_t *q[2];    // [V] peeled vertices
};

// active in-neighbour of v nearest by id (other than v), v if there is none
template <typename OffT>
__device__ __forceinline__ int32_t nearest_in(const Run<OffT> &r, int32_t v) {
    int32_t best = v;
    int64_t dist = INT64_MAX;
    for (int64_t e = ld_off(r.bw_beg, v), e1 = ld_off(r.bw_beg, v + 1); e < e1; e += 4) {
        int32_t u[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) u[q] = e + q < e1 ? ld_adj(r.bw_adj, e + q) : v;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int64_t d = u[q] > v ? (int64_t)u[q] - v : (int64_t)v - u[q];
            if (u[q] != v && d < dist && bitc(r.A, u[q])) {
                best = u[q];
                dist = d;
            }
        }
    }
    return best;
}

__device__ __forceinline__ int32_t cyc_node(const CycBufs &b, int32_t v) {  // v's node (joined ones follow one another)
    if (!VOK(v, 34)) return 0;
    int32_t a = __ldcg(b.rep + v);
    if (!VOK(a, 35)) return 0;
    for (int32_t c; (c = __ldcg(b.rep + a)) != a;) a = c;
    return a;
}

// What a single vertex v puts up for choice: itself to the nodes of its
// out-neighbours, and to itself its in-neighbours.
__device__ __forceinline__ unsigned long long cyc_dist(int32_t a, int32_t b) {
    return (unsigned long long)(a > b ? (int64_t)a - b : (int64_t)b - a) << 31;
}
template <typename OffT>
__device__ __forceinline__ void choose_single(const Run<OffT> &r, const CycBufs &b, int32_t v) {
    unsigned long long best = ~0ull;
    for (int64_t e = ld_off(r.bw_beg, v), e1 = ld_off(r.bw_beg, v + 1); e < e1; ++e) {
        const int32_t u = ld_adj(r.bw_adj, e);
        if (u == v || !bitc(r.A, u)) continue;
        best = min(best, (bitv(r.D, u) ? 1ull << 62 : 0ull) | cyc_dist(u, v) | (unsigned)u);
    }
    if (best != ~0ull) atomicMin(b.key + v, best);
    for (int64_t e = ld_off(r.fw_beg, v), e1 = ld_off(r.fw_beg, v + 1); e < e1; ++e) {
        const int32_t w = ld_adj(r.fw_adj, e);
        if (w != v && bitc(r.A, w) && bitv(r.D, w)) atomicMin(b.key + cyc_node(b, w), cyc_dist(v, w) | (unsigned)v);
    }
}

__device__ __forceinline__ int32_t cyc_next(const CycBufs &b, int32_t node) {
    const unsigned long long k = __ldcg(b.key + node);
    return k == ~0ull ? node : cyc_node(b, (int32_t)(k & 0x7fffffffu));
}

// How many hops a walk over nodes goes from u along consecutive ids in steps
// of dir, all over single vertices: a warp looks at 32 of them at once.  (Hop by
// hop, three dependent reads each, the walks of rings of up to 1,000 took most
// of this kernel: on 97 separate graphs 3.1 ms before, 0.31 so; on 512 graphs in
// one batch 6.5 and 3.0.)
template <typename OffT>
__device__ __forceinline__ int cyc_run(const Run<OffT> &r, const CycBufs &b, int32_t u, int dir) {
    const int64_t x = (int64_t)u + (int64_t)lane_id() * dir;
    const bool single = x >= 0 && x < r.V && bitc(r.A, x) && !bitv(r.D, x);
    const unsigned long long k = single ? __ldcg(b.key + x) : ~0ull;
    const bool hop = k != ~0ull && (int64_t)(k & 0x7fffffffu) == x + dir;
    const unsigned s = __ballot_sync(kFull, single);
    return __ffs(~(__ballot_sync(kFull, hop) & (s >> 1))) - 1;
}

// skip: pointers mostly lead to the id next to their own; runs of such
// pointers are passed in one step.  A descending run (bits in P) ends at the
// last id before whose bit is not set, an ascending one (bits in D) at the
// next.  Each CTA scans a range of words, 512 at a time: a thread per word
// for the carries, then a lane per id; tot holds the ranges' last and first
// unset ids.  (Scanning the pointers themselves, both ways, took 2.4 ms for
// 82 M ids.)  D is left clear.  False if a grid barrier failed.
template <typename OffT>
__device__ __forceinline__ bool cyc_skip(const Run<OffT> &r, const CycBufs &b, int32_t *tot) {
    __shared__ int32_t sw[kWarps], carry[kBlock];
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    const int64_t per = (r.W + gridDim.x - 1) / gridDim.x;
    const int64_t c0 = min(r.W, (int64_t)blockIdx.x * per), c1 = min(r.W, c0 + per);
    for (int dir = 0; dir < 2; ++dir) {
        // dir 0: last unset id of a word (a maximum), dir 1: the first (a maximum of -id), from the other end
        const uint32_t *bits = dir == 0 ? r.P : r.D;
        const auto edge = [&](int64_t w) {
            const uint32_t z = ~__ldcg(bits + w);
            if (z == 0) return INT32_MIN;
            return dir == 0 ? (int32_t)(w * 32 + 31 - __clz(z)) : -(int32_t)(w * 32 + __ffs(z) - 1);
        };
        int32_t best = INT32_MIN;
        for (int64_t w = c0 + threadIdx.x; w < c1; w += kBlock) best = max(best, edge(w));
        best = __reduce_max_sync(kFull, best);
        __syncthreads();
        if (lane == 0) sw[warp] = best;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 0; k < kWarps; ++k) best = max(best, sw[k]);
            tot[dir * gridDim.x + blockIdx.x] = best;
        }
    }
    if (!grid_sync(r.gsync, r.err)) return false;
    for (int dir = 0; dir < 2; ++dir) {
        const uint32_t *bits = dir == 0 ? r.P : r.D;
        int32_t run = INT32_MIN;
        for (int k = threadIdx.x; k < gridDim.x; k += kBlock)
            if (dir == 0 ? k < (int)blockIdx.x : k > (int)blockIdx.x) run = max(run, __ldcg(tot + dir * gridDim.x + k));
        run = __reduce_max_sync(kFull, run);
        __syncthreads();
        if (lane == 0) sw[warp] = run;
        __syncthreads();
        for (int k = 0; k < kWarps; ++k) run = max(run, sw[k]);
        for (int64_t i0 = 0; i0 < c1 - c0; i0 += kBlock) {
            const int64_t i = i0 + threadIdx.x, w = dir == 0 ? c0 + i : c1 - 1 - i;
            const uint32_t m = i < c1 - c0 ? __ldcg(bits + w) : 0u, z = ~m;
            int32_t x = i >= c1 - c0 || z == 0 ? INT32_MIN
                        : dir == 0 ? (int32_t)(w * 32 + 31 - __clz(z)) : -(int32_t)(w * 32 + __ffs(z) - 1);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t y = __shfl_up_sync(kFull, x, o);
                if (lane >= o) x = max(x, y);
            }
            __syncthreads();
            if (lane == 31) sw[warp] = x;
            int32_t before = __shfl_up_sync(kFull, x, 1);
            if (lane == 0) before = INT32_MIN;
            __syncthreads();
            int32_t all = run;
            for (int k = 0; k < kWarps; ++k) {
                if (k < warp) before = max(before, sw[k]);
                all = max(all, sw[k]);
            }
            carry[threadIdx.x] = max(before, run);
            run = all;
            __syncwarp();
            // the warp's 32 words, a lane per id
            for (int k = 0; k < 32; ++k) {
                const uint32_t mk = __shfl_sync(kFull, m, k);
                const int64_t wk = __shfl_sync(kFull, w, k);
                const bool in = i0 + warp * 32 + k < c1 - c0;
                if (!in) break;
                const int64_t v = wk * 32 + lane;
                const int32_t c = carry[warp * 32 + k];
                if (dir == 0) {
                    const uint32_t below = ~mk & (kFull >> (31 - lane));  // unset ids up to mine
                    if (v < r.V) b.skip[v] = below ? (int32_t)(wk * 32 + 31 - __clz(below)) : c;
                } else if ((mk >> lane) & 1u) {
                    const uint32_t above = ~mk & (kFull << lane);
                    if (v < r.V) b.skip[v] = above ? (int32_t)(wk * 32 + __ffs(above) - 1) : -c;
                }
            }
            __syncwarp();
        }
        __syncthreads();
    }
    if (!grid_sync(r.gsync, r.err)) return false;
    for (int64_t w = c0 + threadIdx.x; w < c1; w += kBlock) r.D[w] = 0u;
    return true;
}

template <typename OffT>
__global__ void __launch_bounds__(kBlock, 2) k_cycles(Run<OffT> r, Ext<OffT> x, CycBufs b) {
    pdl_wait();  // predecessor done, its writes visible
    pdl_trigger();
    if (__ldcg(x.ctl + K_TINY)) return;  // the residual was solved in one CTA
    const int64_t gt = (int64_t)blockIdx.x * kBlock + threadIdx.x;
    const int64_t nt = (int64_t)gridDim.x * kBlock;
    const int64_t n = (int64_t)__ldcg(x.ctl + K_WL0);
    if (n < kCycMin) return;
    const int32_t *wl = r.wl[0];
    // the sample: every CTA takes the same one, so all agree without a barrier
    __shared__ int s_near;
    if (threadIdx.x == 0) s_near = 0;
    __syncthreads();
    const int ns = (int)min(n, (int64_t)kCycSample);
    int near = 0;
    for (int k = threadIdx.x; k < ns; k += kBlock) {
        const int32_t v = wl[(int64_t)k * n / ns];
        bool has = false;
        for (int64_t e = ld_off(r.bw_beg, v), e1 = min(ld_off(r.bw_beg, v + 1), e + 16); e < e1; ++e) {
            const int32_t u = ld_adj(r.bw_adj, e);
            if (u == v || !bitc(r.A, u)) continue;
            has |= abs((long long)u - v) <= kCycNear;
        }
        near += has;
    }
    near = __reduce_add_sync(kFull, near);
    if (lane_id() == 0) atomicAdd(&s_near, near);
    __syncthreads();
    if (4 * s_near < ns) return;
    if (gt == 0) x.ctl[K_CYC_ON] = 1ull;
    // pointers, by words of the active map (P, D: pointers to the id before,
    // to the one after)
    for (int64_t w = gt >> 5; w < r.W; w += nt >> 5) {
        const uint32_t m = r.A[w];
        const int32_t v = (int32_t)(w * 32 + lane_id());
        int32_t p = v;
        if ((m >> lane_id()) & 1u) {
            p = nearest_in(r, v);
            b.par[v] = p;
            b.rep[v] = v;
            b.size[v] = 1;
            b.key[v] = ~0ull;
        }
        const uint32_t dn = __ballot_sync(kFull, p == v - 1), up1 = __ballot_sync(kFull, p == v + 1);
        if (lane_id() == 0) {
            r.P[w] = dn;
            r.D[w] = up1;
        }
    }
    if (!grid_sync(r.gsync, r.err)) return;
    if (!cyc_skip(r, b, x.large[1])) return;
    // D, clear from here on: vertices on a cycle found (the trims' claims in
    // it are no longer read).  Walks along the pointers, run by run: a cycle's minimum writes itself
    // and the place where it entered to the end of each run it passes
    for (int64_t i = gt; i < n; i += nt) {
        const int32_t v = wl[i];
        int32_t u = __ldcg(b.par + v), h = v;
        if (u <= v) continue;
        int hops = 0, len = 0, renew = 1;
        // (a mark renewed at powers of two: met again, the walk is in a cycle of
        // higher ids, without v)
        for (int32_t mark = u; hops < kCycMax && u > v; ++hops) {
            h = __ldcg(b.skip + u);
            if (!VOK(h, 39)) break;
            len += abs(u - h) + 1;
            if (h <= v) break;  // v ends descending runs, its own pointer leads up
            u = __ldcg(b.par + h);
            if (u == mark) break;
            if (hops == renew) {
                mark = u;
                renew *= 2;
            }
        }
        if (u == v) ++len;
        else if (h != v) continue;  // met a lower id or another cycle, or too long
        u = __ldcg(b.par + v);
        for (int k = 0; k <= hops; ++k) {
            h = u == v ? v : __ldcg(b.skip + u);
            if (!VOK(h, 39)) break;
            b.key[h] = (unsigned long long)(unsigned)v << 32 | (unsigned)u;
            if (h == v) break;
            u = __ldcg(b.par + h);
        }
        b.size[v] = len;
    }
    if (!grid_sync(r.gsync, r.err)) return;
    for (int64_t i = gt; i - lane_id() < n; i += nt) {
        int32_t v = 0;
        bool left = false;
        if (i < n) {
            v = wl[i];
            const int32_t h = __ldcg(b.skip + v);
            const unsigned long long k = VOK(h, 39) ? __ldcg(b.key + h) : ~0ull;
            const int32_t u = (int32_t)(unsigned)k;
            left = k == ~0ull || (h <= u ? v < h || v > u : v < u || v > h);
            if (left && __ldcg(b.size + v) > 1) {
                // a cycle's minimum whose pointer leads to the id after it: the
                // mark of the ascending run it begins names the place of entry
                // behind it (rep[v] is v already)
                left = false;
                set_bit(r.D, v);
            } else if (!left) {
                b.rep[v] = (int32_t)(k >> 32);
                set_bit(r.D, v);
            }
        }
        wl_append(left, v, b.single, x.ctl + K_CYC_LEFT);
    }
    if (!grid_sync(r.gsync, r.err)) return;
    // The vertices on no cycle (few of a hundred, else nothing comes of it)
    // and the nodes they lead to choose again, and cycles of nodes are joined.
    const int64_t ns1 = (int64_t)__ldcg(x.ctl + K_CYC_LEFT);
    if (ns1 > n / 4) return;
    int64_t joined = 0;
    for (int64_t i = gt; i < n; i += nt) b.key[wl[i]] = ~0ull;  // the first walks' marks
    if (!grid_sync(r.gsync, r.err)) return;
    bool hashed = false;  // the walks' priorities: ids, or a hash of them
    for (int t = 0; t < kCycTries && joined < ns1; ++t) {
        if (t) {
            for (int64_t i = gt; i < ns1; i += nt) {
                const int32_t v = b.single[i];
                b.key[cyc_node(b, v)] = ~0ull;
                for (int64_t e = ld_off(r.fw_beg, v), e1 = ld_off(r.fw_beg, v + 1); e < e1; ++e) {
                    const int32_t w = ld_adj(r.fw_adj, e);
                    if (bitc(r.A, w)) b.key[cyc_node(b, w)] = ~0ull;
                }
            }
            if (!grid_sync(r.gsync, r.err)) return;
        }
        for (int64_t i = gt; i < ns1; i += nt) {
            const int32_t v = b.single[i];
            if (!bitv(r.D, v)) choose_single(r, b, v);
        }
        if (!grid_sync(r.gsync, r.err)) return;
        // Nodes of several vertices choose single ones only, so every cycle
        // has a single vertex: the one of the lowest priority walks it, a warp
        // a walk, and writes down the cycle's lowest id and its number of nodes
        // (par and skip, free by now).  A walk ends at a single vertex of lower
        // priority.  The ids are the priorities (most walks then end at once
        // where ids follow the rings; hashes from the start cost 97 graphs in
        // one call 0.4 ms of 4), for kCycSteps steps at most: up a way whose
        // ids ascend every walk would go on and on.  If any did, the next try
        // takes a hash of the ids: on a way of any length a walk goes a few
        // steps, the logarithm of it.  (Ids and kCycMax steps: a line of 200,000
        // rings and single vertices whose ids ascend 639 ms, of 20,000 301; so
        // 19 and 12.)
        // No node is joined before all walks are done: a walk told that single
        // vertex by its node's size, and where a cycle was being joined could
        // miss it, find the cycle a second time and write a second size.  (The
        // barrier costs ~3 us a try.)
        const auto prio = [hashed](int32_t a) { return hashed ? prio_of((uint32_t)a) : (uint32_t)a; };
        for (int64_t i = gt; i - lane_id() < ns1; i += nt) {
            const int32_t mine = i < ns1 ? b.single[i] : 0;
            int32_t first = mine, my_low = 0;
            int my_len = 0;
            if (i < ns1 && !bitv(r.D, mine)) first = cyc_next(b, mine);
            for (unsigned g = __ballot_sync(kFull, first != mine && !(__ldcg(b.size + first) == 1 && prio(first) < prio(mine)));
                 g; g &= g - 1) {
                const int l = __ffs(g) - 1;
                const int32_t v = __shfl_sync(kFull, mine, l);
                const uint32_t pv = prio(v);
                int32_t u = __shfl_sync(kFull, first, l), low = v, mark = u;
                int len = 1, dir = -1, renew = 2, steps = 0;
                bool found = false;
                // (a mark renewed at powers of two: met again, the walk is in a cycle without v)
                while (len < kCycMax && !(__ldcg(b.size + u) == 1 && prio(u) < pv)) {
                    if (!hashed && ++steps > kCycSteps) {
                        x.ctl[K_CYC_CUT] = 1ull;
                        break;
                    }
                    low = min(low, u);
                    const int c = cyc_run(r, b, u, dir);
                    if (c > 0) {
                        const int64_t jv = ((int64_t)v - u) * dir, jm = ((int64_t)mark - u) * dir;
                        const unsigned lower =
                            __ballot_sync(kFull, lane_id() > 0 && lane_id() <= c && prio(u + lane_id() * dir) < pv);
                        const int jl = lower ? __ffs(lower) - 1 : c + 1;
                        if (jv >= 1 && jv <= c && jv < jl) {
                            len += (int)jv;
                            found = true;
                            break;
                        }
                        if (jl <= c || (jm >= 1 && jm <= c)) break;
                        u += c * dir;
                        len += c;
                    } else {
                        const int32_t nu = cyc_next(b, u);
                        if (abs(nu - u) == 1) dir = nu - u;
                        u = nu;
                        if (u == mark) break;
                        ++len;
                        if (u == v) {
                            found = true;
                            break;
                        }
                    }
                    if (len >= renew) {
                        mark = u;
                        renew = 2 * len;
                    }
                }
                // (else: a single vertex of lower priority, another cycle, too long, or no choice)
                if (found && lane_id() == l) {
                    my_low = low;
                    my_len = len;
                }
            }
            if (i < ns1) {
                b.par[mine] = my_low;
                b.skip[mine] = my_len;
            }
        }
        if (!grid_sync(r.gsync, r.err)) return;
        // the cycles found, which share no node, are joined, a warp a cycle
        for (int64_t i = gt; i - lane_id() < ns1; i += nt) {
            const int32_t mine = i < ns1 ? b.single[i] : 0;
            const int my_len = i < ns1 ? __ldcg(b.skip + mine) : 0;
            const int32_t my_low = my_len ? __ldcg(b.par + mine) : 0;
            for (unsigned g = __ballot_sync(kFull, my_len > 0); g; g &= g - 1) {
                const int l = __ffs(g) - 1;
                const int len = __shfl_sync(kFull, my_len, l);
                const int32_t low = __shfl_sync(kFull, my_low, l);
                int32_t w = __shfl_sync(kFull, mine, l);
                int all = 0, fresh = 0, dir = -1;
                for (int k = 0; k < len;) {
                    const int c = min(cyc_run(r, b, w, dir), len - k);
                    const int32_t nw = c > 0 ? w + c * dir : cyc_next(b, w);  // (read before w's rep changes)
                    const int sz = c > 0 ? c : __ldcg(b.size + w);
                    __syncwarp();
                    if (lane_id() < max(c, 1)) {
                        const int32_t y = w + lane_id() * dir;
                        if (c > 0 || sz == 1) set_bit(r.D, y);
                        if (y != low && VOK(y, 40)) b.rep[y] = low;
                    }
                    __syncwarp();
                    all += sz;
                    fresh += c > 0 ? c : sz == 1;
                    if (c == 0 && abs(nw - w) == 1) dir = nw - w;
                    k += max(c, 1);
                    w = nw;
                }
                if (lane_id() == 0) {
                    b.size[low] = all;
                    atomicAdd(x.ctl + K_CYC_N, (unsigned long long)fresh);
                }
            }
        }
        if (!grid_sync(r.gsync, r.err)) return;
        const int64_t now = (int64_t)__ldcg(x.ctl + K_CYC_N);
        hashed = __ldcg(x.ctl + K_CYC_CUT) != 0;
        if (now == joined && !hashed) break;
        joined = now;
    }
    if (joined == 0) return;
    for (int64_t i = gt; i < n; i += nt) {  // the vertices of joined nodes follow them
        const int32_t v = wl[i], a = __ldcg(b.rep + v), c = cyc_node(b, v);
        if (c != a) b.rep[v] = c;
    }
}

// One round's work of the node peel: the vertices q_in[0, m), taken by
// threads first, first + step, ...; reserve(len) gives the place of len
// vertices in q_out.  Whole warps call it.
template <typename OffT, typename Reserve>
__device__ __forceinline__ void super_round(const Run<OffT> &r, const CycBufs &b, const int32_t *q_in, int64_t m,
                                            int32_t *q_out, int64_t first, int64_t step, Reserve reserve) {
    const int lane = lane_id();
    for (int64_t i = first; i - lane < m; i += step) {
        const bool have = i < m;
        const int32_t t = have ? __ldcg(q_in + i) : 0, rt = have ? __ldcg(b.rep + t) : 0;
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {  // out-edges lower the other's in-count, in-edges its out-count
            const OffT *beg = dir == 0 ? r.fw_beg : r.bw_beg;
            const int32_t *adj = dir == 0 ? r.fw_adj : r.bw_adj;
            int32_t *cnt = dir == 0 ? r.cnt_in : r.cnt_out;
            int64_t e = have ? ld_off(beg, t) : 0;
            const int64_t e1 = have ? ld_off(beg, t + 1) : 0;
            while (__any_sync(kFull, e < e1)) {
                int32_t w[4], rw[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) w[q] = e + q < e1 ? ld_adj(adj, e + q) : -1;
#pragma unroll
                for (int q = 0; q < 4; ++q) rw[q] = w[q] >= 0 && bitc(r.A, w[q]) ? __ldcg(b.rep + w[q]) : rt;
                unsigned kill = 0;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (rw[q] != rt && !bitv(r.D, rw[q]) && atomicSub(cnt + rw[q], 1) == 1 && set_bit(r.D, rw[q]))
                        kill |= 1u << q;
                e += 4;
                // the vertices of the nodes that died: the warp copies them
                unsigned g = __ballot_sync(kFull, kill != 0);
                for (; g; g &= g - 1) {
                    const int l = __ffs(g) - 1;
                    for (unsigned k = __shfl_sync(kFull, kill, l); k; k &= k - 1) {
                        const int q = __ffs(k) - 1;
                        const int32_t mine = q == 0 ? rw[0] : q == 1 ? rw[1] : q == 2 ? rw[2] : rw[3];
                        const int32_t node = __shfl_sync(kFull, mine, l);
                        const int len = __ldcg(b.size + node);
                        const int32_t at0 = (int32_t)__ldcg(b.key + node);
                        unsigned long long at = 0;
                        if (lane == 0) at = reserve(len);
                        at = __shfl_sync(kFull, at, 0);
                        for (int j = lane; j < len; j += 32)
                            if (VOK((long long)at + j, 36) && VOK(at0 + j, 37)) q_out[at + j] = __ldcg(b.order + at0 + j);
                    }
                }
            }
        }
    }
}

// Labels of the listed vertices whose node is dead (in D): their node is an
// SCC (a single vertex too: the peel before found none left, so the mice
// stage's counters take them).  The others go to `rest`.
template <typename OffT>
__device__ __forceinline__ void super_end(const Run<OffT> &r, const Ext<OffT> &x, const CycBufs &b, const int32_t *L,
                                          int64_t n, int32_t *rest, unsigned long long *n_rest, int64_t *sh) {
    const int64_t gt = (int64_t)blockIdx.x * kBlock + threadIdx.x;
    const int64_t nt = (int64_t)gridDim.x * kBlock;
    int64_t done = 0, sccs = 0;
    for (int64_t i = gt; i - lane_id() < n; i += nt) {
        bool keep = false;
        int32_t v = 0;
        if (i < n) {
            v = L[i];
            const int32_t rv = __ldcg(b.rep + v);
            keep = !bitv(r.D, rv);
            if (!keep) {
                r.label[v] = rv;
                r.cls[v] = CLS_MICE;
                clear_bit(r.A, v);
                ++done;
                if (rv == v) {
                    const int len = __ldcg(b.size + v);
                    if (len < kHistCap) {
                        atomicAdd((unsigned long long *)(r.hist + len), 1ull);
                    } else {
                        const unsigned long long at = atomicAdd(r.counters + C_BIG, 1ull);
                        if (at < kBigCap) r.hist[kHistCap + at] = len;
                    }
                    ++sccs;
                }
            }
        }
        wl_append(keep, v, rest, n_rest);
    }
    const int64_t td = block_sum64(done, sh), ts = block_sum64(sccs, sh);
    if (threadIdx.x == 0 && td) {
        atomicAdd(r.counters + C_MICE_V, (unsigned long long)td);
        atomicAdd(r.counters + C_MICE_SCC, (unsigned long long)ts);
    }
}

// The peel of the nodes of the vertices in large[1]; what stays goes back to
// large[0].
template <typename OffT>
__device__ __noinline__ void super_peel(const Run<OffT> &r, const Ext<OffT> &x, const CycBufs &b, int64_t n,
                                        int64_t *sh) {
    __shared__ unsigned long long s_cnt[2];
    const int64_t gt = (int64_t)blockIdx.x * kBlock + threadIdx.x;
    const int64_t nt = (int64_t)gridDim.x * kBlock;
    const int lane = lane_id();
    const int32_t *L = x.large[1];
    unsigned long long *qc = x.ctl + K_SUP_Q;  // 3 rotating counters
    for (int64_t i = gt; i < n; i += nt) {
        const int32_t v = L[i];
        r.cnt_in[v] = 0;
        r.cnt_out[v] = 0;
        if (__ldcg(b.rep + v) == v) {  // the node's place in order, and its cursor
            const unsigned long long at = atomicAdd(x.ctl + K_CYC_MEM, (unsigned long long)__ldcg(b.size + v));
            b.key[v] = at << 32 | at;
        }
    }
    for (int64_t w = gt; w < r.W; w += nt) r.D[w] = 0u;  // D: dead nodes, at their minimum
    if (!grid_sync(r.gsync, r.err)) return;
    for (int64_t i = gt; i < n; i += nt) {
        const int32_t v = L[i];
        const int32_t at = (int32_t)(atomicAdd(b.key + __ldcg(b.rep + v), 1ull << 32) >> 32);
        if (VOK(at, 38)) b.order[at] = v;
    }
    if (!grid_sync(r.gsync, r.err)) return;
    // active edges between nodes; a node's vertices are near each other in the
    // list, so a warp adds up what its lanes have for one node first
    for (int64_t i = gt; i - lane < n; i += nt) {
        const int32_t v = i < n ? L[i] : -1;
        const int32_t rv = v >= 0 ? __ldcg(b.rep + v) : -1;
        int c[2];
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
            const OffT *beg = dir == 0 ? r.fw_beg : r.bw_beg;
            const int32_t *adj = dir == 0 ? r.fw_adj : r.bw_adj;
            c[dir] = 0;
            for (int64_t e = v >= 0 ? ld_off(beg, v) : 0, e1 = v >= 0 ? ld_off(beg, v + 1) : 0; e < e1; e += 4) {
                int32_t w[4], rw[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) w[q] = e + q < e1 ? ld_adj(adj, e + q) : v;
#pragma unroll
                for (int q = 0; q < 4; ++q) rw[q] = w[q] != v && bitc(r.A, w[q]) ? __ldcg(b.rep + w[q]) : rv;
#pragma unroll
                for (int q = 0; q < 4; ++q) c[dir] += rw[q] != rv;
            }
        }
        const unsigned grp = __match_any_sync(kFull, rv);
        const int co = __reduce_add_sync(grp, c[0]), ci = __reduce_add_sync(grp, c[1]);
        if (rv >= 0 && lane == __ffs(grp) - 1) {
            if (co) atomicAdd(r.cnt_out + rv, co);
            if (ci) atomicAdd(r.cnt_in + rv, ci);
        }
    }
    if (!grid_sync(r.gsync, r.err)) return;
    for (int64_t i = gt; i - lane < n; i += nt) {
        const int32_t v = i < n ? L[i] : -1;
        const bool dead = v >= 0 && __ldcg(b.rep + v) == v && (__ldcg(r.cnt_in + v) == 0 || __ldcg(r.cnt_out + v) == 0);
        if (dead) set_bit(r.D, v);
        for (unsigned g = __ballot_sync(kFull, dead); g; g &= g - 1) {
            const int32_t node = __shfl_sync(kFull, v, __ffs(g) - 1);
            const int len = __ldcg(b.size + node);
            const int32_t at0 = (int32_t)__ldcg(b.key + node);
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(qc, (unsigned long long)len);
            at = __shfl_sync(kFull, at, 0);
            for (int j = lane; j < len; j += 32)
                if (VOK((long long)at + j, 36) && VOK(at0 + j, 37)) b.q[0][at + j] = __ldcg(b.order + at0 + j);
        }
    }
    if (!grid_sync(r.gsync, r.err)) return;
    int cur = 0, s = 0;
    for (int64_t guard = 0;; ++guard) {
        if (guard > r.V + 2) {  // every round ends a node; more rounds is a bug
            if (threadIdx.x == 0) atomicCAS(r.err, 0, kErrOverflow);
            return;
        }
        const int64_t m = (int64_t)__ldcg(qc + s);
        if (m == 0) break;
        const int s1 = s == 2 ? 0 : s + 1, s2 = s1 == 2 ? 0 : s1 + 1;
        if (gt == 0) qc[s2] = 0ull;
        if (m > kSuperTail) {
            unsigned long long *qn = qc + s1;
            super_round(r, b, b.q[cur], m, b.q[cur ^ 1], gt, nt,
                        [&](int len) { return atomicAdd(qn, (unsigned long long)len); });
        } else if (blockIdx.x == 0) {
            // few: CTA 0 alone, its rounds a block barrier apart, ending in q[cur ^ 1]
            int64_t k = m;
            int c = cur;
            if (threadIdx.x == 0) s_cnt[0] = s_cnt[1] = 0ull;
            __syncthreads();
            for (int rounds = 0; k > 0; ++rounds) {
                if (c != cur && (k > kSuperTail || rounds >= kSuperTailRounds)) break;
                unsigned long long *qn = &s_cnt[c ^ 1];
                super_round(r, b, b.q[c], k, b.q[c ^ 1], threadIdx.x, kBlock,
                            [&](int len) { return atomicAdd(qn, (unsigned long long)len); });
                __syncthreads();
                k = (int64_t)s_cnt[c ^ 1];
                if (threadIdx.x == 0) s_cnt[c] = 0ull;
                c ^= 1;
                __syncthreads();
            }
            if (threadIdx.x == 0) qc[s1] = (unsigned long long)k;
        }
        if (!grid_sync(r.gsync, r.err)) return;
        s = s1;
        cur ^= 1;
    }
    super_end(r, x, b, L, n, x.large[0], x.ctl + K_LARGE2, sh);
    if (!grid_sync(r.gsync, r.err)) return;
    if (gt == 0) {
        x.ctl[K_LARGE] = __ldcg(x.ctl + K_LARGE2);
        x.ctl[K_LARGE2] = 0ull;
    }
}

template <typename OffT>
__global__ void __launch_bounds__(kBlock, 2) k_super(Run<OffT> r, Ext<OffT> x, CycBufs b) {
    pdl_wait();  // predecessor done, its writes visible
    pdl_trigger();
    if (!__ldcg(x.ctl + K_CYC_ON)) return;
    __shared__ int64_t sh[kWarps];
    const int64_t n = (int64_t)__ldcg(x.ctl + K_LARGE);
    if (n == 0) return;
    const int64_t gt = (int64_t)blockIdx.x * kBlock + threadIdx.x;
    const int64_t nt = (int64_t)gridDim.x * kBlock;
    const int lane = lane_id();
    const int32_t *L = x.large[0];
    unsigned long long *qc = x.ctl + K_SUP_Q;  // 3 rotating counters
    // spans of the descending edges: +1 at the lower node, -1 behind the upper.
    // A vertex has one for all of its edges, to the farthest of them, which
    // covers the others: counts stay below the number of vertices (int32),
    // however many edges there are
    // Which way descends: the way that fewer edges between nodes go, of a
    // sample of the list that every CTA takes alike.  (Edges inside a node say
    // nothing: a line of 40,000 SCCs, half of them rings whose edges lead up, with
    // ids down the line: 432 ms when judged by all edges, 0.5 a line of rings.)
    __shared__ int s_down;
    if (threadIdx.x == 0) s_down = 0;
    __syncthreads();
    const int ns = (int)min(n, (int64_t)kCycSample);
    int down = 0;
    for (int k = threadIdx.x; k < ns; k += kBlock) {
        const int32_t v = L[(int64_t)k * n / ns], rv = __ldcg(b.rep + v);
        for (int64_t e = ld_off(r.fw_beg, v), e1 = min(ld_off(r.fw_beg, v + 1), e + 16); e < e1; ++e) {
            const int32_t w = ld_adj(r.fw_adj, e);
            if (w == v || !bitc(r.A, w)) continue;
            const int32_t rw = __ldcg(b.rep + w);
            down += rw < rv ? 1 : rw > rv ? -1 : 0;
        }
    }
    down = __reduce_add_sync(kFull, down);
    if (lane == 0) atomicAdd(&s_down, down);
    __syncthreads();
    const bool flip = s_down > 0;
    int32_t *diff = r.cnt_in;
    const int64_t per = ((r.W + gridDim.x - 1) / gridDim.x) * 32;  // ids per CTA, whole words
    const int64_t c0 = min(r.V + 1, (int64_t)blockIdx.x * per), c1 = min(r.V + 1, c0 + per);
    for (int64_t i = gt; i <= r.V; i += nt) diff[i] = 0;
    if (!grid_sync(r.gsync, r.err)) return;
    for (int64_t i = gt; i < n; i += nt) {
        const int32_t v = L[i], rv = __ldcg(b.rep + v);
        int32_t far = rv;
        for (int64_t e = ld_off(r.fw_beg, v), e1 = ld_off(r.fw_beg, v + 1); e < e1; e += 4) {
            int32_t w[4], rw[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) w[q] = e + q < e1 ? ld_adj(r.fw_adj, e + q) : v;
#pragma unroll
            for (int q = 0; q < 4; ++q) rw[q] = w[q] != v && bitc(r.A, w[q]) ? __ldcg(b.rep + w[q]) : rv;
#pragma unroll
            for (int q = 0; q < 4; ++q) far = flip ? max(far, rw[q]) : min(far, rw[q]);
        }
        if (far != rv && VOK(far, 41)) {
            atomicAdd(diff + min(rv, far), 1);
            atomicAdd(diff + max(rv, far) + 1, -1);
        }
    }
    if (!grid_sync(r.gsync, r.err)) return;
    {
        int64_t t = 0;
        for (int64_t i = c0 + threadIdx.x; i < c1; i += kBlock) t += diff[i];
        t = block_sum64(t, sh);
        if (threadIdx.x == 0) x.large[1][blockIdx.x] = (int32_t)t;
    }
    if (!grid_sync(r.gsync, r.err)) return;
    {   // D: ids that no span covers
        int64_t run = 0;
        for (int k = threadIdx.x; k < blockIdx.x; k += kBlock) run += x.large[1][k];
        run = block_sum64(run, sh);
        for (int64_t i0 = c0; i0 < c1; i0 += kBlock) {
            const int64_t i = i0 + threadIdx.x;
            int32_t incl = i < c1 ? diff[i] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t y = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += y;
            }
            __syncthreads();
            if (lane == 31) sh[threadIdx.x >> 5] = incl;
            __syncthreads();
            int64_t before = run, all = 0;
            for (int k = 0; k < kWarps; ++k) {
                before += k < (int)(threadIdx.x >> 5) ? sh[k] : 0;
                all += sh[k];
            }
            const unsigned free_ = __ballot_sync(kFull, i < c1 && before + incl == 0);
            if (lane == 0 && i < r.V) r.D[i >> 5] = free_;
            run += all;
        }
    }
    if (!grid_sync(r.gsync, r.err)) return;
    super_end(r, x, b, L, n, x.large[1], x.ctl + K_SUP_LEFT, sh);
    if (!grid_sync(r.gsync, r.err)) return;
    const int64_t n1 = (int64_t)__ldcg(x.ctl + K_SUP_LEFT);
    if (n1 == 0 || 4 * n1 < n) {
        for (int64_t i = gt; i < n1; i += nt) x.large[0][i] = x.large[1][i];
        if (gt == 0) x.ctl[K_LARGE] = (unsigned long long)n1;
        return;
    }
    // most of it is left: the peel, over the list in large[1]
    super_peel(r, x, b, n1, sh);
}

}  // namespace ispan
