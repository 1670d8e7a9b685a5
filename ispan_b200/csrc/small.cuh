// small.cuh -- everything up to the first peel's fixpoint for a small graph,
// in one kernel of one cluster.
//
// On a graph of at most kSmallV vertices every stage kernel costs its launch
// and every search level a grid barrier, three block reductions and the
// latency of status maps in L2 -- about 10 us a level, whatever its work.  Here
// 16 CTAs on 16 SMs, a thread-block cluster, run trim-1-first, the pivots,
// both searches side by side, the pivot SCCs and the peel; each CTA owns a
// sixteenth of the vertices and keeps a copy of the active and visited maps
// (8 KB each) in its shared memory, so a status check is a shared-memory
// access, marks go to the owner through distributed shared memory, and a
// level ends with two cluster barriers.  The edge lists are the only global
// reads (4 MB a direction on scale 16: about 2 us over 16 SMs).  Bound by the
// cluster's meetings (two a level, ~1 us each) and by the latency of list
// reads between them.  Measured, a call, by the stage kernels and so: R-MAT scale
// 10 115 and 70-74 us, scale 16 150 and 104 (the kernel itself: 32 and 66 us);
// 23 planted-cycle graphs of 100 to 5,000 (0.5-0.63 ms now) gained 0.08 ms.
// If nothing is left after the peel, the labels are written here too;
// otherwise the stage kernels go on from the peel's lists.
//
// The stages are those of k_trim1_first, k_bfs, k_giant_residual and k_trim1
// (stages.cuh, bfs.cuh), which larger graphs take: beyond 2^16 vertices the
// maps would crowd the shared memory and 16 SMs' reads bound the searches.
#pragma once
#include <cooperative_groups.h>

#include "stages.cuh"

namespace ispan {

namespace cg = cooperative_groups;

constexpr int kSmallV = 1 << 16;          // vertices, at most
constexpr int64_t kSmallE = 1 << 22;      // edges, at most
constexpr int kSmallCtas = 16;
constexpr int kSmallThreads = 1024;
constexpr int kSmallWords = kSmallV / 32;
constexpr int kSmallOwn = kSmallWords / kSmallCtas;  // words a CTA owns, at most
constexpr int kSmallLane = 16;            // entries of a list a lane reads alone
constexpr int kSmallHub = 4096;           // a longer list is pushed by the whole CTA
// Steps of a push inside a CTA before the cluster meets: more while the whole
// cluster's frontier is a few vertices (a ring of 60,000: 95 ms by 12 steps, 74
// by 128, 72 by 1,024); none once the CTA's own frontier is wide: apart, each CTA
// would then walk most of the graph by itself.  Uniform random graphs of 30,000
// to 65,000 vertices and 0.5 to 4 M edges: 0.41-1.02 ms without that limit,
// 0.12-0.23 with it (0.21-0.41 by the stage kernels).  64 to 1,024 vertices are
// alike there; on a grid of 250 x 250 256 took 2.53 ms and 1,024 1.35, on six
// planted-cycle graphs of 2,000 to 12,000 vertices 64 took 0.81 and 1,024 0.67.
constexpr int kSmallSteps = 12;
constexpr int kSmallFew = 32, kSmallFewSteps = 128;
constexpr int kSmallWide = 1024;
constexpr int kSmallQ = 4096;             // vertices a CTA goes on with; more are left to their owners

struct SmallSmem {
    uint32_t A[kSmallWords];              // active (then: left after the pivot SCCs)
    uint32_t vis[2][kSmallWords];         // reached forward, backward: the owners' state and this CTA's marks since
    uint32_t own[2][kSmallOwn];           // reached, own words (then own[0]: peeled)
    uint32_t inc[2][kSmallOwn];           // marks for own words
    uint32_t fr[2][kSmallOwn];            // own words' frontier: what this CTA is to expand
    uint32_t list[3][kSmallOwn * 64 + kSmallQ];  // frontier, both directions: short, long lists, hubs
    int n[3];
    uint32_t q[kSmallQ];                  // vertices this CTA marked and expands next, direction in bit 31
    int nq;
    int64_t cnt[2][kSmallCtas];           // counts of every CTA, by parity
    unsigned long long key[kSmallCtas];
    int64_t sum[2][kSmallThreads / 32];
};

// Two counts (below 2^31 in all) of every thread, summed over the cluster;
// ends with a cluster barrier.
__device__ __forceinline__ void small_total(cg::cluster_group &cl, SmallSmem &s, int &par, int64_t &a, int64_t &b) {
    const int64_t x = warp_sum64(a | b << 32);
    if (lane_id() == 0) s.sum[par][threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x < 32) {
        const int64_t y = warp_sum64(s.sum[par][threadIdx.x]);
        if (threadIdx.x < kSmallCtas) cl.map_shared_rank(&s, threadIdx.x)->cnt[par][cl.block_rank()] = y;
    }
    cl.sync();
    const int64_t z = warp_sum64(lane_id() < kSmallCtas ? s.cnt[par][lane_id()] : 0);
    a = z & 0xffffffff;
    b = z >> 32;
    par ^= 1;
}

// The own words `own` to every CTA's copy of the whole map: a warp per CTA.
__device__ __forceinline__ void small_spread(cg::cluster_group &cl, const uint32_t *own, uint32_t *map, int w0, int nw) {
    const int warp = threadIdx.x >> 5;
    if (warp < kSmallCtas) {
        uint32_t *to = cl.map_shared_rank(map, warp) + w0;
        for (int k = lane_id(); k < nw; k += 32) to[k] = own[k];
    }
}

// v's out-list (d = 0) or in-list to the lists by length: list[0] up to
// kSmallLane entries, list[1] up to kSmallHub, list[2].
template <typename OffT>
__device__ __forceinline__ void small_list(SmallSmem &s, const Run<OffT> &r, int d, int32_t v) {
    const OffT *beg = d ? r.bw_beg : r.fw_beg;
    const int64_t n = ld_off(beg, v + 1) - ld_off(beg, v);
    const int c = n <= kSmallLane ? 0 : n <= kSmallHub ? 1 : 2;
    const int at = atomicAdd(&s.n[c], 1);
    if (ICHK(at < kSmallOwn * 64 + kSmallQ, 42, at)) s.list[c][at] = (uint32_t)v | (uint32_t)d << 31;
}

// The vertices of the own words m[d] for the directions of `dirs` (bit 0:
// their out-lists, bit 1: their in-lists), listed anew.
template <typename OffT>
__device__ __forceinline__ void small_lists(SmallSmem &s, const Run<OffT> &r, const uint32_t (*m)[kSmallOwn], int dirs,
                                            int w0, int nw) {
    __syncthreads();
    if (threadIdx.x < 3) s.n[threadIdx.x] = 0;
    __syncthreads();
    for (int i = threadIdx.x >> 5; i < 2 * nw; i += kSmallThreads / 32) {
        const int d = i >= nw, k = d ? i - nw : i;
        if (!((dirs >> d) & 1)) continue;
        const uint32_t x = m[d][k];
        const int32_t v = (w0 + k) * 32 + lane_id();
        if ((x >> lane_id()) & 1u) small_list(s, r, d, v);
    }
    __syncthreads();
}

// f(d, v, w) for every entry w of the listed lists: a lane, a warp or the CTA
// reads a list.
template <typename OffT, typename Fn>
__device__ __forceinline__ void small_edges(SmallSmem &s, const Run<OffT> &r, Fn f) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = lane_id();
    const auto part = [&](uint32_t ent, int first, int step) {
        const int d = (int)(ent >> 31);
        const int32_t v = (int32_t)(ent & 0x7fffffffu);
        const OffT *beg = d ? r.bw_beg : r.fw_beg;
        const int32_t *adj = d ? r.bw_adj : r.fw_adj;
        for (int64_t e = ld_off(beg, v) + first, e1 = ld_off(beg, v + 1); e < e1; e += 4 * step) {
            int32_t w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) w[q] = e + q * step < e1 ? ld_adj(adj, e + q * step) : -1;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (w[q] >= 0) f(d, v, w[q]);
        }
    };
    for (int i = tid; i < s.n[0]; i += kSmallThreads) part(s.list[0][i], 0, 1);
    for (int i = warp; i < s.n[1]; i += kSmallThreads / 32) part(s.list[1][i], lane, 32);
    for (int i = 0; i < s.n[2]; ++i) part(s.list[2][i], tid, kSmallThreads);
}

template <typename OffT>
__global__ void __launch_bounds__(kSmallThreads, 1) k_small(Run<OffT> r, Ext<OffT> x) {
    pdl_wait();  // predecessor done, its writes visible
    pdl_trigger();
    extern __shared__ __align__(16) unsigned char small_raw[];
    SmallSmem &s = *reinterpret_cast<SmallSmem *>(small_raw);
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    constexpr int kW = kSmallThreads / 32;
    const int W = (int)r.W, per = (W + kSmallCtas - 1) / kSmallCtas;
    const int w0 = min(W, rank * per), nw = min(W, w0 + per) - w0;  // own words [w0, w0 + nw)
    int par = 0;
    int64_t t0, t1;
    for (int i = tid; i < W; i += kSmallThreads) s.vis[0][i] = s.vis[1][i] = 0u;
    for (int i = tid; i < kSmallOwn; i += kSmallThreads)
        s.own[0][i] = s.own[1][i] = s.inc[0][i] = s.inc[1][i] = s.fr[0][i] = s.fr[1][i] = 0u;
    if (tid == 0) s.nq = 0;
    cl.sync();  // every CTA runs: their shared memory may be written
    // trim-1-first: active map, pivot keys (see k_trim1_first)
    int64_t n_act = 0, n_tr = 0;
    unsigned long long best = 0;
    for (int k = warp; k < nw; k += kW) {
        const int w = w0 + k;
        const int64_t v = (int64_t)w * 32 + lane;
        const bool valid = v < r.V;
        const int64_t od = valid ? ld_off(r.fw_beg, v + 1) - ld_off(r.fw_beg, v) : 0;
        const int64_t id = valid ? ld_off(r.bw_beg, v + 1) - ld_off(r.bw_beg, v) : 0;
        const bool act = od > 0 && id > 0;
        const unsigned am = __ballot_sync(kFull, act), tm = __ballot_sync(kFull, valid && !act);
        if (lane == 0) {
            s.inc[0][k] = am;  // (until it is spread)
            r.T[w] = tm;
            r.D[w] = 0u;
        }
        n_act += act;
        n_tr += valid && !act;
        const unsigned long long prod = (unsigned long long)od * (unsigned long long)id;
        const unsigned long long key =
            act ? (min(prod, 0xffffffffull) << 32) | (0xffffffffull - (unsigned long long)v) : 0ull;
        if (r.nseg == 1) {
            best = max(best, key);
        } else if (am) {  // graphs are contiguous: one holds the whole word unless its ends differ
            const int g = seg_of(r.vbase, r.nseg, min(v, r.V - 1));
            const unsigned grp = __match_any_sync(kFull, g);
            unsigned long long m = grp == kFull ? warp_max_u64(key) : key;
            if (m && (grp != kFull || lane == 0)) atomicMax(r.pivot_key + g, m);
        }
    }
    if (r.nseg == 1) {
        best = warp_max_u64(best);
        if (lane == 0) s.sum[1][warp] = (int64_t)best;
    }
    __threadfence();
    __syncthreads();
    if (r.nseg == 1 && warp == 0) {
        best = warp_max_u64((unsigned long long)s.sum[1][lane]);
        if (lane < kSmallCtas) cl.map_shared_rank(&s, lane)->key[rank] = best;
    }
    small_spread(cl, s.inc[0], s.A, w0, nw);
    small_total(cl, s, par, n_act, n_tr);
    for (int k = tid; k < nw; k += kSmallThreads) s.inc[0][k] = 0u;
    __syncthreads();
    // a mark for w in direction d, if it is new here: at its owner, and this
    // CTA goes on from w (two CTAs may, until they meet: harmless)
    const auto mark = [&](int d, int32_t w) {
        const uint32_t b = 1u << (w & 31);
        const int k = w >> 5;
        if ((s.A[k] & b) && !(s.vis[d][k] & b) && !(atomicOr(&s.vis[d][k], b) & b)) {
            const int o = k / per;
            SmallSmem *to = o == rank ? &s : cl.map_shared_rank(&s, o);
            atomicOr(&to->inc[d][k - o * per], b);
            const int at = atomicAdd(&s.nq, 1);
            if (at < kSmallQ) s.q[at] = (uint32_t)w | (uint32_t)d << 31;
            else atomicOr(&to->fr[d][k - o * per], b);  // its owner does
        }
    };
    // pivots: reached both ways; one graph's is expanded by the whole cluster
    // at once, the others by their owners
    int64_t n_piv = 0;
    for (int g = tid; g < r.nseg; g += kSmallThreads) {
        unsigned long long key = 0;
        if (r.nseg == 1) {
            for (int k = 0; k < kSmallCtas; ++k) key = max(key, s.key[k]);
        } else {
            key = __ldcg(r.pivot_key + g);
        }
        if (!key) continue;
        const uint32_t v = 0xffffffffu - (uint32_t)key, b = 1u << (v & 31);
        const int w = (int)(v >> 5);
        n_piv += rank == 0;
        for (int d = 0; d < 2; ++d) {
            atomicOr(&s.vis[d][w], b);
            if (w >= w0 && w < w0 + nw) {
                atomicOr(&s.own[d][w - w0], b);
                if (r.nseg > 1) atomicOr(&s.fr[d][w - w0], b);
            }
        }
    }
    // (until every CTA has marked its pivots, a mark for one may come: its owner has it reached already)
    t1 = 0;
    small_total(cl, s, par, n_piv, t1);
    if (r.nseg == 1 && n_piv) {
        unsigned long long key = 0;
        for (int k = 0; k < kSmallCtas; ++k) key = max(key, s.key[k]);
        const int64_t v = 0xffffffffu - (uint32_t)key;
        constexpr int kStep = kSmallCtas * kSmallThreads;
        for (int d = 0; d < 2; ++d) {
            const OffT *beg = d ? r.bw_beg : r.fw_beg;
            const int32_t *adj = d ? r.bw_adj : r.fw_adj;
            for (int64_t e = ld_off(beg, v) + rank * kSmallThreads + tid, e1 = ld_off(beg, v + 1); e < e1; e += kStep)
                mark(d, ld_adj(adj, e));
        }
    }
    // both searches, level by level.  A small frontier pushes along its lists
    // and goes on from what it marked for some steps (kSmallSteps), each CTA by
    // itself, before the cluster meets; a wide one is pulled: each unreached
    // vertex looks for a reached one
    int64_t front[2] = {n_piv, n_piv};
    int levels[2] = {0, 0};
    for (int lv = 0; front[0] > 0 || front[1] > 0; ++lv) {
        if (lv > r.V + 2) {  // every level reaches a vertex; more levels is a bug
            if (tid == 0) atomicCAS(r.err, 0, kErrOverflow);
            break;
        }
        bool pull[2];
        int push = 0, nq_left = 0;
        const bool seeded = lv == 0 && r.nseg == 1;  // the pivot's lists are pushed already
        for (int d = 0; d < 2; ++d) {
            pull[d] = front[d] * 64 > r.V && front[d] >= 32;
            push |= front[d] > 0 && !pull[d] && !seeded ? 1 << d : 0;
            if (!pull[d] || front[d] == 0) continue;
            const OffT *beg = d == 0 ? r.bw_beg : r.fw_beg;
            const int32_t *adj = d == 0 ? r.bw_adj : r.fw_adj;
            const uint32_t *vis = s.vis[d];
            for (int k = warp; k < nw; k += kW) {
                const uint32_t c = s.A[w0 + k] & ~s.own[d][k];
                if (!c) continue;
                const int64_t v = (int64_t)(w0 + k) * 32 + lane;
                bool found = false;
                int64_t e = 0, e1 = 0;
                if ((c >> lane) & 1u) {
                    e = ld_off(beg, v);
                    e1 = ld_off(beg, v + 1);
                    const int64_t cap = min(e1, e + (int64_t)kSmallLane);
                    while (e < cap && !found) {
                        int32_t u[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) u[q] = e + q < cap ? ld_adj(adj, e + q) : -1;
#pragma unroll
                        for (int q = 0; q < 4; ++q) found |= u[q] >= 0 && ((vis[u[q] >> 5] >> (u[q] & 31)) & 1u);
                        e = min(e + 4, cap);
                    }
                }
                for (unsigned g = __ballot_sync(kFull, !found && e < e1); g; g &= g - 1) {
                    const int l = __ffs(g) - 1;
                    const int64_t le = __shfl_sync(kFull, e1, l);
                    bool hit = false;
                    for (int64_t b = __shfl_sync(kFull, e, l); b < le && !hit; b += 128) {
                        int32_t u[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) u[q] = b + q * 32 + lane < le ? ld_adj(adj, b + q * 32 + lane) : -1;
                        bool h = false;
#pragma unroll
                        for (int q = 0; q < 4; ++q) h |= u[q] >= 0 && ((vis[u[q] >> 5] >> (u[q] & 31)) & 1u);
                        hit = __any_sync(kFull, h);
                    }
                    if (lane == l) found = hit;
                }
                const unsigned f = __ballot_sync(kFull, found);
                if (lane == 0 && f) s.inc[d][k] = f;  // (no one pushes in this direction now)
            }
        }
        __syncthreads();
        if (seeded) {
            nq_left = min(s.nq, kSmallQ);
        } else if (push) {
            // own words' frontier and what the last steps left over (of a
            // direction that is pulled now: dropped, pulling finds what they
            // lead to), then step by step
            if (tid < 3) s.n[tid] = 0;
            __syncthreads();
            for (int i = warp; i < 2 * nw; i += kW) {
                const int d = i >= nw, k = d ? i - nw : i;
                if (!((push >> d) & 1)) continue;
                uint32_t m = lane == 0 ? atomicExch(&s.fr[d][k], 0u) : 0u;  // (others may leave more meanwhile)
                m = __shfl_sync(kFull, m, 0);
                if ((m >> lane) & 1u) small_list(s, r, d, (w0 + k) * 32 + lane);
            }
            const int steps = front[0] + front[1] <= kSmallFew ? kSmallFewSteps : kSmallSteps;
            for (int step = 0; step < steps; ++step) {
                const int nq = min(s.nq, kSmallQ);
                for (int i = tid; i < nq; i += kSmallThreads) {
                    const uint32_t ent = s.q[i];
                    const int d = (int)(ent >> 31);
                    if ((push >> d) & 1) small_list(s, r, d, (int32_t)(ent & 0x7fffffffu));
                }
                __syncthreads();
                if (tid == 0) s.nq = 0;
                if (s.n[0] + s.n[1] + s.n[2] == 0) break;
                __syncthreads();
                small_edges(s, r, [&](int d, int32_t, int32_t w) { mark(d, w); });
                __syncthreads();
                if (tid < 3) s.n[tid] = 0;
                __syncthreads();
                if (s.nq > kSmallWide) break;
            }
            __syncthreads();
            nq_left = min(s.nq, kSmallQ);
        } else if (tid == 0) {
            s.nq = 0;
        }
        cl.sync();  // all marks have arrived
        t0 = t1 = 0;
        for (int i = tid; i < 2 * nw; i += kSmallThreads) {
            const int d = i >= nw, k = d ? i - nw : i;
            if (front[d] == 0) continue;
            const uint32_t fresh = s.inc[d][k] & ~s.own[d][k];
            s.own[d][k] |= fresh;
            s.inc[d][k] = 0u;
            // found by pulling: this CTA's to expand; by pushing: who marked
            // them does, or left them in fr
            if (pull[d]) s.fr[d][k] = fresh;
            (d ? t1 : t0) += __popc(s.fr[d][k]);
        }
        for (int i = tid; i < nq_left; i += kSmallThreads) ++((s.q[i] >> 31) ? t1 : t0);
        __syncthreads();
        for (int d = 0; d < 2; ++d)
            if (front[d]) small_spread(cl, s.own[d], s.vis[d], w0, nw);
        const int64_t was[2] = {front[0], front[1]};
        small_total(cl, s, par, t0, t1);
        front[0] = t0;
        front[1] = t1;
        for (int d = 0; d < 2; ++d) {
            levels[d] += was[d] > 0;
            if (rank == 0 && tid == 0 && was[d] > 0 && lv < kTraceLevels) {  // diagnostics: mode, frontier
                long long *tr = r.trace + ((long long)d * kTraceLevels + lv) * 4;
                tr[0] = pull[d] ? 1 : 0;
                tr[1] = front[d];
                tr[2] = 0;
                tr[3] = (long long)globaltimer();
            }
        }
    }
    // the pivot SCCs leave (see k_giant_residual)
    int64_t n_fw = 0, n_giant = 0, n_res = 0;
    int gm = 0x7fffffff;
    for (int k = warp; k < nw; k += kW) {
        const int w = w0 + k;
        const uint32_t f = s.own[0][k], b = f & s.own[1][k], res = s.A[w] & ~b;
        __syncwarp();
        if (lane == 0) {
            r.F[w] = f;
            r.B[w] = b;
            n_fw += __popc(f);
            n_giant += __popc(b);
            n_res += __popc(res);
            s.own[0][k] = 0u;  // peeled from here on
            s.fr[0][k] = 0u;
            s.own[1][k] = res;
        }
        if (b && r.nseg == 1) gm = min(gm, w * 32 + __ffs(b) - 1);
        if (r.nseg > 1 && ((b >> lane) & 1u)) {
            const int64_t v = (int64_t)w * 32 + lane;
            const int g = seg_of(r.vbase, r.nseg, v);
            const unsigned grp = __match_any_sync(__activemask(), g);
            if (lane == __ffs(grp) - 1) {
                atomicMin(r.gmin + g, (int)v);
                atomicAdd(r.gsize + g, (unsigned long long)__popc(grp));
            }
        }
    }
    if (r.nseg == 1) {
        gm = warp_min(gm);
        if (lane == 0 && gm != 0x7fffffff) atomicMin(r.gmin, gm);
    }
    __threadfence();
    __syncthreads();
    small_spread(cl, s.own[1], s.A, w0, nw);
    small_total(cl, s, par, n_giant, n_res);
    if (r.nseg == 1 && rank == 0 && tid == 0) r.gsize[0] = (unsigned long long)n_giant;
    if (lane == 0 && n_fw) atomicAdd(r.counters + C_FW_SIZE, (unsigned long long)n_fw);
    // the peel (see k_trim1): counts, then rounds
    int64_t n_peel = 0;
    int rounds = 0;
    if (n_res > 0) {
        const auto active = [&](int32_t v, int32_t w) { return w != v && ((s.A[w >> 5] >> (w & 31)) & 1u); };
        for (int k = tid; k < nw; k += kSmallThreads) s.fr[1][k] = s.fr[0][k] = s.own[1][k];
        for (int i = tid; i < nw * 32; i += kSmallThreads)
            if ((s.own[1][i >> 5] >> (i & 31)) & 1u) r.cnt_out[w0 * 32 + i] = r.cnt_in[w0 * 32 + i] = 0;
        small_lists(s, r, s.fr, 3, w0, nw);
        small_edges(s, r, [&](int d, int32_t v, int32_t w) {
            if (active(v, w)) atomicAdd((d ? r.cnt_in : r.cnt_out) + v, 1);
        });
        __syncthreads();
        t0 = t1 = 0;
        for (int k = warp; k < nw; k += kW) {
            const int32_t v = (w0 + k) * 32 + lane;
            const bool dead = ((s.own[1][k] >> lane) & 1u) && (__ldcg(r.cnt_out + v) == 0 || __ldcg(r.cnt_in + v) == 0);
            const unsigned dm = __ballot_sync(kFull, dead);
            if (lane == 0) s.own[0][k] = s.fr[0][k] = s.fr[1][k] = dm;
            t0 += dead;
        }
        __threadfence();
        small_total(cl, s, par, t0, t1);
        n_peel = t0;
        for (int64_t n = t0; n > 0; ++rounds) {
            if (rounds > r.V) {  // every round peels a vertex
                if (tid == 0) atomicCAS(r.err, 0, kErrOverflow);
                break;
            }
            // out-edges lower the other's in-count, in-edges its out-count
            small_lists(s, r, s.fr, 3, w0, nw);
            small_edges(s, r, [&](int d, int32_t v, int32_t w) {
                if (active(v, w) && atomicSub((d ? r.cnt_out : r.cnt_in) + w, 1) == 1) {
                    const int o = (w >> 5) / per;
                    atomicOr(cl.map_shared_rank(&s.inc[0][(w >> 5) - o * per], o), 1u << (w & 31));
                }
            });
            cl.sync();  // all marks have arrived
            t0 = t1 = 0;
            for (int k = tid; k < nw; k += kSmallThreads) {
                const uint32_t fresh = s.inc[0][k] & ~s.own[0][k];
                s.own[0][k] |= fresh;
                s.fr[0][k] = s.fr[1][k] = fresh;
                s.inc[0][k] = 0u;
                t0 += __popc(fresh);
            }
            small_total(cl, s, par, t0, t1);
            n = t0;
            n_peel += n;
        }
    }
    const int64_t left = n_res - n_peel;
    for (int k = warp; k < nw; k += kW) {
        const int w = w0 + k;
        const int64_t v = (int64_t)w * 32 + lane;
        const uint32_t dead = s.own[0][k], stay = s.own[1][k] & ~dead;
        if (lane == 0) r.A[w] = stay;
        if ((dead >> lane) & 1u) {
            r.label[v] = (int32_t)v;
            r.cls[v] = CLS_TRIM1;
        }
        if (left > 0) {  // the lists of the next stages (see k_trim1)
            const bool st = (stay >> lane) & 1u;
            wl_append(st, (int32_t)v, r.wl[1], x.ctl + K_WL1);
            wl_append(st && (__ldcg(r.cnt_out + v) <= 2 || __ldcg(r.cnt_in + v) <= 2), (int32_t)v, x.cand, x.ctl + K_CAND);
        } else {  // the labels of k_finalize
            const uint32_t b = r.B[w], tm = r.T[w];
            if ((b >> lane) & 1u) r.label[v] = __ldcg(r.gmin + seg_of(r.vbase, r.nseg, v));
            else if ((tm >> lane) & 1u) r.label[v] = (int32_t)v;
        }
    }
    if (rank == 0) {
        if (tid == 0) {
            r.counters[C_ACTIVE0] = (unsigned long long)n_act;
            r.counters[C_GIANT] = (unsigned long long)n_giant;
            r.counters[C_TRIM1] = (unsigned long long)(n_tr + n_peel);
            r.counters[C_FW_LEVELS] = (unsigned long long)levels[0];
            r.counters[C_BW_LEVELS] = (unsigned long long)levels[1];
            r.counters[C_TRIM_ROUNDS] = (unsigned long long)(rounds + 1);
            if (left == 0) atomicAdd((unsigned long long *)(r.hist + 1), (unsigned long long)(n_tr + n_peel));
            if (x.gate_left) cudaGraphSetConditional(x.gate_left, left > 0 ? 1u : 0u);
            x.ctl[K_SMALL_DONE] = left == 0 ? 1ull : 0ull;
        }
        if (left == 0) {
            for (int g = tid; g < r.nseg; g += kSmallThreads) {
                const unsigned long long sz = __ldcg(r.gsize + g);
                if (!sz) continue;
                atomicAdd(r.counters + C_GIANTS, 1ull);
                if (sz < (unsigned long long)kHistCap) {
                    atomicAdd((unsigned long long *)(r.hist + sz), 1ull);
                } else {
                    const unsigned long long k = atomicAdd(r.counters + C_BIG, 1ull);
                    if (k < kBigCap) r.hist[kHistCap + k] = (int64_t)sz;
                }
            }
        }
    }
    cl.sync();  // no CTA leaves while another may still write to it
}

}  // namespace ispan
