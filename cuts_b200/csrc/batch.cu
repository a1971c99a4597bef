// batch.cu -- many queries against one resident graph in one persistent
// launch, captured in a CUDA graph.
//
// Work is a flat space of tasks, query-major: a task is (query q, root u,
// range r of u's level-1 candidate list), or, for the roots whose list is one
// range, 8 or 32 roots -- finding a task's root is two binary searches of ~20
// dependent loads, which with one task per root was most of a small query's
// time (a triangle on 200,000 vertices alone 0.92 ms, 0.45 ms this way).  Roots are the data vertices in
// out-degree order, so every query's root level is a prefix of one sorted
// array, and a per-graph prefix sum of ceil(len / grain) turns a task index
// into (u, r) with two binary searches -- nothing per query is materialised.
// Warps take tasks from one global counter (work stealing across all SMs)
// and run the query's levels depth-first from the task's level-1 range,
// with a 32-candidate frontier per level in shared memory: the trie is
// walked, never stored, so a batch needs no trie arena.  A level step takes 32
// candidates of the shortest joined list, one per lane, tests them in the other
// lists' tables (by search without tables) and compacts them with a ballot; the
// last level is counted for a whole frontier at once (count_frontier).  Counts
// accumulate per warp and are added to the query's counter when the warp moves
// on.  A device-clock budget stops the launch cleanly: tasks not finished mark
// their query incomplete.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "batch.hpp"
#include "device_util.cuh"

namespace cuts {

#define BCK(call)                                                                      \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess)                                                         \
            return set_error(CUTS_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

namespace {

constexpr int kBW = 8;  // warps per block

struct BWarp {  // per-warp depth-first state, shared memory
    uint32_t m[kBatchMaxK];
    uint32_t moff[kBatchMaxK], mdeg[kBatchMaxK], x[kBatchMaxK], xend[kBatchMaxK];
    uint32_t nb[kBatchMaxK], bi[kBatchMaxK], tmin[kBatchMaxK], nj[kBatchMaxK];
    uint32_t joff[kBatchMaxK][kBatchMaxJ], jdeg[kBatchMaxK][kBatchMaxJ];
    uint32_t buf[kBatchMaxK][32];
    // the counted frontier's records, by rank of the lane (count_frontier)
    uint4 rec[32];
    uint2 rec2[32];
    uint32_t starts[32];
};

struct Ctx {
    DevView g;
    const BQuery *Q;
    BWarp *S;
    int lane;
};

// Joined lists of level d for the current prefix; the shortest feeds the
// candidates, restricted to the symmetry window.  Warp-uniform.
__device__ void enter_level(const Ctx &c, uint32_t d) {
    const BLevel &L = c.Q->lv[d];
    const uint32_t nj = L.nj;
    uint32_t my_deg = kFullMask, my_off = 0;
    if (uint32_t(c.lane) < nj) {
        const uint32_t u = c.S->m[L.jpos[c.lane]];
        const uint2 inf = L.jdir[c.lane] ? c.g.in_info[u] : c.g.out_info[u];
        my_off = inf.x;
        my_deg = inf.y;
        c.S->joff[d][c.lane] = my_off;
        c.S->jdeg[d][c.lane] = my_deg;
    }
    uint32_t bd = my_deg, bl = uint32_t(c.lane);
    #pragma unroll
    for (int s = 16; s; s >>= 1) {
        const uint32_t od = __shfl_xor_sync(kFullMask, bd, s), ol = __shfl_xor_sync(kFullMask, bl, s);
        if (od < bd || (od == bd && ol < bl)) { bd = od; bl = ol; }
    }
    const uint32_t moff = __shfl_sync(kFullMask, my_off, int(bl));
    uint32_t lo = 0, hi = kFullMask;
    for (uint32_t msk = L.gt_mask; msk; msk &= msk - 1) lo = max(lo, c.S->m[__ffs(msk) - 1] + 1);
    for (uint32_t msk = L.lt_mask; msk; msk &= msk - 1) hi = min(hi, c.S->m[__ffs(msk) - 1]);
    const uint32_t *lst = c.g.adj + moff;
    const uint32_t s0 = (lo && nj) ? lbound(lst, bd, lo) : 0;
    const uint32_t e0 = nj ? (hi != kFullMask ? lbound(lst, bd, hi) : bd) : 0;
    __syncwarp();
    if (c.lane == 0) {
        c.S->moff[d] = moff;
        c.S->mdeg[d] = nj ? bd : 0;
        c.S->tmin[d] = bl;
        c.S->nj[d] = nj;
        c.S->x[d] = s0;
        c.S->xend[d] = max(s0, e0);
        c.S->nb[d] = 0;
        c.S->bi[d] = 0;
    }
    __syncwarp();
}

// Lane test of candidate list element idx at level d.
__device__ __forceinline__ bool test_candidate(const Ctx &c, uint32_t d, uint32_t idx, uint32_t &cand) {
    const BLevel &L = c.Q->lv[d];
    bool ok = idx < c.S->xend[d];
    const uint32_t v = ok ? __ldg(c.g.adj + c.S->moff[d] + idx) : 0;
    if (ok)
        for (uint32_t j = 0; j < d; ++j)
            if (v == c.S->m[j]) { ok = false; break; }
    ok = ok && v >= L.sig_lo;
    if (ok && L.check_sig) {
        const uint2 o = c.g.out_info[v], i = c.g.in_info[v];
        ok = i.y >= L.qin && o.y >= L.qout;
    }
    if (ok) {
        const uint32_t nj = c.S->nj[d], tm = c.S->tmin[d];
        for (uint32_t t = 0; t < nj; ++t) {
            if (t == tm) continue;
            if (!in_list(c.g, c.S->joff[d][t], c.S->jdeg[d][t], v)) { ok = false; break; }
        }
    }
    cand = v;
    return ok;
}

// Candidates of level d in [x, xend), counted (the last level).
__device__ unsigned long long count_level(const Ctx &c, uint32_t d) {
    const BLevel &L = c.Q->lv[d];
    const uint32_t s0 = c.S->x[d], e0 = c.S->xend[d];
    if (s0 >= e0) return 0;
    if (L.closed_form && c.S->nj[d] == 1) {
        // one list, no signature: the window minus the matched vertices in it
        const uint32_t *lst = c.g.adj + c.S->moff[d];
        const uint32_t mdeg = c.S->mdeg[d];
        bool hit = false;
        if (uint32_t(c.lane) < d) {
            const uint32_t mj = c.S->m[c.lane];
            if ((L.guar_mask >> c.lane) & 1u) {
                // the query's own arc puts m_j in the list: only the window decides
                const uint32_t lo = s0 ? __ldg(lst + s0 - 1) : 0;  // window by position
                hit = (s0 == 0 || mj > lo) && (e0 >= mdeg || mj < __ldg(lst + e0));
            } else {
                const uint32_t p = lbound(lst, mdeg, mj);
                hit = p >= s0 && p < e0 && p < mdeg && __ldg(lst + p) == mj;
            }
        }
        return (e0 - s0) - __popc(__ballot_sync(kFullMask, hit));
    }
    unsigned long long n = 0;
    for (uint32_t x0 = s0; x0 < e0; x0 += 32) {
        uint32_t v;
        const bool ok = test_candidate(c, d, x0 + c.lane, v);
        n += __popc(__ballot_sync(kFullMask, ok));
    }
    return n;
}

// Level d = k-2 counted together with level k-1 (the plan folded them): each
// candidate c of level d adds the last level's closed form, the window of the
// last level's list minus the matched vertices in it, c included.
__device__ unsigned long long count_level_fold(const Ctx &c, uint32_t d) {
    const BLevel &F = c.Q->lv[d + 1];
    const uint32_t s0 = c.S->x[d], e0 = c.S->xend[d];
    if (s0 >= e0) return 0;
    const uint32_t u = c.S->m[F.jpos[0]];
    const uint2 inf = F.jdir[0] ? c.g.in_info[u] : c.g.out_info[u];
    uint32_t lo = 0, hi = kFullMask;
    for (uint32_t msk = F.gt_mask; msk; msk &= msk - 1) lo = max(lo, c.S->m[__ffs(msk) - 1] + 1);
    for (uint32_t msk = F.lt_mask; msk; msk &= msk - 1) hi = min(hi, c.S->m[__ffs(msk) - 1]);
    const uint32_t *fl = c.g.adj + inf.x;
    const uint32_t ws = lo ? lbound(fl, inf.y, lo) : 0;
    const uint32_t we = hi != kFullMask ? lbound(fl, inf.y, hi) : inf.y;
    bool hit = false;
    if (uint32_t(c.lane) < d) {
        const uint32_t mj = c.S->m[c.lane];
        hit = mj >= lo && mj < hi && (((F.guar_mask >> c.lane) & 1u) || contains(fl, inf.y, mj));
    }
    const uint32_t base = (we > ws ? we - ws : 0) - __popc(__ballot_sync(kFullMask, hit));
    const bool guar_c = (F.guar_mask >> d) & 1u;
    unsigned long long n = 0;
    for (uint32_t x0 = s0; x0 < e0; x0 += 32) {
        uint32_t v;
        const bool ok = test_candidate(c, d, x0 + c.lane, v);
        uint32_t add = 0;
        if (ok) {
            const bool h2 = v >= lo && v < hi && (guar_c || contains(fl, inf.y, v));
            add = base - (h2 ? 1u : 0u);
        }
        #pragma unroll
        for (int o = 16; o; o >>= 1) add += __shfl_xor_sync(kFullMask, add, o);
        n += add;
    }
    return n;
}

// Level e = d + 1 counted for the whole frontier of level d (buf[d], nb[d]
// vertices, at most 32), one vertex per lane: each lane finds its own shortest
// list and window -- lists of positions below d are the warp's, the list of
// position d the lane's -- and the lanes' candidate windows are one sequence
// walked 64 candidates a step, as in k_level_flat (engine.cu).  Counting one
// frontier vertex after another left most lanes idle on short lists: 64 mixed
// queries of 3 and 4 vertices on 200,000 vertices / 1.6M edges took 480 ms,
// 207 ms this way (60 ms since, with twins and edge counts).  With a fold at e,
// each candidate adds the closed form of level e + 1.  Returns the lane's part of
// the count.
__device__ unsigned long long count_frontier(const Ctx &c, uint32_t d) {
    const uint32_t e = d + 1, nj = c.Q->lv[e].nj;
    const BLevel &L = c.Q->lv[e];
    const BLevel &F = c.Q->lv[e + 1 < c.Q->k ? e + 1 : e];
    const bool fold = L.fold && e + 2 == c.Q->k;
    // twins: level e + 1 has a vertex's other candidates of level e
    const uint32_t twin = e + 2 == c.Q->k ? L.twin : 0u;
    const DevView &g = c.g;
    BWarp *const S = c.S;
    const int lane = c.lane;
    if (uint32_t(lane) < nj && L.jpos[lane] != d) {
        const uint32_t u = S->m[L.jpos[lane]];
        const uint2 inf = L.jdir[lane] ? g.in_info[u] : g.out_info[u];
        S->joff[e][lane] = inf.x;
        S->jdeg[e][lane] = inf.y;
    }
    __syncwarp();
    const bool have = uint32_t(lane) < S->nb[d];
    const uint32_t v = have ? S->buf[d][lane] : 0u;
    auto m = [&](uint32_t j) { return j == d ? v : S->m[j]; };
    uint32_t moff = 0, mdeg = 0, tmin = 0, s0 = 0, e0 = 0;
    uint2 own[2] = {make_uint2(0, 0), make_uint2(0, 0)};  // v's out- and in-list
    uint32_t f_off = 0, f_deg = 0, f_lo = 0, f_hi = kFullMask, fbase = 0;
    unsigned long long n = 0;
    if (have) {
        mdeg = kFullMask;
        for (uint32_t t = 0; t < nj; ++t) {
            uint2 inf;
            if (L.jpos[t] == d) {
                inf = L.jdir[t] ? g.in_info[v] : g.out_info[v];
                own[L.jdir[t] ? 1 : 0] = inf;
            } else {
                inf = make_uint2(S->joff[e][t], S->jdeg[e][t]);
            }
            if (inf.y < mdeg) { mdeg = inf.y; moff = inf.x; tmin = t; }
        }
        if (nj == 0) mdeg = 0;
        uint32_t lo = 0, hi = kFullMask;
        for (uint32_t k = L.gt_mask; k; k &= k - 1) lo = max(lo, m(__ffs(k) - 1) + 1);
        for (uint32_t k = L.lt_mask; k; k &= k - 1) hi = min(hi, m(__ffs(k) - 1));
        const uint32_t *lst = g.adj + moff;
        const uint32_t mu = nj ? m(L.jpos[tmin]) : 0u;
        const bool mdir = nj && L.jdir[tmin];
        s0 = (lo && nj) ? lbound_own(g, mdir, mu, lst, mdeg, lo, true) : 0;
        e0 = hi != kFullMask ? lbound_own(g, mdir, mu, lst, mdeg, hi, true) : mdeg;
        if (e0 < s0) e0 = s0;
        if (L.closed_form && nj == 1) {
            // one list, no signature: the window minus the matched vertices in it
            uint32_t sub = 0;
            for (uint32_t j = 0; j <= d; ++j) {
                const uint32_t mj = m(j);
                if (mj >= lo && mj < hi && (((L.guar_mask >> j) & 1u) || in_list(g, moff, mdeg, mj))) ++sub;
            }
            n = (e0 - s0) - sub;
        } else if (fold) {
            const uint32_t u = m(F.jpos[0]);
            const uint2 inf = F.jdir[0] ? g.in_info[u] : g.out_info[u];
            f_off = inf.x;
            f_deg = inf.y;
            for (uint32_t k = F.gt_mask; k; k &= k - 1) f_lo = max(f_lo, m(__ffs(k) - 1) + 1);
            for (uint32_t k = F.lt_mask; k; k &= k - 1) f_hi = min(f_hi, m(__ffs(k) - 1));
            const uint32_t *fl = g.adj + f_off;
            const uint32_t ws = f_lo ? lbound(fl, f_deg, f_lo) : 0, we = f_hi != kFullMask ? lbound(fl, f_deg, f_hi) : f_deg;
            uint32_t sub = 0;
            for (uint32_t j = 0; j <= d; ++j) {
                const uint32_t mj = m(j);
                if (mj >= f_lo && mj < f_hi && (((F.guar_mask >> j) & 1u) || in_list(g, f_off, f_deg, mj))) ++sub;
            }
            fbase = (we > ws ? we - ws : 0) - sub;
        }
    }
    if (L.closed_form && nj == 1) return n;
    const bool fold_guar = (F.guar_mask >> e) & 1u;
    const uint32_t len = e0 - s0;
    uint32_t incl = len;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(kFullMask, incl, 31);
    if (!total) return 0;
    const uint32_t lt = (1u << lane) - 1, le = lt | (1u << lane);
    const unsigned live = __ballot_sync(kFullMask, len != 0);
    if (len) {
        const uint32_t r = __popc(live & lt), excl = incl - len;
        S->rec[r] = make_uint4(moff + s0 - excl, uint32_t(lane) | (tmin << 8), own[0].x, own[0].y);
        S->rec2[r] = own[1];
        S->starts[r] = excl;
    }
    __syncwarp();
    const uint32_t my_start = uint32_t(lane) < uint32_t(__popc(live)) ? S->starts[lane] : kFullMask;
    if (twin) {
        __syncwarp();
        S->starts[lane] = 0;  // from here on: candidates of the lane's vertex
        __syncwarp();
    }
    uint32_t started = 0;
    for (uint32_t f0 = 0; f0 < total; f0 += 64) {
        uint4 rc[2];
        uint32_t cv[2], rk[2];
        #pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t rel = my_start - (f0 + 32 * h);
            const uint32_t bits = __reduce_or_sync(kFullMask, rel < 32u ? 1u << rel : 0u);
            rk[h] = started + __popc(bits & le) - 1;
            started += __popc(bits);
            rc[h] = S->rec[rk[h]];
            cv[h] = __ldg(g.adj + (rc[h].x + min(f0 + 32 * h + lane, total - 1)));
        }
        #pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t w = cv[h], owner = rc[h].y & 255u, o_tmin = rc[h].y >> 8;
            bool ok = f0 + 32 * h + lane < total && w >= L.sig_lo;
            if (ok)
                for (uint32_t t = 0; t < nj; ++t) {
                    if (t == o_tmin) continue;
                    uint32_t off, deg;
                    if (L.jpos[t] != d) {
                        off = S->joff[e][t];
                        deg = S->jdeg[e][t];
                    } else if (L.jdir[t]) {
                        off = S->rec2[rk[h]].x;
                        deg = S->rec2[rk[h]].y;
                    } else {
                        off = rc[h].z;
                        deg = rc[h].w;
                    }
                    if (!in_list(g, off, deg, w)) { ok = false; break; }
                }
            if (ok)
                for (uint32_t j = 0; j < d; ++j)
                    if (w == S->m[j]) { ok = false; break; }
            if (ok) ok = w != S->buf[d][owner];
            if (ok && L.check_sig) {
                const uint2 o = g.out_info[w], i = g.in_info[w];
                ok = i.y >= L.qin && o.y >= L.qout;
            }
            if (twin) {
                // lanes of one vertex are neighbours: the first of them adds
                const unsigned mk = __ballot_sync(kFullMask, ok);
                const uint32_t up = __shfl_up_sync(kFullMask, owner, 1);
                const bool head = lane == 0 || up != owner;
                const unsigned next = __ballot_sync(kFullMask, head) & ~le;
                const unsigned seg = (next ? (1u << (__ffs(next) - 1)) - 1u : kFullMask) & ~lt;
                if (head) S->starts[owner] += __popc(mk & seg);
                __syncwarp();
            } else if (fold) {
                const uint32_t o_base = __shfl_sync(kFullMask, fbase, int(owner));
                const uint32_t o_off = __shfl_sync(kFullMask, f_off, int(owner));
                const uint32_t o_deg = __shfl_sync(kFullMask, f_deg, int(owner));
                const uint32_t o_lo = __shfl_sync(kFullMask, f_lo, int(owner));
                const uint32_t o_hi = __shfl_sync(kFullMask, f_hi, int(owner));
                if (ok) {
                    const bool hit = w >= o_lo && w < o_hi && (fold_guar || in_list(g, o_off, o_deg, w));
                    n += o_base - (hit ? 1u : 0u);
                }
            } else {
                n += ok;
            }
        }
    }
    __syncwarp();
    if (twin && len) {
        const unsigned long long q = S->starts[lane], pr = q ? q * (q - 1) : 0;
        n = twin == 2 ? pr / 2 : pr;
    }
    __syncwarp();
    return n;
}

// Next up-to-32 candidates of level d into its frontier buffer.
__device__ void refill(const Ctx &c, uint32_t d) {
    uint32_t v;
    const bool ok = test_candidate(c, d, c.S->x[d] + c.lane, v);
    const unsigned m = __ballot_sync(kFullMask, ok);
    if (ok) c.S->buf[d][__popc(m & ((1u << c.lane) - 1))] = v;
    __syncwarp();
    if (c.lane == 0) {
        c.S->x[d] += 32;
        c.S->nb[d] = __popc(m);
        c.S->bi[d] = 0;
    }
    __syncwarp();
}

// Adds the lanes' parts of one query's count to its counter.
__device__ __forceinline__ void add_count(unsigned long long *__restrict__ to, unsigned long long part, int lane) {
    #pragma unroll
    for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(kFullMask, part, o);
    if (lane == 0 && part) atomicAdd(to, part);
}

// Level d's whole frontier is counted at once (its children are the last
// level stored, or the one folded with it).
__device__ __forceinline__ bool counts_next(const BQuery &Q, uint32_t d) {
    return d + 2 == Q.k || (d + 3 == Q.k && (Q.lv[d + 1].fold || Q.lv[d + 1].twin));
}

// Single-range roots of one task, at most: 32 where they are counted at once, 8
// where the warp goes through them one after another and a root is a frontier or
// two, one where subtrees are deeper: finding the root is then little of the
// work, and 8 subtrees in a row are the launch's tail (a 5-vertex query on 5,000
// vertices / 15,000 edges alone 0.8 ms with one, 2.3 with 8).  Fewer in a launch
// of so few roots that warps would get less than a task each, or 4 tasks of
// 4-vertex queries (one on 1,500 vertices of a directed graph alone 3.7 ms in
// bundles of 8, 1.3 with one root per task before the bundles, 0.55 now).
// The warps are a number, not a device's: shards on several GPUs have to cut
// the same tasks.
constexpr unsigned long long kLaunchWarps = 148 * 4 * kBW;
inline uint32_t roots_per_task(const BQuery &Q, unsigned long long roots) {
    const unsigned long long most = Q.k == 2 || (Q.k == 3 && Q.lv[1].fold) ? 32 : Q.k <= 4 ? 8 : 1;
    return uint32_t(std::max<unsigned long long>(1, std::min(most, roots / ((Q.k <= 3 ? 1 : 4) * kLaunchWarps))));
}

// One vertex of level d's frontier becomes matched; its children are next.
__device__ __forceinline__ void descend(const Ctx &c, uint32_t d) {
    const uint32_t v = c.S->buf[d][c.S->bi[d]];
    __syncwarp();
    if (c.lane == 0) {
        c.S->bi[d]++;
        c.S->m[d] = v;
    }
    __syncwarp();
    enter_level(c, d + 1);
}

__global__ void __launch_bounds__(kBW * 32)
k_batch(DevView g, const BQuery *__restrict__ qs, uint32_t nq,
        const unsigned long long *__restrict__ qbase, const uint32_t *__restrict__ vsorted,
        const unsigned long long *__restrict__ pref0, const unsigned long long *__restrict__ pref1,
        const unsigned long long *__restrict__ pref2, uint32_t grain, uint32_t tgrab,
        unsigned long long *__restrict__ task_ctr, uint32_t *__restrict__ stop,
        unsigned long long *__restrict__ counts, uint32_t *__restrict__ aborted,
        unsigned long long budget_ns, unsigned long long *__restrict__ qtime,
        unsigned long long qlimit, uint32_t shard, uint32_t nshards, uint32_t rshard, uint32_t nrshards) {
    __shared__ BWarp ws[kBW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Ctx c{g, nullptr, &ws[warp], lane};
    const unsigned long long total = qbase[nq];
    // this shard's tasks are t = c * nshards + shard for counter values c
    const unsigned long long ctotal = total > shard ? (total - shard + nshards - 1) / nshards : 0;
    const unsigned long long deadline = budget_ns ? global_ns() + budget_ns : ~0ull;
    uint32_t cur = kFullMask;
    unsigned long long qcount = 0;
    volatile uint32_t *vstop = stop;

    while (true) {
        unsigned long long c0 = 0;
        if (lane == 0) c0 = *vstop ? ctotal : atomicAdd(task_ctr, (unsigned long long)tgrab);
        c0 = __shfl_sync(kFullMask, c0, 0);
        if (c0 >= ctotal) break;
        const unsigned long long c1 = min(c0 + tgrab, ctotal);
        for (unsigned long long cc = c0; cc < c1; ++cc) {
            const unsigned long long t = cc * nshards + shard;
            if (cur == kFullMask || t < qbase[cur] || t >= qbase[cur + 1]) {
                if (cur != kFullMask) add_count(&counts[cur], qcount, lane);
                qcount = 0;
                uint32_t lo = 0, hi = nq - 1;  // last q with qbase[q] <= t
                while (lo < hi) {
                    const uint32_t mid = (lo + hi + 1) >> 1;
                    if (qbase[mid] <= t) lo = mid; else hi = mid - 1;
                }
                cur = lo;
                c.Q = qs + cur;
            }
            if (*vstop || global_ns() > deadline) {
                if (lane == 0) { atomicOr(stop, 1u); aborted[cur] = 1; }
                continue;
            }
            // per-query limit: a query past its share of warp time is dropped,
            // and the work counter skips the rest of its tasks
            if (qlimit) {
                uint32_t skip = 0;
                if (lane == 0) {
                    skip = reinterpret_cast<volatile uint32_t *>(aborted)[cur] ||
                           reinterpret_cast<volatile unsigned long long *>(qtime)[cur] > qlimit;
                    if (skip) {
                        aborted[cur] = 1;
                        const unsigned long long e = qbase[cur + 1];
                        atomicMax(task_ctr, e > shard ? (e - shard + nshards - 1) / nshards : 0ull);
                    }
                }
                if (__shfl_sync(kFullMask, skip, 0)) continue;
            }
            const unsigned long long task_start = qlimit ? global_ns() : 0;
            const BQuery &Q = *c.Q;
            const unsigned long long local = t - qbase[cur];
            const unsigned long long *pref = Q.type == 0 ? pref0 : (Q.type == 1 ? pref1 : pref2);
            bool abandoned = false, dropped = false;
            // the subtree of the root m[0] from the level-1 candidates
            // [x[1], xend[1]) on: depth-first over levels 1..k-2, counting k-1
            auto subtree = [&]() {
                if (Q.k == 2 || (Q.k == 3 && Q.lv[1].fold)) {
                    const unsigned long long r1 = Q.k == 2 ? count_level(c, 1) : count_level_fold(c, 1);
                    if (lane == 0) qcount += r1;  // the warp's
                    return;
                }
                uint32_t d = 1;
                while (d >= 1) {
                    if (c.S->bi[d] < c.S->nb[d]) {
                        if (counts_next(Q, d)) {
                            qcount += count_frontier(c, d);
                            __syncwarp();
                            if (lane == 0) c.S->bi[d] = c.S->nb[d];
                            __syncwarp();
                        } else {
                            descend(c, d);
                            ++d;
                        }
                    } else if (c.S->x[d] < c.S->xend[d]) {
                        const unsigned long long now = global_ns();
                        if (*vstop || now > deadline) { abandoned = true; return; }
                        if (qlimit && reinterpret_cast<volatile unsigned long long *>(qtime)[cur] +
                                              (now - task_start) > qlimit) {
                            dropped = true;
                            return;
                        }
                        refill(c, d);
                    } else {
                        --d;
                    }
                }
            };
            const unsigned long long heavy = pref[Q.heavy_roots];
            if (local >= heavy) {
                // roots of one range each: looked at together, and counted
                // together where level 1 is the last one walked
                const uint32_t per = Q.per;
                const uint32_t ri = Q.heavy_roots + uint32_t(local - heavy) * per + lane;
                uint32_t u = 0;
                bool pass = uint32_t(lane) < per && ri < Q.root_cnt;
                if (pass) {
                    u = vsorted[ri];
                    const uint2 uo = g.out_info[u], ui = g.in_info[u];
                    pass = ui.y >= Q.lv[0].qin && uo.y >= Q.lv[0].qout && (nrshards == 1 || u % nrshards == rshard);
                }
                const unsigned m = __ballot_sync(kFullMask, pass);
                __syncwarp();
                if (pass) c.S->buf[0][__popc(m & ((1u << lane) - 1))] = u;
                if (lane == 0) c.S->nb[0] = __popc(m);
                __syncwarp();
                if (m && counts_next(Q, 0)) {
                    qcount += count_frontier(c, 0);
                } else {
                    const uint32_t nr = __popc(m);
                    for (uint32_t i = 0; i < nr && !abandoned && !dropped; ++i) {
                        __syncwarp();
                        if (lane == 0) c.S->m[0] = c.S->buf[0][i];
                        __syncwarp();
                        enter_level(c, 1);
                        subtree();
                    }
                }
                __syncwarp();
            } else {
                uint32_t lo = 0, hi = Q.heavy_roots - 1;  // root: last j with pref[j] <= local
                while (lo < hi) {
                    const uint32_t mid = (lo + hi + 1) >> 1;
                    if (pref[mid] <= local) lo = mid; else hi = mid - 1;
                }
                const uint32_t u = vsorted[lo];
                const uint32_t r = uint32_t(local - pref[lo]);
                const uint2 uo = g.out_info[u], ui = g.in_info[u];
                if (ui.y < Q.lv[0].qin || uo.y < Q.lv[0].qout) continue;  // level-0 signature
                if (nrshards != 1 && u % nrshards != rshard) continue;
                if (lane == 0) c.S->m[0] = u;
                __syncwarp();
                // level 1: joins all on position 0; the task fixes the list and range
                enter_level(c, 1);
                // the task space was cut on the type's list (out, in or the
                // shorter): make that list the candidate source
                const bool use_in = Q.type == 1 || (Q.type == 2 && ui.y < uo.y);
                const uint2 L1 = use_in ? ui : uo;
                uint32_t tm = 0;
                for (uint32_t t2 = 0; t2 < Q.lv[1].nj; ++t2)
                    if ((Q.lv[1].jdir[t2] != 0) == use_in) { tm = t2; break; }
                const uint32_t *lst = g.adj + L1.x;
                uint32_t lo1 = 0, hi1 = kFullMask;
                if (Q.lv[1].gt_mask) lo1 = u + 1;
                if (Q.lv[1].lt_mask) hi1 = u;
                const uint32_t s0 = lo1 ? lbound(lst, L1.y, lo1) : 0;
                const uint32_t e0 = hi1 != kFullMask ? lbound(lst, L1.y, hi1) : L1.y;
                const uint32_t xs = max(s0, min(r * grain, L1.y));
                const uint32_t xe = min(e0, min(r * grain + grain, L1.y));
                __syncwarp();
                if (lane == 0) {
                    c.S->moff[1] = L1.x;
                    c.S->mdeg[1] = L1.y;
                    c.S->tmin[1] = tm;
                    c.S->x[1] = xs;
                    c.S->xend[1] = max(xs, xe);
                }
                __syncwarp();
                subtree();
            }
            if (abandoned && lane == 0) {
                atomicOr(stop, 1u);
                aborted[cur] = 1;
            }
            if (qlimit && lane == 0) {
                atomicAdd(&qtime[cur], global_ns() - task_start);
                if (dropped) aborted[cur] = 1;
            }
        }
    }
    if (cur != kFullMask) add_count(&counts[cur], qcount, lane);
}

}  // namespace

// ---- host ---------------------------------------------------------------------

int batch_prepare_graph(DeviceGraph &g, uint32_t grain) {
    if (g.batch_vsorted && g.batch_grain == grain) return CUTS_OK;
    const uint32_t n = g.n;
    const int rc = host_degrees(g);
    if (rc) return rc;
    std::vector<uint32_t> vs(n);
    std::iota(vs.begin(), vs.end(), 0u);
    std::stable_sort(vs.begin(), vs.end(),
                     [&](uint32_t a, uint32_t b) { return g.h_out_deg[a] > g.h_out_deg[b]; });
    const int types = g.symmetric ? 1 : 3;
    std::vector<unsigned long long> pref(size_t(types) * (n + 1), 0);
    for (int t = 0; t < types; ++t) {
        unsigned long long *p = pref.data() + size_t(t) * (n + 1);
        for (uint32_t j = 0; j < n; ++j) {
            const uint32_t v = vs[j];
            const uint32_t len = t == 0 ? g.h_out_deg[v]
                                        : (t == 1 ? g.h_in_deg[v] : std::min(g.h_out_deg[v], g.h_in_deg[v]));
            p[j + 1] = p[j] + std::max<uint32_t>(1, (len + grain - 1) / grain);
        }
    }
    cudaFree(g.batch_vsorted);
    cudaFree(g.batch_pref);
    g.batch_vsorted = nullptr;
    g.batch_pref = nullptr;
    BCK(cudaMalloc(&g.batch_vsorted, sizeof(uint32_t) * std::max<uint32_t>(n, 1)));
    BCK(cudaMalloc(&g.batch_pref, sizeof(unsigned long long) * pref.size()));
    BCK(cudaMemcpy(g.batch_vsorted, vs.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice));
    BCK(cudaMemcpy(g.batch_pref, pref.data(), sizeof(unsigned long long) * pref.size(), cudaMemcpyHostToDevice));
    g.batch_grain = grain;
    g.batch_pref_host.swap(pref);
    return CUTS_OK;
}

void Batch::destroy() {
    if (spare) spare->destroy();
    spare.reset();
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    cudaFree(d_queries);
    cudaFree(d_qbase);
    cudaFree(d_counts);
    cudaFree(d_aborted);
    cudaFree(d_qtime);
    cudaFree(d_ctr);
    cudaFreeHost(h_counts);
    cudaFreeHost(h_aborted);
    cudaFreeHost(h_ctr);
    exec = nullptr;
    graph = nullptr;
    d_queries = nullptr;
    d_qbase = nullptr;
    d_counts = nullptr;
    d_aborted = nullptr;
    d_qtime = nullptr;
    d_ctr = nullptr;
    h_counts = nullptr;
    h_aborted = nullptr;
    h_ctr = nullptr;
}

// True when the level engine's plan for q counts its last levels fused,
// orbit-folded or as a pendant pair (prepare() in engine.cu makes the same
// choices).
static bool level_engine_pays(const Query &q, bool symmetric, uint32_t flags) {
    Plan plan;
    if (build_plan(q, symmetric, flags, plan)) return false;
    const uint32_t k = q.k;
    if (k < 3) return false;
    if ((flags & CUTS_FLAG_SYMMETRY_BREAK) && plan.lv[k - 1].ofold) return true;
    if (k >= 4 && plan.lv[k - 3].fold2) return true;  // a pendant pair counted in closed form
    const uint32_t cl = plan.lv[k - 2].fold ? k - 2 : k - 1;
    return plan.lv[cl].fuse != 0 && !(flags & CUTS_FLAG_NO_FUSE);
}

// True when the level engine counts q's last two levels as edges between two
// candidate sets (k_edges): a 4-cycle on 200,000 vertices / 1.6M edges takes
// 18 ms in a launch of its own here and 10 ms there.  Decided by graph and plan
// alone, not by the memory that the tables found: the shards of a batch on
// several GPUs have to take the same parts of a query.
static bool level_engine_edges(const Query &q, const DeviceGraph &g, uint32_t flags) {
    Plan plan;
    return g.ranked && edges_counted(flags) && !build_plan(q, g.symmetric, flags, plan) && edges_shape(plan);
}

int Batch::create(DeviceGraph &dg, const std::vector<const Query *> &qs, uint32_t flags_,
                  const BatchTuning &tune_) {
    g = &dg;
    flags = flags_;
    tune = tune_;
    // CUTS_BATCH_ROUTE=0 keeps every query in the persistent launch, =2 sends
    // every query of 4+ vertices to the level engine (A/B comparisons)
    const char *rt = std::getenv("CUTS_BATCH_ROUTE");
    route_level = !in_launch && !(rt && rt[0] == '0');
    route_all = !in_launch && rt && rt[0] == '2';
    if (tune.grain == 0) tune.grain = 64;
    if (tune.tasks_per_grab == 0) tune.tasks_per_grab = 1;
    BCK(cudaSetDevice(g->device));
    int rc = batch_prepare_graph(*g, tune.grain);
    if (rc) return rc;
    queries = qs;
    nq = uint32_t(qs.size());
    std::vector<BQuery> hq;
    std::vector<unsigned long long> qbase(1, 0);
    aut.assign(nq, 1);
    eligible.assign(nq, 0);
    const uint32_t n = g->n;
    unsigned long long light = 0;  // roots of one range, over all queries of the launch
    if ((rc = device_tables(*g))) return rc;
    for (uint32_t i = 0; i < nq; ++i) {
        const Query &q = *qs[i];
        Plan plan;
        rc = build_plan(q, g->symmetric, flags | CUTS_FLAG_NO_ORBIT_FOLD | CUTS_FLAG_NO_PAIR_FOLD, plan);  // plain fold only
        if (rc) return rc;
        aut[i] = plan.aut;
        BQuery b;
        std::memset(&b, 0, sizeof(b));
        bool ok = q.k >= 2 && q.k <= uint32_t(kBatchMaxK) && n > 0;
        for (uint32_t d = 0; ok && d < q.k; ++d) {
            const LevelPlan &L = plan.lv[d];
            if (L.nj > uint32_t(kBatchMaxJ)) { ok = false; break; }
            BLevel &B = b.lv[d];
            B.nj = L.nj;
            B.qin = L.qin;
            B.qout = L.qout;
            B.check_sig = L.check_sig;
            B.gt_mask = L.gt_mask;
            B.lt_mask = L.lt_mask;
            B.closed_form = L.closed_form;
            B.fold = L.fold;
            B.twin = L.twin;
            B.guar_mask = L.guar_mask;
            B.sig_lo = 0;
            if (d && B.check_sig && g->symmetric && g->ranked) {
                // degree-ranked ids: the signature is a compare of ids
                const uint32_t deg = std::max(B.qin, B.qout);
                B.sig_lo = n - uint32_t(deg < g->stats.out_ge.size() ? g->stats.out_ge[deg] : 0);
                B.check_sig = 0;
            }
            for (uint32_t t = 0; t < L.nj; ++t) {
                B.jpos[t] = L.jpos[t];
                B.jdir[t] = L.jdir[t];
            }
        }
        // queries of 4+ vertices whose counted levels the level engine fuses
        // (or, with symmetry breaking, orbit-folds) run there: its fused
        // count, dense-core rows and hub split have no counterpart in the
        // persistent kernel, which walks one candidate at a time
        if (ok && q.k >= 4 && route_level && (route_all || level_engine_pays(q, g->symmetric, flags))) ok = false;
        const bool edges = ok && q.k >= 4 && route_level && level_engine_edges(q, *g, flags);
        if (edges) ok = false;
        if (ok) {
            b.k = q.k;
            bool has_out = false, has_in = false;
            for (uint32_t t = 0; t < plan.lv[1].nj; ++t) (plan.lv[1].jdir[t] ? has_in : has_out) = true;
            b.type = g->symmetric ? 0 : (has_out && has_in ? 2 : (has_in ? 1 : 0));
            const uint32_t qout0 = plan.lv[0].qout;
            b.root_cnt = qout0 < g->stats.out_ge.size() ? uint32_t(g->stats.out_ge[qout0]) : 0;
            if (b.root_cnt == 0) {
                ok = false;  // no root passes: the count is 0 without a launch
            } else {
                const unsigned long long *pref = g->batch_pref_host.data() + size_t(b.type) * (n + 1);
                // the roots with several tasks each, in out-degree order (where
                // tasks are cut on another list: all of them)
                const size_t over = size_t(tune.grain) + 1;
                const uint64_t longer = over < g->stats.out_ge.size() ? g->stats.out_ge[over] : 0;
                b.heavy_roots = b.type == 0 ? uint32_t(std::min<uint64_t>(b.root_cnt, longer)) : b.root_cnt;
                info_tasks += pref[b.root_cnt];
                light += b.root_cnt - b.heavy_roots;
                hq.push_back(b);
                index.push_back(i);
            }
        }
        eligible[i] = ok ? 1 : edges ? 3 : (b.root_cnt == 0 && b.k ? 2 : 0);
    }
    // eligible: 1 = in the launch, 2 = no root (count 0), 0 = counted by the
    // level engine, 3 = the same, within the launch's budget
    nb = uint32_t(hq.size());
    for (BQuery &b : hq) {
        b.per = roots_per_task(b, light);
        const unsigned long long *pref = g->batch_pref_host.data() + size_t(b.type) * (n + 1);
        qbase.push_back(qbase.back() + pref[b.heavy_roots] + (b.root_cnt - b.heavy_roots + b.per - 1) / b.per);
    }
    total_tasks = qbase.back();
    BCK(cudaMalloc(&d_queries, sizeof(BQuery) * std::max<size_t>(hq.size(), 1)));
    BCK(cudaMalloc(&d_qbase, sizeof(unsigned long long) * qbase.size()));
    BCK(cudaMalloc(&d_counts, sizeof(unsigned long long) * std::max<uint32_t>(nb, 1)));
    BCK(cudaMalloc(&d_aborted, sizeof(uint32_t) * std::max<uint32_t>(nb, 1)));
    BCK(cudaMalloc(&d_qtime, sizeof(unsigned long long) * std::max<uint32_t>(nb, 1)));
    BCK(cudaMalloc(&d_ctr, sizeof(unsigned long long) * 2));
    BCK(cudaMallocHost(&h_counts, sizeof(unsigned long long) * std::max<uint32_t>(nb, 1)));
    BCK(cudaMallocHost(&h_aborted, sizeof(uint32_t) * std::max<uint32_t>(nb, 1)));
    BCK(cudaMallocHost(&h_ctr, sizeof(unsigned long long) * 2));
    if (nb) {
        BCK(cudaMemcpy(d_queries, hq.data(), sizeof(BQuery) * nb, cudaMemcpyHostToDevice));
    }
    BCK(cudaMemcpy(d_qbase, qbase.data(), sizeof(unsigned long long) * qbase.size(), cudaMemcpyHostToDevice));
    qbase_host.swap(qbase);
    return CUTS_OK;
}

int Batch::capture(unsigned long long budget_ns) {
    if (exec && budget_ns == captured_budget && query_budget_ms == captured_query_budget &&
        shard == captured_shard && nshards == captured_nshards && rshard == captured_rshard &&
        nrshards == captured_nrshards)
        return CUTS_OK;
    if (exec) { cudaGraphExecDestroy(exec); exec = nullptr; }
    if (graph) { cudaGraphDestroy(graph); graph = nullptr; }
    int bps = 0;
    BCK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_batch, kBW * 32, 0));
    int sms = 0;
    BCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device));
    if (tune.blocks_per_sm) bps = std::min<int>(bps, int(tune.blocks_per_sm));
    const unsigned long long maxb = (total_tasks / std::max<uint32_t>(nshards, 1) + kBW) / kBW;
    const uint32_t blocks = uint32_t(std::max<unsigned long long>(1, std::min<unsigned long long>(
        (unsigned long long)(std::max(1, bps) * sms), maxb)));
    const unsigned long long *pref = g->batch_pref;
    const size_t stride = size_t(g->n) + 1;
    cudaStream_t s = g->stream;
    BCK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    cudaMemsetAsync(d_counts, 0, sizeof(unsigned long long) * std::max<uint32_t>(nb, 1), s);
    cudaMemsetAsync(d_aborted, 0, sizeof(uint32_t) * std::max<uint32_t>(nb, 1), s);
    cudaMemsetAsync(d_qtime, 0, sizeof(unsigned long long) * std::max<uint32_t>(nb, 1), s);
    const unsigned long long qlimit =
        query_budget_ms > 0 ? (unsigned long long)(query_budget_ms * 1e6 * double(blocks) * kBW) : 0ull;
    cudaMemsetAsync(d_ctr, 0, sizeof(unsigned long long) * 2, s);
    if (nb) {
        k_batch<<<blocks, kBW * 32, 0, s>>>(
            graph_view(*g), d_queries, nb, d_qbase, g->batch_vsorted,
            pref, g->symmetric ? pref : pref + stride, g->symmetric ? pref : pref + 2 * stride, tune.grain,
            tune.tasks_per_grab, d_ctr, reinterpret_cast<uint32_t *>(d_ctr + 1), d_counts, d_aborted,
            budget_ns, d_qtime, qlimit, shard, nshards, rshard, nrshards);
    }
    cudaMemcpyAsync(h_counts, d_counts, sizeof(unsigned long long) * std::max<uint32_t>(nb, 1),
                    cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h_aborted, d_aborted, sizeof(uint32_t) * std::max<uint32_t>(nb, 1), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h_ctr, d_ctr, sizeof(unsigned long long) * 2, cudaMemcpyDeviceToHost, s);
    cudaGraph_t gr = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(s, &gr);
    if (ce != cudaSuccess) return set_error(CUTS_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(ce));
    graph = gr;
    BCK(cudaGraphInstantiate(&exec, graph, 0));
    captured_budget = budget_ns;
    captured_query_budget = query_budget_ms;
    captured_shard = shard;
    captured_nshards = nshards;
    captured_rshard = rshard;
    captured_nrshards = nrshards;
    launch_blocks = blocks;
    return CUTS_OK;
}

int Batch::run(double budget_ms, std::vector<uint64_t> &counts, std::vector<int> &status, float *ms) {
    BCK(cudaSetDevice(g->device));
    const unsigned long long budget_ns = budget_ms > 0 ? (unsigned long long)(budget_ms * 1e6) : 0ull;
    int rc = capture(budget_ns);
    if (rc) return rc;
    counts.assign(nq, 0);
    status.assign(nq, CUTS_OK);
    BCK(cudaEventRecord(g->ev0, g->stream));
    BCK(cudaGraphLaunch(exec, g->stream));
    BCK(cudaEventRecord(g->ev1, g->stream));
    BCK(cudaStreamSynchronize(g->stream));
    float t = 0;
    BCK(cudaEventElapsedTime(&t, g->ev0, g->ev1));
    // tasks below stop_at were all taken (counter values map to c * nshards + shard)
    const unsigned long long stop_at = std::min<unsigned long long>(h_ctr[0] * nshards + shard, total_tasks);
    const bool stopped = reinterpret_cast<uint32_t *>(h_ctr + 1)[0] != 0;
    for (uint32_t b = 0; b < nb; ++b) {
        const uint32_t i = index[b];
        counts[i] = uint64_t(h_counts[b]) * aut[i];
        const bool unfinished = h_aborted[b] || (stopped && qbase_host[b + 1] > stop_at);
        if (unfinished) status[i] = CUTS_ERR_BUDGET;
    }
    // queries outside the batched kernel's limits, and those the level engine
    // is better at: one by one
    double left = budget_ms - t;  // of the launch's budget, where there is one
    std::vector<uint32_t> again;  // the level engine has no room for these
    for (uint32_t i = 0; i < nq; ++i) {
        if (eligible[i] != 0 && eligible[i] != 3) continue;
        CountResult r;
        CountOptions opt;
        opt.flags = flags;
        opt.budget_ms = query_budget_ms;
        if (eligible[i] == 3 && budget_ms > 0) {
            if (left <= 0) {
                status[i] = CUTS_ERR_BUDGET;
                continue;
            }
            opt.budget_ms = query_budget_ms > 0 ? std::min(query_budget_ms, left) : left;
        }
        opt.shard = shard;
        opt.nshards = nshards;
        rc = device_count(*g, *queries[i], opt, r);
        if (eligible[i] == 3 && (rc == CUTS_ERR_CAPACITY || rc == CUTS_ERR_NOMEM)) {
            again.push_back(i);
            continue;
        }
        if (rc) {
            if (eligible[i] == 3) left -= opt.budget_ms;
            status[i] = rc;
            continue;
        }
        if (eligible[i] == 3) left -= r.ms;
        counts[i] = r.count;
        t += r.ms;
    }
    if (!again.empty()) {
        rc = budget_ms > 0 && left <= 0 ? CUTS_ERR_BUDGET
                                        : run_spare(again, budget_ms > 0 ? left : 0, counts, status, t);
        if (rc)
            for (uint32_t i : again) status[i] = rc;
    }
    if (ms) *ms = t;
    return CUTS_OK;
}

int Batch::run_spare(const std::vector<uint32_t> &which, double budget_ms, std::vector<uint64_t> &counts,
                     std::vector<int> &status, float &ms) {
    if (!spare || spare_of != which) {
        if (spare) spare->destroy();
        spare = std::make_unique<Batch>();
        spare_of.clear();
        spare->in_launch = true;
        std::vector<const Query *> qs;
        for (uint32_t i : which) qs.push_back(queries[i]);
        const int rc = spare->create(*g, qs, flags, tune);
        if (rc) {
            spare->destroy();
            spare.reset();
            return rc;
        }
        spare_of = which;
    }
    spare->set_query_budget(query_budget_ms);
    // the shard by roots, as the level engine takes it on the other GPUs
    spare->rshard = shard;
    spare->nrshards = nshards;
    std::vector<uint64_t> c;
    std::vector<int> st;
    float t = 0;
    const int rc = spare->run(budget_ms, c, st, &t);
    if (rc) return rc;
    for (size_t j = 0; j < which.size(); ++j) {
        counts[which[j]] = c[j];
        status[which[j]] = st[j];
    }
    ms += t;
    return CUTS_OK;
}

// ---- allocation-free entry point ---------------------------------------------
//
// For callers that may not allocate GPU memory themselves: code running inside
// a host framework that owns every device allocation (a memory pool that must
// account for all bytes, a plugin sandbox).
// They pass the graph and the output buffer they already own; the engine's
// own scratch for this path -- the per-query plans and the work counter --
// lives in the fixed array below, which every GPU that loads this library
// holds until the process exits.
namespace {

constexpr uint32_t kNoAllocMaxQueries = 64;  // queries per call

struct NoAllocScratch {
    BQuery queries[kNoAllocMaxQueries];
    unsigned long long task_ctr;
    uint32_t stop;
    uint32_t longest;  // the graph's longest list
    uint32_t aborted[kNoAllocMaxQueries];
};

static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoAllocScratch)];

// Device address of g_noalloc_scratch per device ordinal (the host-side
// symbol is only a stand-in, never a device address), and the launch shape.
constexpr int kNoAllocMaxDevices = 64;
NoAllocScratch *g_noalloc_ptr[kNoAllocMaxDevices] = {};
uint32_t g_noalloc_blocks[kNoAllocMaxDevices] = {};
std::mutex g_noalloc_mutex;

// The query plans travel as kernel parameters, copied into the scratch array
// by a one-block kernel: the launch records them by value when it is queued,
// so the call needs no host staging buffer and returns without waiting.
constexpr uint32_t kNoAllocPlansPerLaunch = 16;  // 16 x 660 B of parameters
struct NoAllocPlans {
    BQuery q[kNoAllocPlansPerLaunch];
};

__global__ void k_noalloc_plans(const NoAllocPlans plans, uint32_t first, uint32_t count,
                                NoAllocScratch *__restrict__ sc) {
    const uint32_t words = count * uint32_t(sizeof(BQuery) / 4);
    const uint32_t *src = reinterpret_cast<const uint32_t *>(plans.q);
    uint32_t *dst = reinterpret_cast<uint32_t *>(sc->queries + first);
    for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
    // the work counter and the stop flag start at zero
    if (first == 0 && threadIdx.x == 0) {
        sc->task_ctr = 0;
        sc->stop = 0;
        sc->longest = 0;
    }
}

// The longest list, for the number of slices (one launch more than the plans':
// it saves the empty slices' tasks, an atomic each, on graphs without hubs).
__global__ void __launch_bounds__(256)
k_noalloc_longest(const uint2 *__restrict__ info_out, const uint2 *__restrict__ info_in, uint32_t n,
                  NoAllocScratch *__restrict__ sc) {
    uint32_t len = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        len = max(len, max(info_out[v].y, info_in[v].y));
    len = __reduce_max_sync(kFullMask, len);
    if ((threadIdx.x & 31) == 0) atomicMax(&sc->longest, len);
}

// Tasks are (slice, query, block of up to 32 roots): the lanes look at the
// block's roots at once, and of each root that passes the level-0 signature the
// warp runs the slice's part of its level-1 list depth first, with the same
// level steps as k_batch.  Slice r of (up to) kSlices holds the blocks b of
// kSliceLen level-1 candidates with b % slices == r, so a hub's work is spread
// over as many warps; the slices above 0, empty for most roots, come first, and
// there are only as many as the longest list has.  With the whole list of a root
// as one task, hubs were the launch's tail: 16 queries of 2-4 vertices on 50,001
// vertices / 300,000 edges took 67.5 ms, 3.7 ms this way (frontiers counted at
// once and twins included).  Slice 0, where nearly all work is, has blocks of 32
// in calls with roots enough; of fewer roots a block takes so many that every
// warp gets several (na_block): 4 queries on 200 vertices 0.20 ms in blocks of
// 32, 0.06 this way, one of 6 vertices on 3,000 vertices / 9,000 edges 0.91 and
// 0.27 (0.08 and 0.47 with one root per task).  No budget: every query runs to
// completion.
constexpr uint32_t kSlices = 16;
constexpr uint32_t kSliceLen = 32;

// Roots per block of slice 0 for `roots` (query, root) pairs on `warps` warps: 4
// blocks a warp or more, 16 where subtrees are deep (5 vertices and more).
uint32_t na_block(unsigned long long roots, uint32_t warps, bool deep) {
    const unsigned long long per = roots / ((unsigned long long)warps * (deep ? 16 : 4));
    return uint32_t(std::max<unsigned long long>(1, std::min<unsigned long long>(32, per)));
}

__global__ void __launch_bounds__(kBW * 32)
k_batch_noalloc(DevView g, NoAllocScratch *__restrict__ sc, uint32_t nq, uint32_t blk, uint32_t deep,
                unsigned long long *__restrict__ counts) {
    __shared__ BWarp ws[kBW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Ctx c{g, nullptr, &ws[warp], lane};
    // the task space, in shared memory (registers are what this kernel is short of)
    __shared__ unsigned long long upper, total;  // tasks of the slices above 0, and all
    __shared__ uint32_t slices, nblk[2], upblk;
    if (threadIdx.x == 0) {
        slices = min(kSlices, (max(sc->longest, 1u) - 1) / kSliceLen + 1);
        // blocks of the slices above 0: most such tasks find nothing, but a few
        // roots of deep queries in one are a tail where there are few slices
        upblk = max(blk, deep ? min(8u, slices) : 32u);
        nblk[0] = (g.n - 1) / upblk + 1;
        nblk[1] = (g.n - 1) / blk + 1;
        upper = (unsigned long long)nq * nblk[0] * (slices - 1);
        total = upper + (unsigned long long)nq * nblk[1];
    }
    __syncthreads();
    uint32_t cur = kFullMask;
    unsigned long long qcount = 0;
    while (true) {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(&sc->task_ctr, 1ull);
        t = __shfl_sync(kFullMask, t, 0);
        if (t >= total) break;
        const bool first = t >= upper;  // slice 0
        const uint32_t nb = nblk[first], roots = first ? blk : upblk;
        const unsigned long long at = first ? t - upper : t;
        const uint32_t run = uint32_t(at / nb), u0 = uint32_t(at - (unsigned long long)run * nb) * roots;
        const uint32_t q = first ? run : run % nq, slice = first ? 0u : slices - 1 - run / nq;
        if (q != cur) {
            if (cur != kFullMask) add_count(&counts[cur], qcount, lane);
            qcount = 0;
            cur = q;
            c.Q = sc->queries + q;
        }
        const BQuery &Q = *c.Q;
        if (Q.k < 2) continue;
        // the block's roots with level-1 candidates in this slice
        bool pass = false;
        if (uint32_t(lane) < roots && u0 + lane < g.n) {
            const uint2 uo = g.out_info[u0 + lane], ui = g.in_info[u0 + lane];
            uint32_t len = kFullMask;
            for (uint32_t j = 0; j < Q.lv[1].nj; ++j) len = min(len, Q.lv[1].jdir[j] ? ui.y : uo.y);
            pass = ui.y >= Q.lv[0].qin && uo.y >= Q.lv[0].qout && len != kFullMask && len > slice * kSliceLen;
        }
        for (unsigned todo = __ballot_sync(kFullMask, pass); todo; todo &= todo - 1) {
            if (lane == 0) c.S->m[0] = u0 + __ffs(todo) - 1;
            __syncwarp();
            enter_level(c, 1);  // the whole shortest level-1 list
            const uint32_t xend = c.S->xend[1];
            for (uint32_t x0 = slice * kSliceLen; x0 < xend; x0 += slices * kSliceLen) {
                __syncwarp();
                if (lane == 0) {
                    c.S->x[1] = x0;
                    c.S->xend[1] = min(x0 + kSliceLen, xend);
                    c.S->nb[1] = 0;
                    c.S->bi[1] = 0;
                }
                __syncwarp();
                if (Q.k == 2 || (Q.k == 3 && Q.lv[1].fold)) {
                    const unsigned long long r1 = Q.k == 2 ? count_level(c, 1) : count_level_fold(c, 1);
                    if (lane == 0) qcount += r1;  // the warp's
                    continue;
                }
                uint32_t d = 1;
                while (d >= 1) {
                    if (c.S->bi[d] < c.S->nb[d]) {
                        if (counts_next(Q, d)) {
                            qcount += count_frontier(c, d);
                            __syncwarp();
                            if (lane == 0) c.S->bi[d] = c.S->nb[d];
                            __syncwarp();
                        } else {
                            descend(c, d);
                            ++d;
                        }
                    } else if (c.S->x[d] < c.S->xend[d]) {
                        refill(c, d);
                    } else {
                        --d;
                    }
                }
            }
            __syncwarp();
        }
    }
    if (cur != kFullMask) add_count(&counts[cur], qcount, lane);
}

}  // namespace

int count_noalloc(const uint32_t *info_out, const uint32_t *info_in, const uint32_t *adj, uint32_t n,
                  int symmetric, const Query *const *qs, uint32_t nq, uint32_t flags,
                  unsigned long long *counts, cudaStream_t stream) {
    if (!info_out || !adj || !counts || (nq && !qs))
        return set_error(CUTS_ERR_ARG, "cuts_count_noalloc: null argument");
    if (nq > kNoAllocMaxQueries)
        return set_error(CUTS_ERR_LIMIT, "cuts_count_noalloc: more than 64 queries in one call");
    if (flags & CUTS_FLAG_SYMMETRY_BREAK)
        return set_error(CUTS_ERR_ARG, "cuts_count_noalloc: symmetry breaking is not available here");
    // the query plans, built on the stack (fixed size, no allocation)
    NoAllocPlans table[kNoAllocMaxQueries / kNoAllocPlansPerLaunch];
    const bool sym = symmetric != 0 || info_in == nullptr;
    bool deep = false;
    for (uint32_t i = 0; i < nq; ++i) {
        if (!qs[i]) return set_error(CUTS_ERR_ARG, "cuts_count_noalloc: null query");
        const Query &q = *qs[i];
        if (q.k > uint32_t(kBatchMaxK))
            return set_error(CUTS_ERR_LIMIT, "cuts_count_noalloc: query with more than 10 vertices");
        Plan plan;
        int rc = build_plan(q, sym, flags | CUTS_FLAG_NO_ORBIT_FOLD | CUTS_FLAG_NO_PAIR_FOLD, plan);  // plain fold only
        if (rc) return rc;
        BQuery &b = table[i / kNoAllocPlansPerLaunch].q[i % kNoAllocPlansPerLaunch];
        std::memset(&b, 0, sizeof(b));
        b.k = q.k;
        deep = deep || q.k >= 5;
        for (uint32_t d = 0; d < q.k; ++d) {
            const LevelPlan &L = plan.lv[d];
            if (L.nj > uint32_t(kBatchMaxJ))
                return set_error(CUTS_ERR_LIMIT, "cuts_count_noalloc: more than 8 joined lists at a level");
            BLevel &B = b.lv[d];
            B.nj = L.nj;
            B.qin = L.qin;
            B.qout = L.qout;
            B.check_sig = L.check_sig;
            B.gt_mask = L.gt_mask;
            B.lt_mask = L.lt_mask;
            B.closed_form = L.closed_form;
            B.fold = L.fold;
            B.twin = L.twin;
            B.guar_mask = L.guar_mask;
            B.sig_lo = 0;
            for (uint32_t t = 0; t < L.nj; ++t) {
                B.jpos[t] = L.jpos[t];
                B.jdir[t] = L.jdir[t];
            }
        }
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices)
        return set_error(CUTS_ERR_CUDA, "cuts_count_noalloc: no current CUDA device");
    NoAllocScratch *sc = nullptr;
    uint32_t blocks = 0;
    {
        // once per device, with that device current: the scratch array's
        // device address and the persistent grid size
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!g_noalloc_ptr[dev]) {
            void *p = nullptr;
            if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p)
                return set_error(CUTS_ERR_CUDA, "cuts_count_noalloc: cudaGetSymbolAddress failed");
            int bps = 0, sms = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_batch_noalloc, kBW * 32, 0) != cudaSuccess ||
                cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
                return set_error(CUTS_ERR_CUDA, "cuts_count_noalloc: device query failed");
            g_noalloc_blocks[dev] = uint32_t(std::max(1, bps) * std::max(1, sms));
            g_noalloc_ptr[dev] = static_cast<NoAllocScratch *>(p);
        }
        sc = g_noalloc_ptr[dev];
        blocks = g_noalloc_blocks[dev];
    }
    // nothing to count: the caller's counts buffer (nq entries) is not touched
    if (nq == 0) return CUTS_OK;
    // counts start at zero on every call
    if (cudaMemsetAsync(counts, 0, sizeof(unsigned long long) * nq, stream) != cudaSuccess)
        return set_error(CUTS_ERR_CUDA, "cuts_count_noalloc: memset failed");
    if (n == 0) return CUTS_OK;
    for (uint32_t first = 0; first < nq; first += kNoAllocPlansPerLaunch) {
        const uint32_t cnt = std::min(kNoAllocPlansPerLaunch, nq - first);
        k_noalloc_plans<<<1, 256, 0, stream>>>(table[first / kNoAllocPlansPerLaunch], first, cnt, sc);
        if (cudaGetLastError() != cudaSuccess)
            return set_error(CUTS_ERR_CUDA, "cuts_count_noalloc: plan upload failed");
    }
    const DevView view{reinterpret_cast<const uint2 *>(info_out),
                       reinterpret_cast<const uint2 *>(sym ? info_out : info_in), adj, n, nullptr, nullptr,
                       nullptr, 0, nullptr};
    const uint32_t blk = na_block((unsigned long long)nq * n, blocks * kBW, deep);
    k_noalloc_longest<<<std::min<uint32_t>((n - 1) / 256 + 1, blocks), 256, 0, stream>>>(view.out_info, view.in_info, n, sc);
    const unsigned long long total =
        (unsigned long long)nq * ((n - 1) / blk + 1) * kSlices;  // at most
    const uint32_t grid = uint32_t(std::min<unsigned long long>(blocks, (total + kBW - 1) / kBW));
    k_batch_noalloc<<<std::max<uint32_t>(grid, 1), kBW * 32, 0, stream>>>(view, sc, nq, blk, deep ? 1 : 0, counts);
    if (cudaGetLastError() != cudaSuccess)
        return set_error(CUTS_ERR_CUDA, "cuts_count_noalloc: launch failed");
    return CUTS_OK;
}

}  // namespace cuts
