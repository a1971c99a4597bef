// engine.cu -- device layout, level kernels and the chunked level driver.
//
// Method (the reference's, device_funcs.cu:267-405 and host_funcs.cu:
// 39-171): a vertex-at-a-time join along the matching order.  Level L_0
// holds the root candidates; level L_i holds (vertex, parent index) trie
// entries, each extending one entry of L_{i-1} by a data vertex that lies
// in every joined adjacency list, is not matched yet and passes the degree
// signature.  The last level is counted, not stored.
//
// B200 layout of the work:
//   * a warp takes up to 32 parent entries, one per lane, handed out by a global
//     work cursor in turns (work stealing across all SMs of a persistent grid);
//   * each parent's smallest joined list supplies its candidates, the windows of
//     all lanes one sequence walked 64 a step; membership in the other lists is
//     one table read (in_list), a search of the list without tables;
//   * the last two or three levels are counted together where the plan allows:
//     closed forms and folds (k_level_flat), pairs of one candidate set (k_pairs,
//     k_fused), edges between two (k_edges);
//   * survivors are placed with a warp ballot/popc into a per-warp shared
//     staging buffer and flushed with one global atomic per buffer, so the
//     next level is written in coalesced runs;
//   * each stored entry carries an upper bound on its own child count (the
//     shortest list it will join at the next level); a tile-sum + scan
//     planner cuts every level into chunks whose bound fits the level's
//     capacity, and the driver expands chunk by chunk depth-first, so the
//     trie never exceeds the arena whatever the graph.
#include <cuda_runtime.h>

#include <algorithm>
#include <cerrno>
#include <charconv>
#include <chrono>
#include <climits>
#include <cstdlib>
#include <cstdio>
#include <memory>
#include <cstring>
#include <string>
#include <vector>

#include <omp.h>

#include "device_util.cuh"
#include "engine.hpp"

namespace cuts {

#define CK(call)                                                                       \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess)                                                         \
            return set_error(CUTS_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

namespace {

constexpr uint32_t kFull = 0xffffffffu;
constexpr int kWarps = 8;       // warps per block in the level kernels
constexpr int kOutBuf = 128;    // per-warp staged output entries
constexpr uint32_t kTile = 256; // planner tile (parents)

// Plan + level pointers, resident in device memory for the run.
struct RunParams {
    Plan plan;
    uint32_t stored;   // levels kept in HBM: k-1 when counting, k when dumping
    // level whose entries keep, in their ub slot, the adj offset their vertex
    // was drawn from (the last stored level before a fused count: its child
    // bound is never read); kFull = none
    uint32_t pos_lvl;
    uint32_t fuse_stride;  // words per warp row of the fused kernel's scratch
    uint32_t *fuse_scratch;
    uint32_t edges;        // levels k-2 and k-1 are counted by k_edges
    uint32_t pairs;        // the fused count runs in k_pairs (else k_fused)
    uint32_t *fuse_big;    // the fused kernel's deferred parents (arrays, pool or bitmaps)
    uint32_t fuse_big_cap;
    uint32_t fuse_pool_words;
    uint32_t *vert[kMaxK];
    uint32_t *par[kMaxK];
    uint32_t *ub[kMaxK];
    // device-time budget: kernels take no more work once budget_ns has
    // passed since *stamp (written by k_roots) and raise *over instead
    unsigned long long budget_ns;
    unsigned long long *stamp;
    uint32_t *over;
};

// Absolute device-clock deadline of a budgeted run (0 = none).
__device__ __forceinline__ unsigned long long run_deadline(const RunParams *rp) {
    const unsigned long long b = rp->budget_ns;
    return b ? *rp->stamp + b : 0ull;
}

// True (and the run flagged) once the deadline has passed; lane 0 calls it.
__device__ __forceinline__ bool past_deadline(const RunParams *rp, unsigned long long deadline) {
    if (!deadline || global_ns() <= deadline) return false;
    atomicOr(rp->over, 1u);
    return true;
}

// Orbit fold (a pendant's closed form summed over its attachment orbit O):
// the part of the weight fixed by positions below `upto`,
//   sum_{x in O, x < upto} ( |L(m_x)| - #{j < upto : m_j in L(m_x)} ),
// where m(j) gives the matched vertex of position j.
template <class M>
__device__ __forceinline__ uint32_t orbit_base(const DevView &g, const LevelPlan &F, uint32_t upto, bool loops, M m) {
    uint32_t base = 0;
    for (uint32_t xm = F.ofold & ((1u << upto) - 1); xm; xm &= xm - 1) {
        const uint32_t x = __ffs(xm) - 1;
        const uint2 inf = F.jdir[0] ? g.in_info[m(x)] : g.out_info[m(x)];
        uint32_t sub = 0;
        for (uint32_t j = 0; j < upto; ++j)
            if (((F.oguar[x] >> j) & 1u) || ((loops || j != x) && in_list(g, inf.x, inf.y, m(j)))) ++sub;
        base += inf.y - sub;
    }
    return base;
}

// The weight of candidate t at position c given the base of positions below
// c: each earlier orbit list holds t (implied by the query's arcs, checked at
// plan time), and when c is in the orbit, t's own list holds every m_j, j < c.
__device__ __forceinline__ uint32_t orbit_weight(const DevView &g, const LevelPlan &F, uint32_t c,
                                                 uint32_t base, uint32_t t, bool loops) {
    uint32_t w = base - __popc(F.ofold & ((1u << c) - 1));
    if ((F.ofold >> c) & 1u) {
        const uint2 ti = F.jdir[0] ? g.in_info[t] : g.out_info[t];
        w += ti.y - c;
        if (loops && in_list(g, ti.x, ti.y, t)) --w;
    }
    return w;
}

// Pendant pair (plan fold2 at level k-3; A = level k-2's plan, B = level
// k-1's, both joining the same list): with m(j) the matched vertex of
// position j <= k-3, the number of (t1, t2) with t1 in A's window of the
// list, t2 in B's, both unmatched, t1 != t2, and -- kind 2 -- t2 above
// (below) t1 on the same window.  O(log degree) per candidate.  Adds |A'|
// (the level k-2 size) to lvl2.  The lists' own vertex is in them only where
// there are self-loops, so a star tests nothing (3-star, 1M vertices / 10M
// edges, plain / symmetry breaking 60 / 107 ms with its table tests per
// candidate, 40 / 71 without; 21 / 38 in an instance of its own).
template <class M>
__device__ uint64_t pendant_pairs(const DevView &g, const LevelPlan &A, const LevelPlan &B, uint32_t kind,
                                  uint32_t lvl, bool loops, M m, unsigned long long &lvl2) {
    const uint32_t pen = 1u << (lvl + 1);
    uint32_t lo[2], hi[2], s0[2], e0[2], off[2], len[2], cnt[2], u[2];
    auto has = [&](int r, uint32_t guar, uint32_t j, uint32_t mj) {
        return ((guar >> j) & 1u) || ((loops || mj != u[r]) && in_list(g, off[r], len[r], mj));
    };
    for (int r = 0; r < 2; ++r) {
        const LevelPlan &L = r ? B : A;
        u[r] = m(L.jpos[0]);
        const uint2 inf = L.jdir[0] ? g.in_info[u[r]] : g.out_info[u[r]];
        off[r] = inf.x;
        len[r] = inf.y;
        lo[r] = 0;
        hi[r] = kFullMask;
        for (uint32_t msk = L.gt_mask & ~pen; msk; msk &= msk - 1) lo[r] = max(lo[r], m(__ffs(msk) - 1) + 1);
        for (uint32_t msk = L.lt_mask & ~pen; msk; msk &= msk - 1) hi[r] = min(hi[r], m(__ffs(msk) - 1));
        const uint32_t *l = g.adj + off[r];
        const bool dir = L.jdir[0] != 0;
        s0[r] = lo[r] ? lbound_own(g, dir, u[r], l, len[r], lo[r], loops) : 0;
        e0[r] = hi[r] != kFullMask ? lbound_own(g, dir, u[r], l, len[r], hi[r], loops) : len[r];
        if (e0[r] < s0[r]) e0[r] = s0[r];
        const uint32_t guar = r ? B.guar_mask : A.guar1;
        uint32_t sub = 0;
        for (uint32_t j = 0; j <= lvl; ++j) {
            const uint32_t mj = m(j);
            if (mj >= lo[r] && mj < hi[r] && has(r, guar, j, mj)) ++sub;
        }
        cnt[r] = e0[r] - s0[r] - sub;
    }
    lvl2 += cnt[0];
    if (kind == 2) return uint64_t(cnt[0]) * (cnt[0] - (cnt[0] ? 1 : 0)) / 2;
    // |A'| |B'| - |A' n B'|
    uint64_t both = 0;
    const uint32_t wlo = max(lo[0], lo[1]), whi = min(hi[0], hi[1]);
    if (wlo < whi) {
        // one list: its entries in both windows form the window [wlo, whi)
        const uint32_t a = max(s0[0], s0[1]), b = min(e0[0], e0[1]);
        both = b > a ? b - a : 0;
        // matched vertices lying in both windows and lists
        for (uint32_t j = 0; j <= lvl; ++j) {
            const uint32_t mj = m(j);
            if (mj < wlo || mj >= whi) continue;
            if (has(0, A.guar1, j, mj) && has(1, B.guar_mask, j, mj)) --both;
        }
    }
    return uint64_t(cnt[0]) * cnt[1] - both;
}

enum Mode { kExpand = 0, kCountMode = 1, kBytesMode = 2 };

// The parents [pa, pa + total) of one launch.  Either the host knows them
// (n null), or the launch was queued behind the one that writes their number:
// then *n is read here, slice `slice` of `slices` of it is taken (root
// slices), and an expanding launch whose children may not fit the level
// (*bound > cap) raises *stop, which every later launch of the chain obeys,
// so the host can go on from this level in chunks.
struct Parents {
    const uint32_t *n;
    uint32_t a, b;             // host-known range
    uint32_t slice, slices;
    const unsigned long long *bound;
    unsigned long long cap;
    uint32_t *stop;
    uint32_t code;             // what *stop says about this launch (never 0)
};

__device__ __forceinline__ void parents_of(const Parents &P, uint32_t &pa, uint32_t &total) {
    if (!P.n) {
        pa = P.a;
        total = P.b - P.a;
        return;
    }
    pa = total = 0;
    if (*reinterpret_cast<volatile uint32_t *>(P.stop)) return;
    if (P.bound && *P.bound > P.cap) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *P.stop = P.code;
        return;
    }
    const uint32_t n = *P.n;
    if (!n) return;
    const uint32_t per = (n - 1) / P.slices + 1;
    const unsigned long long a = (unsigned long long)P.slice * per, end = a + per;
    if (a >= n) return;
    pa = uint32_t(a);
    // (as min(per, n - pa) in 32 bits, nvcc 12.9.86 gave `per` for a short
    // last slice in k_fused)
    total = uint32_t((end < n ? end : n) - a);
}

// ---- level 0: signature scan (device_funcs.cu:267-279) ---------------
__global__ void k_roots(DevView g, const RunParams *__restrict__ rp, uint32_t shard, uint32_t nshards,
                        uint32_t *__restrict__ n0, unsigned long long *__restrict__ bound) {
    const Plan &P = rp->plan;
    const uint32_t qin = P.lv[0].qin, qout = P.lv[0].qout;
    // L_0 entries carry the child bound for level 1, whose joins all use
    // position 0 (only needed when level 1 is stored)
    const bool need_ub = rp->stored >= 2;
    bool use_out = false, use_in = false;
    if (P.k >= 2)
        for (uint32_t t = 0; t < P.lv[1].nj; ++t) (P.lv[1].jdir[t] ? use_in : use_out) = true;
    uint32_t *vert0 = rp->vert[0], *ub0 = rp->ub[0];
    const int lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x == 0 && rp->budget_ns) *rp->stamp = global_ns();
    unsigned long long sum = 0;  // of the child bounds
    for (uint32_t base = blockIdx.x * blockDim.x; base < g.n; base += gridDim.x * blockDim.x) {
        const uint32_t u = base + threadIdx.x;
        bool ok = false;
        uint32_t ub = UINT_MAX;
        if (u < g.n && u % nshards == shard) {  // rank striding, device_funcs.cu:273
            const uint2 o = g.out_info[u], i = g.in_info[u];
            ok = o.y >= qout && i.y >= qin;
            if (use_out) ub = min(ub, o.y);
            if (use_in) ub = min(ub, i.y);
        }
        const unsigned m = __ballot_sync(kFull, ok);
        if (m) {
            uint32_t pos = 0;
            if (lane == 0) pos = atomicAdd(n0, uint32_t(__popc(m)));
            pos = __shfl_sync(kFull, pos, 0) + __popc(m & ((1u << lane) - 1));
            if (ok) {
                vert0[pos] = u;
                if (need_ub) {
                    ub0[pos] = ub;
                    sum += ub;
                }
            }
        }
    }
    #pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
    if (lane == 0 && sum) atomicAdd(bound, sum);
}

// ---- levels 1..k-1 -----------------------------------------------------
// MODE kExpand: write L_lvl from parents [pa, pb) of L_{lvl-1}.
// MODE kCountMode: last level, accumulate the count.
// MODE kBytesMode: accumulate the algorithmic bytes of the last level.
template <int MODE>
__global__ void __launch_bounds__(kWarps * 32)
k_level(DevView g, const RunParams *__restrict__ rp, uint32_t lvl, uint32_t pa, uint32_t pb,
        uint32_t grain, uint32_t *__restrict__ cursor, uint32_t *__restrict__ out_n,
        uint32_t out_cap, uint32_t *__restrict__ err, unsigned long long *__restrict__ acc) {
    __shared__ LevelPlan sL, sN;
    __shared__ uint32_t *s_vert[kMaxK];
    __shared__ uint32_t *s_par[kMaxK];
    __shared__ uint32_t s_k, s_sym, s_stored;
    __shared__ uint32_t wm[kWarps][kMaxK];
    __shared__ uint32_t joff[kWarps][kMaxJ], jdeg[kWarps][kMaxJ];
    __shared__ uint32_t ob_v[MODE == kExpand ? kWarps : 1][kOutBuf];
    __shared__ uint32_t ob_p[MODE == kExpand ? kWarps : 1][kOutBuf];
    __shared__ uint32_t ob_u[MODE == kExpand ? kWarps : 1][kOutBuf];

    {
        const uint32_t words = sizeof(LevelPlan) / 4;
        const uint32_t *srcL = reinterpret_cast<const uint32_t *>(&rp->plan.lv[lvl]);
        uint32_t *dL = reinterpret_cast<uint32_t *>(&sL);
        for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) dL[i] = srcL[i];
        const uint32_t nl = lvl + 1 < rp->plan.k ? lvl + 1 : lvl;
        const uint32_t *srcN = reinterpret_cast<const uint32_t *>(&rp->plan.lv[nl]);
        uint32_t *dN = reinterpret_cast<uint32_t *>(&sN);
        for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) dN[i] = srcN[i];
        if (threadIdx.x < kMaxK) {
            s_vert[threadIdx.x] = rp->vert[threadIdx.x];
            s_par[threadIdx.x] = rp->par[threadIdx.x];
        }
        if (threadIdx.x == 0) { s_k = rp->plan.k; s_sym = rp->plan.symmetric; s_stored = rp->stored; }
    }
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t lanemask_lt = (1u << lane) - 1;
    uint32_t *my_m = wm[warp];
    const uint32_t k = s_k;
    const bool sym = s_sym != 0;
    // entries of L_lvl need a child bound when level lvl+1 is stored too; at
    // the position level the slot keeps where the vertex sits in its list
    const bool store_pos = MODE == kExpand && lvl == rp->pos_lvl;
    const bool need_ub = (MODE == kExpand && lvl + 1 < s_stored) || store_pos;
    uint32_t *out_v = MODE == kExpand ? rp->vert[lvl] : nullptr;
    uint32_t *out_p = MODE == kExpand ? rp->par[lvl] : nullptr;
    uint32_t *out_u = MODE == kExpand ? rp->ub[lvl] : nullptr;
    // next-level joins on the child itself (position lvl) bound its children
    bool ub_out = false, ub_in = false;
    if (need_ub && !store_pos)
        for (uint32_t t = 0; t < sN.nj; ++t)
            if (sN.jpos[t] == lvl) (sN.jdir[t] ? ub_in : ub_out) = true;
    const uint32_t nj = sL.nj;
    const bool check_sig = sL.check_sig != 0;
    const bool load_info = check_sig || ub_out || ub_in;

    uint32_t cached_q = kFull;  // lane 0: L_{lvl-2} index whose path is in my_m[0..lvl-2]
    uint32_t obn = 0;           // staged outputs (warp-uniform)
    unsigned long long local = 0;
    const uint32_t total = pb - pa;
    const unsigned long long deadline = run_deadline(rp);

    auto flush = [&]() {
        if constexpr (MODE != kExpand) return;
        __syncwarp();
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(out_n, obn);
        base = __shfl_sync(kFull, base, 0);
        if (base + obn <= out_cap && base + obn >= base) {
            for (uint32_t i = lane; i < obn; i += 32) {
                out_v[base + i] = ob_v[warp][i];
                out_p[base + i] = ob_p[warp][i];
                if (need_ub) out_u[base + i] = ob_u[warp][i];
            }
        } else if (lane == 0) {
            atomicOr(err, 1u);
        }
        obn = 0;
        __syncwarp();
    };

    while (true) {
        uint32_t start = 0;
        if (lane == 0) start = past_deadline(rp, deadline) ? total : atomicAdd(cursor, grain);
        start = __shfl_sync(kFull, start, 0);
        if (start >= total) break;
        const uint32_t end = min(start + grain, total);
        for (uint32_t pi = start; pi < end; ++pi) {
            const uint32_t p = pa + pi;
            // rebuild the parent's partial match (device_funcs.cu:39-55),
            // reusing the ancestors shared with the previous parent
            if (lane == 0) {
                my_m[lvl - 1] = s_vert[lvl - 1][p];
                if (lvl >= 2) {
                    uint32_t q = s_par[lvl - 1][p];
                    if (q != cached_q) {
                        cached_q = q;
                        for (int j = int(lvl) - 2; j >= 0; --j) {
                            my_m[j] = s_vert[j][q];
                            if (j > 0) q = s_par[j][q];
                        }
                    }
                }
            }
            __syncwarp();

            // joined lists; the shortest supplies the candidates
            uint32_t my_deg = kFull, my_off = 0;
            if (uint32_t(lane) < nj) {
                const uint32_t u = my_m[sL.jpos[lane]];
                const uint2 inf = sL.jdir[lane] ? g.in_info[u] : g.out_info[u];
                my_off = inf.x;
                my_deg = inf.y;
                joff[warp][lane] = my_off;
                jdeg[warp][lane] = my_deg;
            }
            uint32_t bd = my_deg, bl = uint32_t(lane);
            #pragma unroll
            for (int s = 16; s; s >>= 1) {
                const uint32_t od = __shfl_xor_sync(kFull, bd, s), ol = __shfl_xor_sync(kFull, bl, s);
                if (od < bd || (od == bd && ol < bl)) { bd = od; bl = ol; }
            }
            if (nj == 0) { __syncwarp(); continue; }  // unreachable for validated orders
            const uint32_t tmin = bl, mdeg = bd;
            const uint32_t moff = __shfl_sync(kFull, my_off, int(tmin));
            __syncwarp();

            if constexpr (MODE == kBytesMode) {
                if (lane == 0) {
                    unsigned long long b = 8;
                    for (uint32_t t = 0; t < nj; ++t) b += 4ull * jdeg[warp][t] + 8;
                    local += b;
                }
                __syncwarp();
                continue;
            }

            // symmetry-breaking window [lo, hi) on the candidate value
            uint32_t lo = 0, hi = kFull;
            for (uint32_t msk = sL.gt_mask; msk; msk &= msk - 1) lo = max(lo, my_m[__ffs(msk) - 1] + 1);
            for (uint32_t msk = sL.lt_mask; msk; msk &= msk - 1) hi = min(hi, my_m[__ffs(msk) - 1]);
            const uint32_t *mlist = g.adj + moff;
            const uint32_t s0 = lo ? lbound(mlist, mdeg, lo) : 0;
            const uint32_t e0 = hi != kFull ? lbound(mlist, mdeg, hi) : mdeg;

            if (MODE == kCountMode && sL.closed_form) {  // uniform branch
                // one joined list, no signature: every list element in the
                // window except the already-matched vertices extends
                if (s0 < e0) {
                    bool hit = false;
                    if (uint32_t(lane) < lvl) {
                        const uint32_t mj = my_m[lane];
                        hit = mj >= lo && mj < hi && contains(mlist, mdeg, mj);
                    }
                    const uint32_t sub = __popc(__ballot_sync(kFull, hit));
                    if (lane == 0) local += (e0 - s0) - sub;
                }
                __syncwarp();
                continue;
            }

            uint32_t ubp = kFull;
            if (need_ub) {
                uint32_t d = kFull;
                if (uint32_t(lane) < sN.nj && sN.jpos[lane] < lvl) {
                    const uint32_t u = my_m[sN.jpos[lane]];
                    d = (sN.jdir[lane] ? g.in_info[u] : g.out_info[u]).y;
                }
                ubp = warp_min(d);
            }

            for (uint32_t x0 = s0; x0 < e0; x0 += 32) {
                const uint32_t x = x0 + lane;
                bool ok = x < e0;
                const uint32_t c = ok ? __ldg(mlist + x) : 0;
                ok = ok && c >= sL.sig_lo;
                if (ok)
                    for (uint32_t j = 0; j < lvl; ++j)
                        if (c == my_m[j]) { ok = false; break; }
                uint2 co = make_uint2(0, 0), ci = make_uint2(0, 0);
                if (ok && load_info) {
                    co = g.out_info[c];
                    ci = sym ? co : g.in_info[c];
                }
                if (ok && check_sig) ok = ci.y >= sL.qin && co.y >= sL.qout;
                if (ok)
                    for (uint32_t t = 0; t < nj; ++t) {
                        if (t == tmin) continue;
                        if (!contains(g.adj + joff[warp][t], jdeg[warp][t], c)) { ok = false; break; }
                    }
                if constexpr (MODE == kCountMode) {
                    local += ok;
                } else {
                    uint32_t ub = ubp;
                    if (ub_out) ub = min(ub, co.y);
                    if (ub_in) ub = min(ub, ci.y);
                    if (store_pos) ub = moff + x;
                    const unsigned m = __ballot_sync(kFull, ok);
                    const uint32_t nn = __popc(m);
                    if (obn + nn > uint32_t(kOutBuf)) flush();
                    if (ok) {
                        const uint32_t r = obn + __popc(m & lanemask_lt);
                        ob_v[warp][r] = c;
                        ob_p[warp][r] = p;
                        ob_u[warp][r] = ub;
                    }
                    obn += nn;
                }
            }
            __syncwarp();
        }
    }
    if constexpr (MODE == kExpand) {
        if (obn) flush();
    } else {
        #pragma unroll
        for (int s = 16; s; s >>= 1) local += __shfl_xor_sync(kFull, local, s);
        if (lane == 0 && local) atomicAdd(acc, local);
    }
}

// ---- levels 1..k-1, flattened form ------------------------------------
// A warp takes up to 32 consecutive parents, one per lane.  Each lane
// rebuilds its parent's partial match (pointer chases of all lanes in flight
// at once), gathers its joined lists and picks the shortest.  The candidate
// lists of the parents are then one concatenated sequence, walked 64
// candidates a step, so all lanes stay busy whether the lists hold 2 or
// 20,000 entries.  The non-empty parents are compacted to ranks and what a
// candidate needs of its owner (where its window lies in the adjacency array,
// the first other list to test, the owner's lane) is one 16-byte record in
// shared memory; the owner of candidate f is the number of windows starting
// at or before f, from one warp-wide OR of the start bits of the step and a
// population count (a binary search over the scan took 5 dependent shuffles,
// and 6 more fetched the record).  Membership in the other lists is a
// one-load table test (in_list) and injectivity is checked after it, on the
// few that pass; a signature on a degree-ranked symmetric graph is a compare
// of ids (sig_lo).  What bounds it: instruction issue where the lists are
// L1/L2 resident, L2 latency otherwise.  Measured against the form with
// galloping searches, a shuffle search for the owner and 32 parents per warp
// always (whole counts): house, 100,000 vertices / 500,000 edges, plain
// 75.5 -> 23.5 ms; 5-cycle, 200,003 / 1M, symmetry breaking 649 -> 347 ms;
// 4-cycle, 10,000 / 40,000 0.252 -> 0.176 ms; a directed four-vertex query,
// 150,001 / 1.5M arcs 6.98 -> 3.43 ms.
constexpr int kFW = 4;    // warps per block
// Turns a warp should get: a parent has at most max_deg candidates, 64 a step,
// so with lists of up to 64 entries all parents cost about the same and one
// turn of total / warps parents each is best (each turn is an atomic on one
// address: with 8 turns the 10,000-vertex 4-cycle took 194 us, not 117); with
// hubs among them one turn each left the 5-cycle's expansions at 19 % of warps
// active (count 344 ms; 8 turns 274 ms, 16 turns 301 ms; a directed query 3.35,
// 2.2 and 3.3 ms).
inline uint32_t flat_turns(uint32_t max_deg) { return std::min(8u, std::max(1u, max_deg / 64)); }
constexpr int kFJ = 8;    // joined lists per level in this form (more: warp-per-parent kernel)

// Words of dynamic shared memory per warp: the parents' matches, their joined
// lists, the owners' records and start offsets, and the staged output.
__host__ __device__ inline uint32_t flat_words(uint32_t lvl, uint32_t nj, bool expand) {
    return 32 * lvl + 64 * nj + 128 + 32 + (expand ? 3 * kOutBuf : 0);
}

// What a counted level counts with it, one instance each: nothing, the last
// level by a plain or an orbit fold, both of a pendant pair, a twin.  One
// instance with all of them behind branches in its inner loop issued three
// times the instructions (3-path, 1M vertices / 10M edges, plain 28 -> 7.7 ms,
// symmetry breaking 0.77 -> 0.28; 3-star above; a directed four-vertex query
// with twins 2.8 -> 1.8).
enum Folded { kNoFold = 0, kPlainFold, kOrbitFold, kPendants, kTwins, kFolds };

// MODE kExpand writes L_lvl (adding its entries' child bounds to *acc where
// acc is given), kCountMode counts, kBytesMode adds the bytes the
// count reads (with any FOLD).
template <int MODE, int FOLD>
__global__ void __launch_bounds__(kFW * 32, FOLD ? 8 : 10)
k_level_flat(DevView g, const RunParams *__restrict__ rp, uint32_t lvl, uint32_t turns, const Parents parents,
             uint32_t *__restrict__ cursor, uint32_t *__restrict__ out_n, uint32_t out_cap,
             uint32_t *__restrict__ err, unsigned long long *__restrict__ acc,
             unsigned long long *__restrict__ acc2, unsigned long long *__restrict__ acc3) {
    uint32_t pa, total;
    parents_of(parents, pa, total);
    if (!total) return;
    __shared__ LevelPlan sL, sN, sN2;
    __shared__ uint32_t *s_vert[kMaxK];
    __shared__ uint32_t *s_par[kMaxK];
    extern __shared__ __align__(16) uint32_t dyn[];
    {
        const uint32_t words = sizeof(LevelPlan) / 4;
        const uint32_t nl = lvl + 1 < rp->plan.k ? lvl + 1 : lvl;
        const uint32_t nl2 = lvl + 2 < rp->plan.k ? lvl + 2 : nl;
        for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) {
            reinterpret_cast<uint32_t *>(&sL)[i] = reinterpret_cast<const uint32_t *>(&rp->plan.lv[lvl])[i];
            reinterpret_cast<uint32_t *>(&sN)[i] = reinterpret_cast<const uint32_t *>(&rp->plan.lv[nl])[i];
            if (FOLD == kPendants) reinterpret_cast<uint32_t *>(&sN2)[i] = reinterpret_cast<const uint32_t *>(&rp->plan.lv[nl2])[i];
        }
        if (threadIdx.x < kMaxK) {
            s_vert[threadIdx.x] = rp->vert[threadIdx.x];
            s_par[threadIdx.x] = rp->par[threadIdx.x];
        }
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t lanemask_lt = (1u << lane) - 1, lanemask_le = lanemask_lt | (1u << lane);
    const bool sym = rp->plan.symmetric != 0;
    const uint32_t nj = sL.nj;
    uint32_t *const wbase = dyn + warp * flat_words(lvl, nj, MODE == kExpand);
    uint4 *const rec = reinterpret_cast<uint4 *>(wbase);      // [rank]: {window base - start, lane | source join << 8,
                                                              //          first other list's offset, its length}
    uint32_t *const starts = wbase + 128;                     // [rank]
    uint32_t *const sm_off = starts + 32;                     // [join][lane]
    uint32_t *const sm_deg = sm_off + 32 * nj;                // [join][lane]
    uint32_t *const sm_m = sm_deg + 32 * nj;                  // [position][lane]
    uint32_t *const ob_v = sm_m + 32 * lvl;                   // staged output (expand)
    uint32_t *const ob_p = ob_v + kOutBuf, *const ob_u = ob_p + kOutBuf;
    // pendant pair: this level (k-3) also counts levels k-2 and k-1
    const uint32_t fold2 = FOLD == kPendants ? sL.fold2 : 0u;
    // twins: this level (k-2) also counts level k-1, from each parent's number
    // of candidates (counted into `starts`' place by the parent's lane)
    const uint32_t twin = FOLD == kTwins ? sL.twin : 0u;
    unsigned long long local3 = 0;
    const bool store_pos = MODE == kExpand && lvl == rp->pos_lvl;
    const bool need_ub = (MODE == kExpand && lvl + 1 < rp->stored) || store_pos;
    uint32_t *out_v = MODE == kExpand ? rp->vert[lvl] : nullptr;
    uint32_t *out_p = MODE == kExpand ? rp->par[lvl] : nullptr;
    uint32_t *out_u = MODE == kExpand ? rp->ub[lvl] : nullptr;
    bool ub_out = false, ub_in = false;
    if (need_ub && !store_pos)
        for (uint32_t t = 0; t < sN.nj; ++t)
            if (sN.jpos[t] == lvl) (sN.jdir[t] ? ub_in : ub_out) = true;
    const bool check_sig = sL.check_sig != 0;
    const uint32_t sig_lo = sL.sig_lo;
    const bool closed = MODE == kCountMode && sL.closed_form;
    // level k-2 counting level k-1 too: each candidate c adds the last
    // level's closed form, |window of L| - matched vertices in it, where L
    // is an earlier vertex's list and c itself is one of the matched
    const bool fold = MODE == kBytesMode ? sL.fold != 0 : FOLD == kPlainFold || FOLD == kOrbitFold;
    const bool fold_guar_c = fold && ((sN.guar_mask >> lvl) & 1u);
    const bool loops = rp->plan.data_loops != 0;
    // parents per warp and turn: fewer than 32 where that would leave a warp
    // fewer than `turns` turns; 32 where no candidates are walked, so that every
    // parent costs the same few loads (an edge, 1M vertices in 4 root slices:
    // 0.22 ms with 8 turns, 0.14 this way; 200,000 in 16: 0.26 and 0.15)
    const uint32_t nturns = turns * gridDim.x * kFW;
    const uint32_t grab = closed || MODE == kBytesMode ? 32u : min(32u, (total + nturns - 1) / nturns);
    const unsigned long long deadline = run_deadline(rp);
    unsigned long long local = 0, local2 = 0;
    uint32_t obn = 0;

    auto flush = [&]() {
        if constexpr (MODE != kExpand) return;
        __syncwarp();
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(out_n, obn);
        base = __shfl_sync(kFullMask, base, 0);
        if (base + obn <= out_cap && base + obn >= base) {
            for (uint32_t i = lane; i < obn; i += 32) {
                out_v[base + i] = ob_v[i];
                out_p[base + i] = ob_p[i];
                if (need_ub) out_u[base + i] = ob_u[i];
            }
        } else if (lane == 0) {
            atomicOr(err, 1u);
        }
        obn = 0;
        __syncwarp();
    };

    while (true) {
        uint32_t start = 0;
        if (lane == 0) start = past_deadline(rp, deadline) ? total : atomicAdd(cursor, grab);
        start = __shfl_sync(kFullMask, start, 0);
        if (start >= total) break;
        const uint32_t p = pa + start + lane;
        const bool have = uint32_t(lane) < grab && start + lane < total;
        // this lane's parent: partial match into column `lane`
        if (have) {
            uint32_t e = p;
            for (int j = int(lvl) - 1; j >= 0; --j) {
                sm_m[32 * j + lane] = s_vert[j][e];
                if (j > 0) e = s_par[j][e];
            }
        }
        // joined lists, shortest first
        uint32_t moff = 0, mdeg = 0, tmin = 0, s0 = 0, e0 = 0, ubp = kFullMask;
        uint32_t f_off = 0, f_deg = 0, f_lo = 0, f_hi = kFullMask, fbase = 0;
        if (have) {
            mdeg = kFullMask;
            for (uint32_t t = 0; t < nj; ++t) {
                const uint32_t u = sm_m[32 * sL.jpos[t] + lane];
                const uint2 inf = sL.jdir[t] ? g.in_info[u] : g.out_info[u];
                sm_off[32 * t + lane] = inf.x;
                sm_deg[32 * t + lane] = inf.y;
                if (inf.y < mdeg) { mdeg = inf.y; moff = inf.x; tmin = t; }
            }
            if (nj == 0) mdeg = 0;
            uint32_t lo = 0, hi = kFullMask;
            for (uint32_t msk = sL.gt_mask; msk; msk &= msk - 1) lo = max(lo, sm_m[32 * (__ffs(msk) - 1) + lane] + 1);
            for (uint32_t msk = sL.lt_mask; msk; msk &= msk - 1) hi = min(hi, sm_m[32 * (__ffs(msk) - 1) + lane]);
            const uint32_t *lst = g.adj + moff;
            const uint32_t mu = nj ? sm_m[32 * sL.jpos[tmin] + lane] : 0;
            const bool mdir = nj && sL.jdir[tmin];
            s0 = lo ? lbound_own(g, mdir, mu, lst, mdeg, lo, loops) : 0;
            e0 = hi != kFullMask ? lbound_own(g, mdir, mu, lst, mdeg, hi, loops) : mdeg;
            if (e0 < s0) e0 = s0;
            if (need_ub)
                for (uint32_t t = 0; t < sN.nj; ++t)
                    if (sN.jpos[t] < lvl) {
                        const uint32_t u = sm_m[32 * sN.jpos[t] + lane];
                        ubp = min(ubp, (sN.jdir[t] ? g.in_info[u] : g.out_info[u]).y);
                    }
            if (MODE == kBytesMode ? fold && sN.ofold : FOLD == kOrbitFold) {
                fbase = orbit_base(g, sN, lvl, loops, [&](uint32_t j) { return sm_m[32 * j + lane]; });
            } else if (fold) {
                const uint32_t u = sm_m[32 * sN.jpos[0] + lane];
                const uint2 inf = sN.jdir[0] ? g.in_info[u] : g.out_info[u];
                f_off = inf.x;
                f_deg = inf.y;
                for (uint32_t msk = sN.gt_mask; msk; msk &= msk - 1) f_lo = max(f_lo, sm_m[32 * (__ffs(msk) - 1) + lane] + 1);
                for (uint32_t msk = sN.lt_mask; msk; msk &= msk - 1) f_hi = min(f_hi, sm_m[32 * (__ffs(msk) - 1) + lane]);
                const uint32_t *fl = g.adj + f_off;
                const uint32_t ws = f_lo ? lbound(fl, f_deg, f_lo) : 0;
                const uint32_t we = f_hi != kFullMask ? lbound(fl, f_deg, f_hi) : f_deg;
                uint32_t sub = 0;
                for (uint32_t j = 0; j < lvl; ++j) {
                    const uint32_t mj = sm_m[32 * j + lane];
                    if (j == sN.jpos[0] && !loops) continue;  // not in its own list
                    if (mj >= f_lo && mj < f_hi && (((sN.guar_mask >> j) & 1u) || in_list(g, f_off, f_deg, mj))) ++sub;
                }
                fbase = (we > ws ? we - ws : 0) - sub;
            }
            if (MODE == kBytesMode) {
                // what this kernel's algorithm reads for the parent: its own
                // and its ancestors' (vertex, parent) entries, the joined
                // vertices' info, then either the closed form's tests or the
                // streamed candidate window plus, per candidate, the signature
                // gather and one membership test per other list
                auto test = [&](uint32_t l) { return g.tab ? 32u : 4u * (32u - __clz(l | 1u)); };
                unsigned long long b = 8ull * lvl + 8ull * nj;
                const uint32_t len = e0 - s0;
                if (sL.closed_form) {  // the count kernel's closed form
                    b += uint64_t(lvl) * test(mdeg);
                } else {
                    uint32_t per = check_sig ? 8 : 0;
                    for (uint32_t t = 0; t < nj; ++t)
                        if (t != tmin) per += test(sm_deg[32 * t + lane]);
                    if (fold) {
                        b += 8 + uint64_t(lvl) * test(f_deg);
                        if (!fold_guar_c) per += test(f_deg);
                    }
                    b += 4ull * len + uint64_t(len) * per;
                }
                local += b;
            }
            if (closed) {
                // one list, no signature: the window minus the matched vertices in it
                uint32_t sub = 0;
                for (uint32_t j = 0; j < lvl; ++j) {
                    const uint32_t mj = sm_m[32 * j + lane];
                    if (j == sL.jpos[0] && !loops) continue;  // not in its own list
                    if (mj >= lo && mj < hi && (((sL.guar_mask >> j) & 1u) || in_list(g, moff, mdeg, mj))) ++sub;
                }
                local += (e0 - s0) - sub;
            }
        }
        if (MODE == kBytesMode || closed) continue;
        // concatenated candidate sequence of the parents; the non-empty ones
        // by rank
        const uint32_t len = e0 - s0;
        uint32_t incl = len;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t ftotal = __shfl_sync(kFullMask, incl, 31);
        if (!ftotal) { __syncwarp(); continue; }
        const unsigned live = __ballot_sync(kFullMask, len != 0);
        if (len) {
            const uint32_t r = __popc(live & lanemask_lt), excl = incl - len, to = tmin ? 0u : 1u;
            const uint32_t oo = nj > 1 ? sm_off[32 * to + lane] : 0u, od = nj > 1 ? sm_deg[32 * to + lane] : 0u;
            rec[r] = make_uint4(moff + s0 - excl, uint32_t(lane) | (tmin << 8), oo, od);
            starts[r] = excl;
        }
        __syncwarp();
        const uint32_t my_start = uint32_t(lane) < uint32_t(__popc(live)) ? starts[lane] : kFullMask;
        if (FOLD == kTwins) {
            __syncwarp();
            starts[lane] = 0;  // from here on: candidates of the lane's parent
            __syncwarp();
        }
        uint32_t started = 0;  // windows that start before this step
        for (uint32_t fstep = 0; fstep < ftotal; fstep += 64) {
            // two candidates per lane, their loads in flight together
            uint4 rc[2];
            uint32_t cv[2];
            bool okv[2];
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t rel = my_start - (fstep + 32 * h);
                const uint32_t bits = __reduce_or_sync(kFullMask, rel < 32u ? 1u << rel : 0u);
                const uint32_t own = started + __popc(bits & lanemask_le) - 1;
                started += __popc(bits);
                const uint32_t f = fstep + 32 * h + lane;
                okv[h] = f < ftotal;
                rc[h] = rec[own];
                cv[h] = __ldg(g.adj + (rc[h].x + min(f, ftotal - 1)));  // the base may lie below zero: 32-bit sum
            }
            if (nj > 1) {
                if (g.tab) {
                    uint32_t nb[2], b[2];
                    Bucket bk[2];
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        nb[h] = (rc[h].w + 3) >> 2;
                        b[h] = tab_bucket(nb[h], cv[h]);
                        bk[h] = load_bucket(g.tab, rc[h].z, b[h]);
                    }
                    #pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (okv[h] && !bucket_has(bk[h], cv[h]))
                            okv[h] = tab_continue(g.tab, rc[h].z, nb[h], b[h], bk[h], cv[h]);
                } else {
                    #pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (okv[h]) okv[h] = contains(g.adj + rc[h].z, rc[h].w, cv[h]);
                }
            }
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (fstep + 32 * h >= ftotal) break;
                bool ok = okv[h];
                const uint32_t c = cv[h], owner = rc[h].y & 255u, o_tmin = rc[h].y >> 8;
                if (ok && nj > 2)
                    for (uint32_t t = (o_tmin < 2 ? 2u : 1u); t < nj; ++t)
                        if (t != o_tmin && !in_list(g, sm_off[32 * t + owner], sm_deg[32 * t + owner], c)) {
                            ok = false;
                            break;
                        }
                ok = ok && c >= sig_lo;
                if (ok)
                    for (uint32_t j = 0; j < lvl; ++j)
                        if (c == sm_m[32 * j + owner]) { ok = false; break; }
                uint2 co = make_uint2(0, 0), ci = make_uint2(0, 0);
                if (ok && (check_sig || ub_out || ub_in)) {
                    co = g.out_info[c];
                    ci = sym ? co : g.in_info[c];
                    if (check_sig) ok = ci.y >= sL.qin && co.y >= sL.qout;
                }
                if constexpr (MODE == kCountMode) {
                    if constexpr (FOLD == kTwins) {
                        // lanes of one parent are neighbours: the first of them adds
                        const unsigned m = __ballot_sync(kFullMask, ok);
                        const uint32_t up = __shfl_up_sync(kFullMask, owner, 1);
                        const bool head = lane == 0 || up != owner;
                        const unsigned heads = __ballot_sync(kFullMask, head);
                        const unsigned next = heads & ~lanemask_le;
                        const unsigned seg = (next ? (1u << (__ffs(next) - 1)) - 1u : kFullMask) & ~lanemask_lt;
                        if (head) starts[owner] += __popc(m & seg);
                        __syncwarp();
                    } else if constexpr (FOLD == kPendants) {
                        if (ok) {
                            const uint64_t p2 = pendant_pairs(g, sN, sN2, fold2, lvl, loops,
                                [&](uint32_t j) { return j == lvl ? c : sm_m[32 * j + owner]; }, local3);
                            local += p2;
                            ++local2;
                        }
                    } else if constexpr (FOLD == kOrbitFold) {
                        const uint32_t o_fbase = __shfl_sync(kFullMask, fbase, int(owner));
                        if (ok) {
                            local += orbit_weight(g, sN, lvl, o_fbase, c, loops);
                            ++local2;
                        }
                    } else if constexpr (FOLD == kPlainFold) {
                        const uint32_t o_fbase = __shfl_sync(kFullMask, fbase, int(owner));
                        const uint32_t o_foff = __shfl_sync(kFullMask, f_off, int(owner));
                        const uint32_t o_fdeg = __shfl_sync(kFullMask, f_deg, int(owner));
                        const uint32_t o_flo = __shfl_sync(kFullMask, f_lo, int(owner));
                        const uint32_t o_fhi = __shfl_sync(kFullMask, f_hi, int(owner));
                        if (ok) {
                            const bool hit = c >= o_flo && c < o_fhi &&
                                             (fold_guar_c || in_list(g, o_foff, o_fdeg, c));
                            local += o_fbase - (hit ? 1u : 0u);
                            ++local2;
                        }
                    } else {
                        local += ok;
                    }
                } else {
                    uint32_t ub = need_ub ? __shfl_sync(kFullMask, ubp, int(owner)) : 0u;
                    if (ub_out) ub = min(ub, co.y);
                    if (ub_in) ub = min(ub, ci.y);
                    // where c sits in the list it came from
                    if (store_pos) ub = rc[h].x + fstep + 32 * h + lane;
                    const unsigned m = __ballot_sync(kFullMask, ok);
                    const uint32_t nn = __popc(m);
                    if (obn + nn > uint32_t(kOutBuf)) flush();
                    if (ok) {
                        const uint32_t r = obn + __popc(m & lanemask_lt);
                        ob_v[r] = c;
                        ob_p[r] = pa + start + owner;
                        ob_u[r] = ub;
                        local += ub;
                    }
                    obn += nn;
                }
            }
        }
        __syncwarp();
        if (FOLD == kTwins && have && len) {
            const unsigned long long n = starts[lane], pr = n ? n * (n - 1) : 0;
            local2 += n;
            local += twin == 2 ? pr / 2 : pr;
        }
        __syncwarp();
    }
    if constexpr (MODE == kExpand) {
        if (obn) flush();
        if (acc && need_ub && !store_pos) {
            #pragma unroll
            for (int s = 16; s; s >>= 1) local += __shfl_xor_sync(kFullMask, local, s);
            if (lane == 0 && local) atomicAdd(acc, local);
        }
    } else {
        #pragma unroll
        for (int s = 16; s; s >>= 1) {
            local += __shfl_xor_sync(kFullMask, local, s);
            local2 += __shfl_xor_sync(kFullMask, local2, s);
            local3 += __shfl_xor_sync(kFullMask, local3, s);
        }
        if (lane == 0 && local) atomicAdd(acc, local);
        if (lane == 0 && local2 && acc2) atomicAdd(acc2, local2);
        if (lane == 0 && local3 && acc3) atomicAdd(acc3, local3);
    }
}

// ---- fused count of levels p and c = p + 1 ---------------------------
// When the plan fuses the counted level c with p = c - 1, c's candidates for
// a vertex s chosen at p are the members t of p's candidate set S (same
// parent) that lie in s's list.  One warp per parent at level p - 1: build S
// once (the usual scan of the shortest joined list, membership in the
// others, ballot compaction) into the warp's scratch row, then intersect S
// with the list of every s in S, 32 vertices s at a time (one per lane), and
// count (or, for a folded c, add the last level's closed form per t).
// Level p is never written to the trie.
//
// The work of one parent grows like |S|^2, so a hub parent would keep one
// warp busy long after the others finish.  Phase 1 therefore defers every
// parent with |S| > kBigS: it copies S into a pool and records the parent;
// phase 2 (a second launch, after a one-block scan of the deferred parents'
// group counts) hands out their groups of 32 vertices s to all warps.
constexpr int kZW = 4;          // warps per block
constexpr uint32_t kBigS = 256;  // default |S| above which a parent is split

// Parents deferred by phase 1 and their saved candidate sets.
struct FusedBig {
    unsigned long long *n;  // [0] entries appended, [1] pool words taken
    uint32_t *gi;           // parent index (in L_{p-1}) of each entry
    uint32_t *soff;         // offset of its S in the pool
    uint32_t *ns;           // |S|
    uint32_t *pref;         // inclusive prefix sum of groups of 32 (phase 2)
    uint32_t *pool;
    uint32_t cap;
    unsigned long long pool_words;
};

// 12 resident blocks (48 warps) per SM at 40 registers: the kernel waits on
// dependent L2 loads, and the extra warps outweigh the spills that cap costs.
template <int MODE>
__global__ void __launch_bounds__(kZW * 32, 12)
k_fused(DevView g, const RunParams *__restrict__ rp, uint32_t p, const Parents parents, uint32_t phase,
        uint32_t split, uint32_t *__restrict__ cursor, uint32_t *__restrict__ scratch, uint32_t stride, FusedBig big,
        unsigned long long *__restrict__ acc, unsigned long long *__restrict__ acc_c,
        unsigned long long *__restrict__ acc_p) {
    uint32_t pa, total;
    parents_of(parents, pa, total);
    if (!total) return;
    __shared__ LevelPlan sP, sC, sF;
    __shared__ uint32_t *s_vert[kMaxK];
    __shared__ uint32_t *s_par[kMaxK];
    __shared__ uint32_t wm[kZW][kMaxK];
    __shared__ uint32_t joff[kZW][kMaxJ], jdeg[kZW][kMaxJ], jver[kZW][kMaxJ];
    __shared__ uint32_t xoff[kZW][kMaxJ], xdeg[kZW][kMaxJ];
    {
        const uint32_t words = sizeof(LevelPlan) / 4;
        const uint32_t c = p + 1;
        const uint32_t f = c + 1 < rp->plan.k ? c + 1 : c;
        const uint32_t *a = reinterpret_cast<const uint32_t *>(&rp->plan.lv[p]);
        const uint32_t *b = reinterpret_cast<const uint32_t *>(&rp->plan.lv[c]);
        const uint32_t *d = reinterpret_cast<const uint32_t *>(&rp->plan.lv[f]);
        for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) {
            reinterpret_cast<uint32_t *>(&sP)[i] = a[i];
            reinterpret_cast<uint32_t *>(&sC)[i] = b[i];
            reinterpret_cast<uint32_t *>(&sF)[i] = d[i];
        }
        if (threadIdx.x < kMaxK) {
            s_vert[threadIdx.x] = rp->vert[threadIdx.x];
            s_par[threadIdx.x] = rp->par[threadIdx.x];
        }
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t lanemask_lt = (1u << lane) - 1;
    uint32_t *my_m = wm[warp];
    uint32_t *const row = scratch + size_t(blockIdx.x * kZW + warp) * stride;

    const uint32_t c = p + 1;
    // the counted level c is folded when level c carries the fold flag
    const bool cfold = sC.fold != 0;
    const uint32_t tp = sC.fuse_tp;
    const uint32_t extra = sC.fuse_extra;
    const bool sig_c = sC.check_sig && (sC.qin > sP.qin || sC.qout > sP.qout);
    const uint32_t below = (1u << p) - 1;
    const bool c_gt_s = (sC.gt_mask >> p) & 1u, c_lt_s = (sC.lt_mask >> p) & 1u;
    const bool fguar_t = cfold && ((sF.guar_mask >> c) & 1u);
    const bool loops = rp->plan.data_loops != 0;
    // an extra list of c on position p itself changes with s: per-s loop
    bool extra_on_p = false;
    for (uint32_t t = 0; t < sC.nj; ++t)
        if (((extra >> t) & 1u) && sC.jpos[t] == p) extra_on_p = true;
    unsigned long long local = 0, local_c = 0, local_p = 0;
    uint32_t cached_q = kFullMask;
    const bool phase2 = phase == 2;
    uint32_t nbig = 0;
    if (phase2) {
        const unsigned long long n0 = big.n[0];
        nbig = n0 < big.cap ? uint32_t(n0) : big.cap;
        total = nbig ? big.pref[nbig - 1] : 0;
    }
    const unsigned long long deadline = run_deadline(rp);
    auto probes = [](uint32_t len) { return 32u - __clz(len | 1u); };

    // level c for the vertices s = S[i0 .. i0+32) of one parent
    auto group = [&](const uint32_t *S, uint32_t ns, uint32_t i0, uint32_t lo_c, uint32_t hi_c) {
        if (!extra_on_p) {
            // one s per lane; the 32 (s, t) sequences are concatenated and
            // spread over all lanes, as in k_level_flat
            const uint32_t i = i0 + lane;
            // the iterated range starts at itb (in S when iters, else in the
            // adjacency array); the probed one is [ostart, oend) of S or of
            // the list at ooff
            uint32_t sv = kFullMask, itb = 0, ooff = 0, ostart = 0, oend = 0, nit = 0, iters = 1;
            uint32_t fbase = 0, foff = 0, fdeg = 0, flo = 0, fhi = kFullMask;
            if (i < ns) {
                sv = S[i];
                const uint2 is = sC.jdir[tp] ? g.in_info[sv] : g.out_info[sv];
                const uint32_t lsoff = is.x, ds = is.y;
                uint32_t lo_t = lo_c, hi_t = hi_c;
                if (c_gt_s) lo_t = max(lo_t, sv + 1);
                if (c_lt_s) hi_t = min(hi_t, sv);
                const uint32_t ts = lo_t ? lbound(S, ns, lo_t) : 0;
                const uint32_t te = hi_t != kFullMask ? lbound(S, ns, hi_t) : ns;
                const uint32_t *Ls = g.adj + lsoff;
                const bool sdir = sC.jdir[tp] != 0;
                const uint32_t ls0 = lo_t ? lbound_own(g, sdir, sv, Ls, ds, lo_t, loops) : 0;
                const uint32_t ls1 = hi_t != kFullMask ? lbound_own(g, sdir, sv, Ls, ds, hi_t, loops) : ds;
                const uint32_t nS = te > ts ? te - ts : 0, nL = ls1 > ls0 ? ls1 - ls0 : 0;
                iters = nS <= nL ? 1u : 0u;  // iterate the shorter side
                nit = iters ? nS : nL;
                itb = iters ? ts : lsoff + ls0;
                ooff = iters ? lsoff : 0;
                ostart = iters ? ls0 : ts;
                oend = iters ? ls1 : te;
                if (cfold && sF.ofold) {
                    fbase = orbit_base(g, sF, p + 1, loops, [&](uint32_t j) { return j == p ? sv : my_m[j]; });
                } else if (cfold) {
                    // folded last level: f_base(s) = |window of L_F| - matched in it
                    const uint32_t jf = sF.jpos[0];
                    const uint32_t u = jf == p ? sv : my_m[jf];
                    const uint2 inf = sF.jdir[0] ? g.in_info[u] : g.out_info[u];
                    foff = inf.x;
                    fdeg = inf.y;
                    for (uint32_t msk = sF.gt_mask; msk; msk &= msk - 1) {
                        const uint32_t j = __ffs(msk) - 1;
                        flo = max(flo, (j == p ? sv : my_m[j]) + 1);
                    }
                    for (uint32_t msk = sF.lt_mask; msk; msk &= msk - 1) {
                        const uint32_t j = __ffs(msk) - 1;
                        fhi = min(fhi, j == p ? sv : my_m[j]);
                    }
                    const uint32_t *fl = g.adj + foff;
                    const uint32_t ws = flo ? lbound(fl, fdeg, flo) : 0;
                    const uint32_t we = fhi != kFullMask ? lbound(fl, fdeg, fhi) : fdeg;
                    uint32_t sub = 0;
                    for (uint32_t j = 0; j <= p; ++j) {
                        const uint32_t mj = j == p ? sv : my_m[j];
                        if (mj >= flo && mj < fhi && (((sF.guar_mask >> j) & 1u) || contains(fl, fdeg, mj))) ++sub;
                    }
                    fbase = (we > ws ? we - ws : 0) - sub;
                }
                if (MODE == kBytesMode) {
                    const unsigned long long by = 12 + 4ull * nit + uint64_t(nit) * 4 * probes(iters ? ds : nS) +
                                                  (sig_c ? 8ull * nit : 0) +
                                                  (cfold ? 8 + 4ull * (p + 1) * probes(fdeg) : 0);
                    local += by;
                }
            }
            if (MODE == kBytesMode) return;
            uint32_t incl = nit;
            #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
                if (lane >= o) incl += y;
            }
            const uint32_t ftotal = __shfl_sync(kFullMask, incl, 31);
            const uint32_t excl = incl - nit;
            uint32_t gal_owner = kFullMask, gal = 0;
            for (uint32_t fstep = 0; fstep < ftotal; fstep += 32) {
                const uint32_t f = fstep + lane;
                uint32_t owner = 0;
                #pragma unroll
                for (int step = 16; step; step >>= 1) {
                    const uint32_t probe = __shfl_sync(kFullMask, incl, int(owner + step - 1));
                    if (probe <= f) owner += step;
                }
                owner = min(owner, 31u);
                const int ow = int(owner);
                const uint32_t o_excl = __shfl_sync(kFullMask, excl, ow);
                const uint32_t o_sv = __shfl_sync(kFullMask, sv, ow);
                const uint32_t o_itb = __shfl_sync(kFullMask, itb, ow);
                const uint32_t o_ooff = __shfl_sync(kFullMask, ooff, ow);
                const uint32_t o_ostart = __shfl_sync(kFullMask, ostart, ow);
                const uint32_t o_oend = __shfl_sync(kFullMask, oend, ow);
                const uint32_t o_iters = __shfl_sync(kFullMask, iters, ow);
                uint32_t o_fbase = 0, o_foff = 0, o_fdeg = 0, o_flo = 0, o_fhi = 0;
                if (cfold) o_fbase = __shfl_sync(kFullMask, fbase, ow);
                if (cfold && !sF.ofold) {  // the plain fold's list and window
                    o_foff = __shfl_sync(kFullMask, foff, ow);
                    o_fdeg = __shfl_sync(kFullMask, fdeg, ow);
                    o_flo = __shfl_sync(kFullMask, flo, ow);
                    o_fhi = __shfl_sync(kFullMask, fhi, ow);
                }
                bool ok = f < ftotal;
                if (owner != gal_owner) {
                    gal_owner = owner;
                    gal = o_ostart;
                }
                uint32_t t = 0;
                if (ok) {
                    const uint32_t y = f - o_excl;
                    if (o_iters) {
                        t = S[o_itb + y];
                        const uint32_t *Lo = g.adj + o_ooff;
                        const uint32_t pos = lbound_from(Lo, o_oend, gal, t);
                        gal = pos;
                        ok = pos < o_oend && __ldg(Lo + pos) == t;
                    } else {
                        t = __ldg(g.adj + o_itb + y);
                        const uint32_t pos = lbound_from(S, o_oend, gal, t);
                        gal = pos;
                        ok = pos < o_oend && S[pos] == t;
                    }
                }
                if (ok && t == o_sv) ok = false;
                if (ok && extra)
                    for (uint32_t tt = 0; tt < sC.nj; ++tt)
                        if ((extra >> tt) & 1u)
                            if (!contains(g.adj + xoff[warp][tt], xdeg[warp][tt], t)) { ok = false; break; }
                ok = ok && t >= sC.sig_lo;
                if (ok && sig_c) {
                    const uint2 o = g.out_info[t], i2 = g.in_info[t];
                    ok = i2.y >= sC.qin && o.y >= sC.qout;
                }
                if (ok) {
                    ++local_c;
                    if (cfold && sF.ofold) {
                        local += orbit_weight(g, sF, c, o_fbase, t, loops);
                    } else if (cfold) {
                        const bool h = t >= o_flo && t < o_fhi && (fguar_t || contains(g.adj + o_foff, o_fdeg, t));
                        local += o_fbase - (h ? 1u : 0u);
                    } else {
                        ++local;
                    }
                }
            }
            __syncwarp();
            return;
        }
        // a list of c on p itself: one s at a time, lane-parallel over t
        const uint32_t iend = min(i0 + 32, ns);
        for (uint32_t i = i0; i < iend; ++i) {
            const uint32_t sv = S[i];
            const uint2 is = sC.jdir[tp] ? g.in_info[sv] : g.out_info[sv];
            const uint32_t *Ls = g.adj + is.x;
            const uint32_t ds = is.y;
            uint32_t lo_t = lo_c, hi_t = hi_c;
            if (c_gt_s) lo_t = max(lo_t, sv + 1);
            if (c_lt_s) hi_t = min(hi_t, sv);
            const uint32_t ts = lo_t ? lbound(S, ns, lo_t) : 0;
            const uint32_t te = hi_t != kFullMask ? lbound(S, ns, hi_t) : ns;
            if (ts >= te) continue;
            __syncwarp();
            if (uint32_t(lane) < sC.nj && ((extra >> lane) & 1u) && sC.jpos[lane] == p) {
                const uint2 inf = sC.jdir[lane] ? g.in_info[sv] : g.out_info[sv];
                xoff[warp][lane] = inf.x;
                xdeg[warp][lane] = inf.y;
            }
            uint32_t fbase = 0, fdeg = 0, flo = 0, fhi = kFullMask;
            const uint32_t *fl = nullptr;
            if (cfold && sF.ofold) {
                fbase = orbit_base(g, sF, p + 1, loops, [&](uint32_t j) { return j == p ? sv : my_m[j]; });
            } else if (cfold) {
                const uint32_t jf = sF.jpos[0];
                const uint32_t u = jf == p ? sv : my_m[jf];
                const uint2 inf = sF.jdir[0] ? g.in_info[u] : g.out_info[u];
                fl = g.adj + inf.x;
                fdeg = inf.y;
                for (uint32_t msk = sF.gt_mask; msk; msk &= msk - 1) {
                    const uint32_t j = __ffs(msk) - 1;
                    flo = max(flo, (j == p ? sv : my_m[j]) + 1);
                }
                for (uint32_t msk = sF.lt_mask; msk; msk &= msk - 1) {
                    const uint32_t j = __ffs(msk) - 1;
                    fhi = min(fhi, j == p ? sv : my_m[j]);
                }
                const uint32_t ws = flo ? lbound(fl, fdeg, flo) : 0;
                const uint32_t we = fhi != kFullMask ? lbound(fl, fdeg, fhi) : fdeg;
                bool hit = false;
                if (uint32_t(lane) <= p) {
                    const uint32_t mj = uint32_t(lane) == p ? sv : my_m[lane];
                    hit = mj >= flo && mj < fhi && (((sF.guar_mask >> lane) & 1u) || contains(fl, fdeg, mj));
                }
                fbase = (we > ws ? we - ws : 0) - __popc(__ballot_sync(kFullMask, hit));
            }
            __syncwarp();
            const uint32_t ls0 = lo_t ? lbound(Ls, ds, lo_t) : 0;
            const uint32_t ls1 = hi_t != kFullMask ? lbound(Ls, ds, hi_t) : ds;
            const uint32_t nS = te - ts, nL = ls1 > ls0 ? ls1 - ls0 : 0;
            const bool iterS = nS <= nL;
            const uint32_t nit = iterS ? nS : nL;
            if (MODE == kBytesMode) {
                const unsigned long long by = 12 + 4ull * nit + uint64_t(nit) * 4 * probes(iterS ? ds : nS) +
                                              (sig_c ? 8ull * nit : 0) + (cfold ? 8 + 4ull * (p + 1) * probes(fdeg) : 0);
                if (lane == 0) local += by;
                continue;
            }
            uint32_t gal = iterS ? ls0 : ts;
            for (uint32_t y0 = 0; y0 < nit; y0 += 32) {
                const uint32_t y = y0 + lane;
                bool ok = y < nit;
                uint32_t t = 0;
                if (ok) {
                    if (iterS) {
                        t = S[ts + y];
                        const uint32_t pos = lbound_from(Ls, ls1, gal, t);
                        gal = pos;
                        ok = pos < ls1 && __ldg(Ls + pos) == t;
                    } else {
                        t = __ldg(Ls + ls0 + y);
                        const uint32_t pos = lbound_from(S, te, gal, t);
                        gal = pos;
                        ok = pos < te && S[pos] == t;
                    }
                }
                if (ok && t == sv) ok = false;
                if (ok && extra)
                    for (uint32_t tt = 0; tt < sC.nj; ++tt)
                        if ((extra >> tt) & 1u)
                            if (!contains(g.adj + xoff[warp][tt], xdeg[warp][tt], t)) { ok = false; break; }
                ok = ok && t >= sC.sig_lo;
                if (ok && sig_c) {
                    const uint2 o = g.out_info[t], i2 = g.in_info[t];
                    ok = i2.y >= sC.qin && o.y >= sC.qout;
                }
                if (ok) {
                    ++local_c;
                    if (cfold && sF.ofold) {
                        local += orbit_weight(g, sF, c, fbase, t, loops);
                    } else if (cfold) {
                        const bool h = t >= flo && t < fhi && (fguar_t || contains(fl, fdeg, t));
                        local += fbase - (h ? 1u : 0u);
                    } else {
                        ++local;
                    }
                }
            }
        }
        __syncwarp();
    };

    while (true) {
        uint32_t gi = 0;
        if (lane == 0) gi = past_deadline(rp, deadline) ? total : atomicAdd(cursor, 1u);
        gi = __shfl_sync(kFullMask, gi, 0);
        if (gi >= total) break;
        // phase 2: work item gi is group grp of deferred parent b
        uint32_t q0, b = 0, grp = 0;
        if (!phase2) {
            q0 = pa + gi;
        } else {
            uint32_t lo = 0, hi = nbig - 1;  // first b with pref[b] > gi
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (big.pref[mid] > gi) hi = mid; else lo = mid + 1;
            }
            b = lo;
            grp = gi - (b ? big.pref[b - 1] : 0);
            q0 = big.gi[b];
        }
        if (lane == 0) {  // matched vertices of the parent at level p-1
            my_m[p - 1] = s_vert[p - 1][q0];
            if (p >= 2) {
                uint32_t q = s_par[p - 1][q0];
                if (q != cached_q) {
                    cached_q = q;
                    for (int j = int(p) - 2; j >= 0; --j) {
                        my_m[j] = s_vert[j][q];
                        if (j > 0) q = s_par[j][q];
                    }
                }
            }
        }
        __syncwarp();
        const uint32_t *S = row;
        uint32_t ns = 0;
        if (!phase2) {
            // level p: joined lists, the shortest supplies S
            const uint32_t njp = sP.nj;
            uint32_t md = kFullMask, mo = 0;
            if (uint32_t(lane) < njp) {
                const uint32_t u = my_m[sP.jpos[lane]];
                const uint2 inf = sP.jdir[lane] ? g.in_info[u] : g.out_info[u];
                mo = inf.x;
                md = inf.y;
                joff[warp][lane] = mo;
                jdeg[warp][lane] = md;
                jver[warp][lane] = u;
            }
            uint32_t bd = md, bl = uint32_t(lane);
            #pragma unroll
            for (int o = 16; o; o >>= 1) {
                const uint32_t od = __shfl_xor_sync(kFullMask, bd, o), ol = __shfl_xor_sync(kFullMask, bl, o);
                if (od < bd || (od == bd && ol < bl)) { bd = od; bl = ol; }
            }
            const uint32_t moff = __shfl_sync(kFullMask, mo, int(bl)), mdeg = njp ? bd : 0, tmin = bl;
            __syncwarp();
            uint32_t lo = 0, hi = kFullMask;
            for (uint32_t msk = sP.gt_mask; msk; msk &= msk - 1) lo = max(lo, my_m[__ffs(msk) - 1] + 1);
            for (uint32_t msk = sP.lt_mask; msk; msk &= msk - 1) hi = min(hi, my_m[__ffs(msk) - 1]);
            const uint32_t *mlist = g.adj + moff;
            const uint32_t mu = njp ? my_m[sP.jpos[tmin]] : 0;  // the vertex whose list supplies S
            const bool mdir = njp && sP.jdir[tmin];
            uint32_t s0 = kFullMask;
            if (lo && p >= 2 && rp->pos_lvl == p - 1 && lo == my_m[p - 1] + 1) {
                // the window starts right after the parent's own vertex: when
                // that vertex was drawn from this very list, its offset is known
                const uint32_t apos = rp->ub[p - 1][q0];
                if (apos >= moff && apos - moff < mdeg) s0 = apos - moff + 1;
            }
            if (s0 == kFullMask) s0 = lo ? lbound_own(g, mdir, mu, mlist, mdeg, lo, loops) : 0;
            const uint32_t e0 = hi != kFullMask ? lbound_own(g, mdir, mu, mlist, mdeg, hi, loops) : mdeg;
            // this lane's candidates rise, so its lower bounds in the first
            // two other lists rise too: gallop from the last
            uint32_t gp0 = 0, gp1 = 0;
            for (uint32_t x0 = s0; x0 < e0; x0 += 32) {
                const uint32_t x = x0 + lane;
                bool ok = x < e0;
                const uint32_t v = ok ? __ldg(mlist + x) : 0;
                if (ok)
                    for (uint32_t j = 0; j < p; ++j)
                        if (v == my_m[j]) { ok = false; break; }
                ok = ok && v >= sP.sig_lo;
                if (ok && sP.check_sig) {
                    const uint2 o = g.out_info[v], i = g.in_info[v];
                    ok = i.y >= sP.qin && o.y >= sP.qout;
                }
                if (ok) {
                    uint32_t r = 0;
                    for (uint32_t t = 0; t < njp; ++t) {
                        if (t == tmin) continue;
                        const uint32_t *lst = g.adj + joff[warp][t];
                        const uint32_t len2 = jdeg[warp][t];
                        const uint32_t ut = jver[warp][t];
                        if (g.core_bits && ut >= g.core0 && v >= g.core0) {
                            // both in the dense core: one bit of ut's row
                            const uint32_t bi = v - g.core0;
                            const uint32_t w = __ldg(g.core_bits + size_t(ut - g.core0) * (kCore / 32) + (bi >> 5));
                            if (!((w >> (bi & 31)) & 1u)) { ok = false; break; }
                            continue;
                        }
                        if (r < 2) {
                            const uint32_t pos = lbound_from(lst, len2, r == 0 ? gp0 : gp1, v);
                            if (r == 0) gp0 = pos; else gp1 = pos;
                            if (pos >= len2 || __ldg(lst + pos) != v) { ok = false; break; }
                        } else if (!contains(lst, len2, v)) {
                            ok = false;
                            break;
                        }
                        ++r;
                    }
                }
                const unsigned m = __ballot_sync(kFullMask, ok);
                if (ok) {
                    const uint32_t idx = ns + __popc(m & lanemask_lt);
                    row[idx] = v;
                }
                ns += __popc(m);
                if (MODE == kBytesMode && lane == 0) {
                    uint32_t per = sP.check_sig ? 8 : 0;
                    for (uint32_t t = 0; t < njp; ++t)
                        if (t != tmin) per += 4 * probes(jdeg[warp][t]);
                    const unsigned long long by = 4ull * min(32u, e0 - x0) + uint64_t(min(32u, e0 - x0)) * per;
                    local += by;
                }
            }
            __syncwarp();
            if (MODE == kCountMode && ns > split) {
                // defer: save S in the pool for phase 2 (or keep it here when full)
                unsigned long long off = 0;
                uint32_t e = kFullMask;
                if (lane == 0 && big.n[1] < big.pool_words) {
                    off = atomicAdd(&big.n[1], (unsigned long long)ns);
                    if (off + ns <= big.pool_words) {
                        const unsigned long long e64 = atomicAdd(&big.n[0], 1ull);
                        if (e64 < big.cap) e = uint32_t(e64);
                    }
                }
                e = __shfl_sync(kFullMask, e, 0);
                off = __shfl_sync(kFullMask, off, 0);
                if (e != kFullMask) {
                    for (uint32_t i = lane; i < ns; i += 32) big.pool[off + i] = row[i];
                    if (lane == 0) {
                        big.gi[e] = q0;
                        big.soff[e] = uint32_t(off);
                        big.ns[e] = ns;
                    }
                    __syncwarp();
                    continue;
                }
            }
            if (lane == 0) {
                local_p += ns;
                if (MODE == kBytesMode) local += 8ull * p + 8ull * njp + 4ull * ns;
            }
        } else {
            S = big.pool + big.soff[b];
            ns = big.ns[b];
            if (lane == 0 && grp == 0) local_p += ns;
        }
        // extra lists of level c on positions below p: fixed for this parent
        if (uint32_t(lane) < sC.nj && ((extra >> lane) & 1u) && sC.jpos[lane] < p) {
            const uint32_t u = my_m[sC.jpos[lane]];
            const uint2 inf = sC.jdir[lane] ? g.in_info[u] : g.out_info[u];
            xoff[warp][lane] = inf.x;
            xdeg[warp][lane] = inf.y;
        }
        __syncwarp();
        // level c over the vertices s of S
        uint32_t lo_c = 0, hi_c = kFullMask;
        for (uint32_t msk = sC.gt_mask & below; msk; msk &= msk - 1) lo_c = max(lo_c, my_m[__ffs(msk) - 1] + 1);
        for (uint32_t msk = sC.lt_mask & below; msk; msk &= msk - 1) hi_c = min(hi_c, my_m[__ffs(msk) - 1]);
        if (!phase2) {
            for (uint32_t i0 = 0; i0 < ns; i0 += 32) group(S, ns, i0, lo_c, hi_c);
        } else {
            group(S, ns, grp * 32, lo_c, hi_c);
        }
    }
    #pragma unroll
    for (int o = 16; o; o >>= 1) {
        local += __shfl_xor_sync(kFullMask, local, o);
        local_c += __shfl_xor_sync(kFullMask, local_c, o);
    }
    if (lane == 0) {
        if (local) atomicAdd(acc, local);
        if (MODE == kCountMode) {
            if (local_c) atomicAdd(acc_c, local_c);
            if (local_p) atomicAdd(acc_p, local_p);
        }
    }
}

// Inclusive prefix sum of the deferred parents' work items, ceil(len / per)
// each (one block).
__global__ void __launch_bounds__(1024)
k_fused_scan(const unsigned long long *__restrict__ nb, uint32_t cap, const uint32_t *__restrict__ len, uint32_t per,
             uint32_t *__restrict__ pref) {
    __shared__ uint32_t wsum[32];
    __shared__ uint32_t carry;
    const unsigned long long n0 = nb[0];
    const uint32_t n = n0 < cap ? uint32_t(n0) : cap;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (uint32_t base = 0; base < n; base += blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        uint32_t v = i < n ? (len[i] + per - 1) / per : 0, x = v;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFullMask, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        if (w == 0) {
            uint32_t s = lane < int(blockDim.x / 32) ? wsum[lane] : 0;
            #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFullMask, s, o);
                if (lane >= o) s += y;
            }
            wsum[lane] = s;
        }
        __syncthreads();
        const uint32_t pre = carry + (w ? wsum[w - 1] : 0) + x;
        if (i < n) pref[i] = pre;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = pre;
        __syncthreads();
    }
}

// ---- fused count on symmetric graphs: pairs of a candidate set ----------
// With p and c = p + 1 fused, level c is every pair (s, t) of one parent's
// candidate set S (level p) with t in s's list.  On a symmetric graph the pairs
// are unordered: each {a < b} of S with b in a's list is
// found once and counted for s = a, t = b and for s = b, t = a, as far as the
// plan's order between p and c and t's own tests (window, extra lists,
// signature: `adm`) allow.  A pair's weight is A(s) + B(t) (1 + 0 without a
// fold; see pair_a / pair_b).
//
// A warp takes up to 32 parents, one per lane, so the fixed chain per parent
// (trie path, lists' info, window) runs for all of them at once, and builds
// their sets, up to kPS vertices a round, into one shared-memory buffer by the
// candidate walk of k_level_flat.  Then every vertex a of the buffer is an
// item whose partners are walked the same way, 64 pairs a step: the rest of
// its set, tested in a's table, or a's neighbours above it, tested for
// membership in the set through the tables of the parent's lists, whichever
// are fewer -- one 32-byte load per pair either way.  Vertices of a set with
// kPC or more in the dense core are rows of the core bitmap instead: per row
// the admissible members above and below it are 32 popcounts, and the sums
// over t of B(t) come from the rows of t, so no pair is visited at all.
// Parents with more than kPS candidates are left to a second launch that
// deals them out in pieces of kPK candidates (their core members as bitmaps
// from k_pair_bits); a piece pairs its vertices with neighbours above only.
//
// Bound: L2 latency, instruction issue and the instruction cache (46 % of issue
// slots in the 4-clique + pendant's hub slice).  Whole counts against the form with one parent per
// warp, a hash table of S in shared memory and a degree gather per pair (and,
// without an order between p and c, galloping intersections): 4-clique +
// pendant, 1M vertices / 10M edges, symmetry breaking 33.4 -> 6.6 ms; triangle
// there, plain 75.5 -> 6.2 ms; triangle, 4M / 40M, symmetry breaking 20.2 ->
// 9.1 to 10.3 ms.
constexpr int kPW = 4;            // warps per block
constexpr uint32_t kPS = 512;     // candidates of one round, shared memory words per warp
constexpr uint32_t kPC = 32;      // core members from which a set's core part is counted by rows
constexpr uint32_t kPK = 64;      // candidates per piece of a deferred parent
constexpr uint32_t kPG = 1024;    // candidates a warp keeps of the root parents it took

// True when phase 1 leaves a parent with a window of `len` candidates to phase
// 2: one longer than the split, or, of root parents (p = 1: their sets need no
// tests, so pieces repeat none), one that takes what the warp keeps of a turn,
// `before` candidates up to and with this one, past kPG -- neighbouring hubs
// would be the launch's tail.  The host asks with the longest list and a whole
// turn of them whether phase 2 has to be launched: the rule grows with both.
__host__ __device__ inline bool pair_defers(uint32_t p, uint32_t split, uint32_t len, uint64_t before) {
    return len > split || (p == 1 && before > kPG && len >= kPK / 4);
}

struct PairBig {
    unsigned long long *n;  // [0] deferred parents, [1] their pieces
    uint32_t *q;            // parent index in L_{p-1}
    uint32_t *len;          // candidates in its window
    uint32_t *pref;         // inclusive prefix sum of pieces
    uint32_t *bits;         // per parent: core members of S, then of T (kCore / 32 words each)
    uint32_t cap;
    uint32_t max_pieces;    // what the list may hold of pieces
};

// Pieces a list may hold: their prefix sums and phase 2's work cursor are 32
// bits wide, and cap parents of up to max_deg candidates need not fit (262,144
// sets of 2^20 candidates are 2^32 pieces).  CUTS_FUSE_PIECES=<n> lowers it
// (tests use small values).
constexpr uint32_t kMaxPieces = 1u << 31;

inline uint32_t list_pieces() {
    const char *e = std::getenv("CUTS_FUSE_PIECES");
    return e ? uint32_t(std::min<unsigned long>(std::strtoul(e, nullptr, 10), kMaxPieces)) : kMaxPieces;
}

// A place in the list for a parent of len candidates, or kFullMask where the
// list is full: its pieces are reserved first, in 64 bits.
__device__ __forceinline__ uint32_t list_place(const PairBig &big, uint32_t len) {
    const unsigned long long pieces = len / kPK + 1;
    if (atomicAdd(&big.n[1], pieces) + pieces > big.max_pieces) return kFullMask;
    const unsigned long long slot = atomicAdd(&big.n[0], 1ull);
    return slot < big.cap ? uint32_t(slot) : kFullMask;
}

// Per-lane columns in shared memory, [row][lane].
enum PairRow : int { kRowLo = 0, kRowHi, kRowLoC, kRowHiC, kRowBase, kRowFOff, kRowFDeg, kRowFLo, kRowFHi, kPairRows };

__host__ __device__ inline uint32_t pair_words(uint32_t p, uint32_t njp) {
    return kPS + kPS / 4 + 128 + 4 * 32 + 2 * (kCore / 32) + 32 * (kPairRows + p + 2 * njp);
}

// The pair kernel's weights: none, a fold in general, and a fold under which
// every member of S is admissible as t and A(v) - B(v) is the same for all v of
// one parent, so that a pair weighs the same in both orders.
enum PairFold { kNoWeights = 0, kWeights, kEvenWeights };

// Every member of S is admissible as t: C tests nothing beyond P.
__host__ __device__ inline bool pair_same_set(const LevelPlan &P, const LevelPlan &C, uint32_t p) {
    const uint32_t below = (1u << p) - 1;
    const bool sig = C.sig_lo <= P.sig_lo && (!C.check_sig || (P.check_sig && C.qin <= P.qin && C.qout <= P.qout));
    return !C.fuse_extra && sig && (C.gt_mask & below) == (P.gt_mask & below) && (C.lt_mask & below) == (P.lt_mask & below);
}

// A(v) - B(v) is the same for every v of one parent: both or neither of p and
// c in the orbit and every membership given by the query's arcs, or a plain fold
// that treats both alike.
__host__ __device__ inline bool pair_even(const LevelPlan &F, uint32_t p) {
    const uint32_t c = p + 1, below = (1u << p) - 1;
    if (!F.ofold) return ((F.guar_mask >> p) & 1u) == ((F.guar_mask >> c) & 1u);
    if (((F.ofold >> p) & 1u) != ((F.ofold >> c) & 1u)) return false;
    for (uint32_t x = 0; x < p; ++x)
        if (((F.ofold >> x) & 1u) && !((F.oguar[x] >> p) & 1u)) return false;
    return !((F.ofold >> p) & 1u) || (F.oguar[p] & below) == below;
}

// What the level-p and level-c tests of one warp's parents need.
struct PairCtx {
    const DevView &g;
    const LevelPlan &P, &C, &F;
    uint32_t p, extra;
    bool cfold, ts;             // ts: every member of S is admissible as t
    const uint32_t *m;          // [position][lane]
    const uint32_t *off, *deg;  // [join of p][lane]
    const uint32_t *row;        // [PairRow][lane]
};

// in_list for the tests off the hot path (weights, t's own tests, third and
// later lists): one load site, the tables known to be there.
__device__ __forceinline__ uint32_t pair_list_has(const uint32_t *tab, uint32_t off, uint32_t len, uint32_t v) {
    if (!len) return 0;
    const uint32_t nb = (len + 3) >> 2;
    uint32_t b = tab_bucket(nb, v);
    while (true) {
        const Bucket bk = load_bucket(tab, off, b);
        if (bucket_has(bk, v)) return 1;
        if (bk.k[7] == kTabEmpty) return 0;
        b = b + 1 == nb ? 0 : b + 1;
    }
}

__device__ __forceinline__ bool pair_sig(const DevView &g, const LevelPlan &L, uint32_t v) {
    if (v < L.sig_lo) return false;
    if (!L.check_sig) return true;
    const uint32_t d = g.out_info[v].y;  // symmetric: both degrees
    return d >= L.qin && d >= L.qout;
}

// v, above a member of S of the parent in column l and in the list of its
// join 0, is in S too.  Being above a member, v passes the lower bounds; being
// in a list of m_j it is not m_j unless there are self-loops, so without them
// only the positions that P does not join (`free_pos`) are compared.
__device__ __forceinline__ bool pair_above_in_set(const PairCtx &x, uint32_t l, uint32_t free_pos, uint32_t v) {
    if (x.P.lt_mask && v >= x.row[32 * kRowHi + l]) return false;
    for (uint32_t t = 1; t < x.P.nj; ++t)
        if (!pair_list_has(x.g.tab, x.off[32 * t + l], x.deg[32 * t + l], v)) return false;
    for (uint32_t k = free_pos; k; k &= k - 1)
        if (x.m[32 * (__ffs(k) - 1) + l] == v) return false;
    return !x.P.check_sig || pair_sig(x.g, x.P, v);
}

// v, known to lie in join t0 of the parent in column l, is in its S.
__device__ __forceinline__ bool pair_in_set(const PairCtx &x, uint32_t l, uint32_t t0, uint32_t v) {
    if (v < x.row[32 * kRowLo + l] || v >= x.row[32 * kRowHi + l]) return false;
    for (uint32_t t = 0; t < x.P.nj; ++t)
        if (t != t0 && !pair_list_has(x.g.tab, x.off[32 * t + l], x.deg[32 * t + l], v)) return false;
    for (uint32_t j = 0; j < x.p; ++j)
        if (x.m[32 * j + l] == v) return false;
    return pair_sig(x.g, x.P, v);
}

// The member v of S is admissible as t.
__device__ __forceinline__ bool pair_adm(const PairCtx &x, uint32_t l, uint32_t v) {
    if (x.ts) return true;
    if (v < x.row[32 * kRowLoC + l] || v >= x.row[32 * kRowHiC + l]) return false;
    for (uint32_t t = 0; t < x.C.nj; ++t)
        if ((x.extra >> t) & 1u) {
            const uint2 inf = x.g.out_info[x.m[32 * x.C.jpos[t] + l]];
            if (!pair_list_has(x.g.tab, inf.x, inf.y, v)) return false;
        }
    return pair_sig(x.g, x.C, v);
}

// A(v): the weight of v at position p, without what t adds -- the orbit base
// with v at p minus the orbit positions below c (each of their lists holds
// t), or the plain fold's base minus v's own membership.
template <bool LOOPS>
__device__ __forceinline__ uint32_t pair_a(const PairCtx &x, uint32_t l, uint32_t v) {
    if (!x.cfold) return 1;
    const LevelPlan &F = x.F;
    uint32_t a = x.row[32 * kRowBase + l];
    if (F.ofold) {
        for (uint32_t xm = F.ofold & ((1u << x.p) - 1); xm; xm &= xm - 1) {
            const uint32_t o = __ffs(xm) - 1;
            bool in = (F.oguar[o] >> x.p) & 1u;
            if (!in) {
                const uint2 inf = x.g.out_info[x.m[32 * o + l]];
                in = pair_list_has(x.g.tab, inf.x, inf.y, v);
            }
            a -= in;
        }
        if ((F.ofold >> x.p) & 1u) {
            const uint2 inf = x.g.out_info[v];
            a += inf.y;
            for (uint32_t j = 0; j < x.p; ++j)
                if (((F.oguar[x.p] >> j) & 1u) || pair_list_has(x.g.tab, inf.x, inf.y, x.m[32 * j + l])) --a;
            if (LOOPS) a -= pair_list_has(x.g.tab, inf.x, inf.y, v);
        }
        return a - __popc(F.ofold & ((1u << (x.p + 1)) - 1));
    }
    const bool in = v >= x.row[32 * kRowFLo + l] && v < x.row[32 * kRowFHi + l] &&
                    (((F.guar_mask >> x.p) & 1u) || pair_list_has(x.g.tab, x.row[32 * kRowFOff + l], x.row[32 * kRowFDeg + l], v));
    return a - in;
}

// B(v): what v at position c adds (an orbit vertex its own list outside the
// core; the plain fold loses v itself).  Sums wrap in 32 bits, totals do not.
template <bool LOOPS>
__device__ __forceinline__ uint32_t pair_b(const PairCtx &x, uint32_t l, uint32_t v) {
    if (!x.cfold) return 0;
    const LevelPlan &F = x.F;
    const uint32_t c = x.p + 1;
    if (F.ofold) {
        if (!((F.ofold >> c) & 1u)) return 0u;
        const uint2 inf = x.g.out_info[v];
        return inf.y - c - (LOOPS ? pair_list_has(x.g.tab, inf.x, inf.y, v) : 0u);
    }
    const bool in = v >= x.row[32 * kRowFLo + l] && v < x.row[32 * kRowFHi + l] &&
                    (((F.guar_mask >> c) & 1u) || pair_list_has(x.g.tab, x.row[32 * kRowFOff + l], x.row[32 * kRowFDeg + l], v));
    return in ? 0xffffffffu : 0u;
}

// One lane's parent q0 at level p - 1: matched vertices, joined lists, windows
// and fold data into its columns; the shortest list and its window out.
struct PairParent {
    uint32_t moff, s0, e0, tmin;
};

__device__ __forceinline__ PairParent pair_parent(const DevView &g, const RunParams *rp, const LevelPlan &P,
                                                  const LevelPlan &C, const LevelPlan &F, bool cfold, bool loops, uint32_t p,
                                                  uint32_t *const *s_vert, uint32_t *const *s_par, uint32_t q0,
                                                  uint32_t lane, uint32_t *m, uint32_t *off, uint32_t *deg,
                                                  uint32_t *row) {
    uint32_t e = q0;
    for (int j = int(p) - 1; j >= 0; --j) {
        m[32 * j + lane] = s_vert[j][e];
        if (j > 0) e = s_par[j][e];
    }
    PairParent r{0, 0, 0, 0};
    uint32_t mdeg = kFullMask;
    for (uint32_t t = 0; t < P.nj; ++t) {
        const uint2 inf = g.out_info[m[32 * P.jpos[t] + lane]];
        off[32 * t + lane] = inf.x;
        deg[32 * t + lane] = inf.y;
        if (inf.y < mdeg) { mdeg = inf.y; r.moff = inf.x; r.tmin = t; }
    }
    uint32_t lo = 0, hi = kFullMask, loc = 0, hic = kFullMask;
    const uint32_t below = (1u << p) - 1;
    for (uint32_t k = P.gt_mask; k; k &= k - 1) lo = max(lo, m[32 * (__ffs(k) - 1) + lane] + 1);
    for (uint32_t k = P.lt_mask; k; k &= k - 1) hi = min(hi, m[32 * (__ffs(k) - 1) + lane]);
    for (uint32_t k = C.gt_mask & below; k; k &= k - 1) loc = max(loc, m[32 * (__ffs(k) - 1) + lane] + 1);
    for (uint32_t k = C.lt_mask & below; k; k &= k - 1) hic = min(hic, m[32 * (__ffs(k) - 1) + lane]);
    row[32 * kRowLo + lane] = lo;
    row[32 * kRowHi + lane] = hi;
    row[32 * kRowLoC + lane] = loc;
    row[32 * kRowHiC + lane] = hic;
    const uint32_t mu = m[32 * P.jpos[r.tmin] + lane];
    const uint32_t *lst = g.adj + r.moff;
    r.s0 = kFullMask;
    if (lo && p >= 2 && rp->pos_lvl == p - 1 && lo == m[32 * (p - 1) + lane] + 1) {
        // the window starts right after the parent's own vertex: when that
        // vertex was drawn from this very list, its offset is known
        const uint32_t apos = rp->ub[p - 1][q0];
        if (apos >= r.moff && apos - r.moff < mdeg) r.s0 = apos - r.moff + 1;
    }
    if (r.s0 == kFullMask) r.s0 = lo ? lbound_own(g, false, mu, lst, mdeg, lo, loops) : 0;
    r.e0 = hi != kFullMask ? lbound_own(g, false, mu, lst, mdeg, hi, loops) : mdeg;
    if (r.e0 < r.s0) r.e0 = r.s0;
    if (cfold && F.ofold) {
        // the orbit base of the positions below p
        uint32_t base = 0;
        for (uint32_t xm = F.ofold & below; xm; xm &= xm - 1) {
            const uint32_t o = __ffs(xm) - 1;
            const uint2 inf = g.out_info[m[32 * o + lane]];
            base += inf.y;
            for (uint32_t j = 0; j < p; ++j)
                if (((F.oguar[o] >> j) & 1u) || pair_list_has(g.tab, inf.x, inf.y, m[32 * j + lane])) --base;
        }
        row[32 * kRowBase + lane] = base;
    } else if (cfold) {
        // the plain fold's list and window, fixed by the positions below p
        const uint2 inf = g.out_info[m[32 * F.jpos[0] + lane]];
        uint32_t flo = 0, fhi = kFullMask;
        for (uint32_t k = F.gt_mask & below; k; k &= k - 1) flo = max(flo, m[32 * (__ffs(k) - 1) + lane] + 1);
        for (uint32_t k = F.lt_mask & below; k; k &= k - 1) fhi = min(fhi, m[32 * (__ffs(k) - 1) + lane]);
        const uint32_t *fl = g.adj + inf.x;
        const uint32_t ws = flo ? lbound(fl, inf.y, flo) : 0, we = fhi != kFullMask ? lbound(fl, inf.y, fhi) : inf.y;
        uint32_t sub = 0;
        for (uint32_t j = 0; j < p; ++j) {
            const uint32_t mj = m[32 * j + lane];
            if (mj >= flo && mj < fhi && (((F.guar_mask >> j) & 1u) || pair_list_has(g.tab, inf.x, inf.y, mj))) ++sub;
        }
        row[32 * kRowBase + lane] = (we > ws ? we - ws : 0) - sub;
        row[32 * kRowFOff + lane] = inf.x;
        row[32 * kRowFDeg + lane] = inf.y;
        row[32 * kRowFLo + lane] = flo;
        row[32 * kRowFHi + lane] = fhi;
    }
    return r;
}

// The plan's pieces and the shared layout, the same in both pair kernels.
#define PAIR_PROLOGUE()                                                                                       \
    __shared__ LevelPlan sP, sC, sF;                                                                          \
    __shared__ uint32_t *s_vert[kMaxK];                                                                       \
    __shared__ uint32_t *s_par[kMaxK];                                                                        \
    extern __shared__ __align__(16) uint32_t dyn[];                                                           \
    {                                                                                                         \
        const uint32_t words = sizeof(LevelPlan) / 4, f = p + 2 < rp->plan.k ? p + 2 : p + 1;                 \
        for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) {                                          \
            reinterpret_cast<uint32_t *>(&sP)[i] = reinterpret_cast<const uint32_t *>(&rp->plan.lv[p])[i];    \
            reinterpret_cast<uint32_t *>(&sC)[i] = reinterpret_cast<const uint32_t *>(&rp->plan.lv[p + 1])[i]; \
            reinterpret_cast<uint32_t *>(&sF)[i] = reinterpret_cast<const uint32_t *>(&rp->plan.lv[f])[i];    \
        }                                                                                                     \
        if (threadIdx.x < kMaxK) {                                                                            \
            s_vert[threadIdx.x] = rp->vert[threadIdx.x];                                                      \
            s_par[threadIdx.x] = rp->par[threadIdx.x];                                                        \
        }                                                                                                     \
    }                                                                                                         \
    __syncthreads();                                                                                          \
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;                                               \
    const uint32_t njp = sP.nj;                                                                               \
    uint32_t *const wbase = dyn + warp * pair_words(p, njp);                                                  \
    uint4 *const rec = reinterpret_cast<uint4 *>(wbase);                                                      \
    uint32_t *const starts = wbase + 128;                                                                     \
    uint32_t *const segs = starts + 32;   /* [lane]: first entry of its segment that is a row */              \
    uint32_t *const sege = segs + 32;     /* [lane]: its segment's end, or kFullMask for a piece */           \
    uint32_t *const itemA = sege + 32;    /* [rank]: A of the item's vertex */                                \
    uint32_t *const Sb = itemA + 32;      /* core members of S, then of T */                                  \
    uint32_t *const Tb = Sb + kCore / 32;                                                                     \
    uint32_t *const S = Tb + kCore / 32;                                                                      \
    uint8_t *const So = reinterpret_cast<uint8_t *>(S + kPS);  /* the member's column */                      \
    uint32_t *const row = S + kPS + kPS / 4;                                                                  \
    uint32_t *const col_off = row + 32 * kPairRows, *const col_deg = col_off + 32 * njp;                      \
    uint32_t *const col_m = col_deg + 32 * njp;                                                               \
    const uint32_t below = (1u << p) - 1;                                                                     \
    const bool cfold = FOLD != 0;                                                                             \
    const uint32_t extra = sC.fuse_extra;                                                                     \
    const bool ts = FOLD == kEvenWeights || pair_same_set(sP, sC, p);                                         \
    const PairCtx x{g, sP, sC, sF, p, extra, cfold, ts, col_m, col_off, col_deg, row};

// LOOPS: the graph has self-loops.
template <int FOLD, bool TALLY, bool LOOPS>
__global__ void __launch_bounds__(kPW * 32, 8)
k_pairs(DevView g, const RunParams *__restrict__ rp, uint32_t p, const Parents parents, uint32_t phase, uint32_t split,
        uint32_t *__restrict__ cursor, PairBig big, unsigned long long *__restrict__ acc,
        unsigned long long *__restrict__ acc_c, unsigned long long *__restrict__ acc_p,
        unsigned long long *__restrict__ acc_bytes) {
    uint32_t pa, total;
    parents_of(parents, pa, total);
    if (!total) return;
    PAIR_PROLOGUE()
    const uint32_t lanemask_lt = (1u << lane) - 1, lanemask_le = lanemask_lt | (1u << lane);
    // t above s only, below s only, or both
    const bool t_up = !((sC.lt_mask >> p) & 1u), t_down = !((sC.gt_mask >> p) & 1u);
    // even weights: counted in one order, times the number of orders at the end
    constexpr bool once = FOLD == kEvenWeights;
    const bool o1 = once || t_up, o2 = !once && t_down;
    const bool phase2 = phase == 2;
    uint32_t nbig = 0;
    if (phase2) {
        const unsigned long long n0 = big.n[0];
        nbig = n0 < big.cap ? uint32_t(n0) : big.cap;
        total = nbig ? big.pref[nbig - 1] : 0;
    }
    const uint32_t nwarps = gridDim.x * kPW;
    // a few grabs per warp at least: parents differ in work
    const uint32_t grab = min(phase2 ? 1u : 32u, max(1u, total / (4 * nwarps)));
    const unsigned long long deadline = run_deadline(rp);
    unsigned long long local = 0, local_c = 0, local_p = 0, tb = 0;
    const bool kconst = FOLD != kWeights || pair_even(sF, p);
    const uint32_t orders = (o1 ? 1u : 0u) + (o2 ? 1u : 0u);
    const uint32_t times = once && t_up && t_down ? 2u : 1u;
    // even weights: a hit costs one of them and no test, in an instance without
    // the code of the others, for the fold's inner loop is bound by the
    // instruction cache.  Triangle + pendant, 60-regular graph of 700,003
    // vertices, plain 17.2 -> 11.9 ms; 50,000, symmetry breaking 0.50 -> 0.37;
    // power law, 1M / 10M, 2.93 -> 2.59; 4-clique + pendant there 7.8 -> 6.3.
    // degs: B is the degree less this
    const uint32_t degs = once && !LOOPS && ((sF.ofold >> (p + 1)) & 1u) ? p + 1 : 0u;
    uint32_t free_pos = below;  // positions below p whose lists P does not join (all with self-loops)
    if (!LOOPS)
        for (uint32_t t = 0; t < njp; ++t) free_pos &= ~(1u << sP.jpos[t]);

    while (true) {
        uint32_t start = 0;
        if (lane == 0) start = past_deadline(rp, deadline) ? total : atomicAdd(cursor, grab);
        start = __shfl_sync(kFullMask, start, 0);
        if (start >= total) break;
        // this lane's parent and the candidates [pos, end) of its window left
        uint32_t pos = 0, end = 0, b = kFullMask;
        bool piece = false;  // part of a window only: pairs with neighbours above
        PairParent pp{0, 0, 0, 0};
        if (uint32_t(lane) < grab && start + lane < total) {
            uint32_t q0 = pa + start + lane, ch = 0;
            if (phase2) {
                const uint32_t gi = start + lane;
                uint32_t lo = 0, hi = nbig - 1;  // first b with pref[b] > gi
                while (lo < hi) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (big.pref[mid] > gi) hi = mid; else lo = mid + 1;
                }
                b = lo;
                ch = gi - (b ? big.pref[b - 1] : 0);
                q0 = big.q[b];
            }
            pp = pair_parent(g, rp, sP, sC, sF, cfold, LOOPS, p, s_vert, s_par, q0, lane, col_m, col_off, col_deg, row);
            pos = pp.s0;
            end = pp.e0;
            if (TALLY) tb += 8ull * p + 8ull * njp;
            if (phase2) {
                piece = true;
                pos = min(pp.s0 + ch * kPK, end);
                end = min(pos + kPK, end);
            }
        }
        if (!phase2) {
            uint32_t before = 0;
            if (p == 1) {
                before = end - pos;
                #pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(kFullMask, before, o);
                    if (lane >= o) before += y;
                }
            }
            if (pair_defers(p, split, end - pos, before)) {
                piece = true;
                const uint32_t slot = list_place(big, end - pos);
                if (slot != kFullMask) {
                    big.q[slot] = pa + start + lane;
                    big.len[slot] = end - pos;
                    end = pos;
                }  // else: the list is full, this warp counts it piece by piece
            }
        }
        while (true) {
            // ---- the next round: whole windows (pieces of kPS) while they fit
            const uint32_t take = min(end - pos, kPS);
            uint32_t incl = take;
            #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
                if (lane >= o) incl += y;
            }
            const uint32_t len = incl <= kPS ? take : 0u;  // a prefix of the lanes
            const unsigned live = __ballot_sync(kFullMask, len != 0);
            if (!live) break;
            const uint32_t ftotal = __shfl_sync(kFullMask, incl, 31 - __clz(live));
            if (len) {
                const uint32_t r = __popc(live & lanemask_lt), excl = incl - len, to = pp.tmin ? 0u : 1u;
                rec[r] = make_uint4(pp.moff + pos - excl, uint32_t(lane) | (pp.tmin << 8),
                                    njp > 1 ? col_off[32 * to + lane] : 0u, njp > 1 ? col_deg[32 * to + lane] : 0u);
                starts[r] = excl;
                pos += len;
            }
            __syncwarp();
            // ---- the sets, in order of the lanes
            uint32_t ns = 0;
            {
                const uint32_t my_start = uint32_t(lane) < uint32_t(__popc(live)) ? starts[lane] : kFullMask;
                uint32_t started = 0;
                for (uint32_t fstep = 0; fstep < ftotal; fstep += 32) {
                    const uint32_t rel = my_start - fstep;
                    const uint32_t bits = __reduce_or_sync(kFullMask, rel < 32u ? 1u << rel : 0u);
                    const uint4 rc = rec[started + __popc(bits & lanemask_le) - 1];
                    started += __popc(bits);
                    const uint32_t f = fstep + lane, owner = rc.y & 255u, tmin = rc.y >> 8;
                    bool ok = f < ftotal;
                    const uint32_t v = __ldg(g.adj + (rc.x + min(f, ftotal - 1)));
                    ok = ok && v >= sP.sig_lo;
                    if (ok && njp > 1) ok = in_list(g, rc.z, rc.w, v);
                    if (ok && njp > 2)
                        for (uint32_t t = (tmin < 2 ? 2u : 1u); t < njp; ++t)
                            if (t != tmin && !pair_list_has(g.tab, col_off[32 * t + owner], col_deg[32 * t + owner], v)) {
                                ok = false;
                                break;
                            }
                    if (ok)
                        for (uint32_t j = 0; j < p; ++j)
                            if (v == col_m[32 * j + owner]) { ok = false; break; }
                    if (ok && sP.check_sig) ok = pair_sig(g, sP, v);
                    const unsigned m = __ballot_sync(kFullMask, ok);
                    if (ok) {
                        const uint32_t i = ns + __popc(m & lanemask_lt);
                        S[i] = v;
                        So[i] = uint8_t(owner);
                    }
                    ns += __popc(m);
                    if (TALLY && f < ftotal) tb += 4 + 32ull * (njp - 1) + (sP.check_sig ? 8 : 0);
                }
            }
            __syncwarp();
            if (lane == 0) local_p += ns;
            // ---- segments: [lo, hi) of the lane, its core members from cut on
            uint32_t lo = 0;
            for (uint32_t n = ns; n;) {  // first member whose column is >= lane
                const uint32_t half = n >> 1;
                if (So[lo + half] < lane) { lo += half + 1; n -= half + 1; }
                else n = half;
            }
            uint32_t hi = __shfl_down_sync(kFullMask, lo, 1);
            if (lane == 31) hi = ns;
            uint32_t cut = hi;
            if (g.core_bits && (piece ? b != kFullMask && hi > lo : hi - lo >= kPC)) {
                uint32_t c0 = lo;
                for (uint32_t n = hi - lo; n;) {
                    const uint32_t half = n >> 1;
                    if (S[c0 + half] < g.core0) { c0 += half + 1; n -= half + 1; }
                    else n = half;
                }
                if (piece || hi - c0 >= kPC) cut = c0;
            }
            segs[lane] = cut;
            sege[lane] = piece ? kFullMask : hi;
            __syncwarp();
            // ---- items: each member that is no row, with its partners above
            for (uint32_t i0 = 0; i0 < ns; i0 += 32) {
                const uint32_t i = i0 + lane;
                uint32_t ilen = 0, ibase = 0, ioff = 0, ideg = 0, ow = 0, mode = 0, a = 0;
                if (i < ns) {
                    ow = So[i];
                    a = S[i];
                    if (i < segs[ow]) {
                        const uint32_t se = sege[ow];
                        const uint32_t lenS = se == kFullMask ? kFullMask : se - i - 1;
                        if (lenS) {
                            const uint2 inf = g.out_info[a];
                            uint32_t bw = __ldg(g.bwd_out + a);
                            if (LOOPS && bw < inf.y && __ldg(g.adj + inf.x + bw) == a) ++bw;
                            const uint32_t lenN = inf.y - bw;
                            if (TALLY) tb += 12;
                            mode = lenN < lenS ? 1u : 0u;
                            ilen = min(lenN, lenS);
                            ibase = mode ? inf.x + bw : i + 1;
                            ioff = mode ? col_off[ow] : inf.x;
                            ideg = mode ? col_deg[ow] : inf.y;
                        }
                    }
                }
                uint32_t iincl = ilen;
                #pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(kFullMask, iincl, o);
                    if (lane >= o) iincl += y;
                }
                const uint32_t itotal = __shfl_sync(kFullMask, iincl, 31);
                if (!itotal) continue;
                const unsigned ilive = __ballot_sync(kFullMask, ilen != 0);
                if (ilen) {
                    const uint32_t r = __popc(ilive & lanemask_lt), excl = iincl - ilen;
                    rec[r] = make_uint4(ibase - excl, ow | (mode << 8) | (i << 16), ioff, ideg);
                    starts[r] = excl;
                    if (FOLD) itemA[r] = o1 ? pair_a<LOOPS>(x, ow, a) : 0u;
                }
                __syncwarp();
                const uint32_t my_start = uint32_t(lane) < uint32_t(__popc(ilive)) ? starts[lane] : kFullMask;
                uint32_t started = 0, hits = 0;  // hits: of a batch without weights
                for (uint32_t fstep = 0; fstep < itotal; fstep += 64) {
                    uint4 rc[2];
                    uint32_t tv[2], rk[2];
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t rel = my_start - (fstep + 32 * h);
                        const uint32_t bits = __reduce_or_sync(kFullMask, rel < 32u ? 1u << rel : 0u);
                        rk[h] = started + __popc(bits & lanemask_le) - 1;
                        started += __popc(bits);
                        rc[h] = rec[rk[h]];
                        const uint32_t at = rc[h].x + min(fstep + 32 * h + lane, itotal - 1);
                        tv[h] = (rc[h].y & 256u) ? __ldg(g.adj + at) : S[at];
                    }
                    uint32_t nb[2], bu[2];
                    Bucket bk[2];
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        nb[h] = (rc[h].w + 3) >> 2;
                        bu[h] = tab_bucket(nb[h], tv[h]);
                        bk[h] = load_bucket(g.tab, rc[h].z, bu[h]);
                    }
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        bool ok = fstep + 32 * h + lane < itotal;
                        const uint32_t t = tv[h];
                        if (TALLY && ok) tb += 32 + ((rc[h].y & 256u) ? 4 : 0);
                        if (ok && !bucket_has(bk[h], t)) ok = tab_continue(g.tab, rc[h].z, nb[h], bu[h], bk[h], t);
                        if (ok && (rc[h].y & 256u))
                            ok = FOLD ? pair_in_set(x, rc[h].y & 255u, 0, t)
                                      : pair_above_in_set(x, rc[h].y & 255u, free_pos, t);
                        if (!FOLD && ts) {
                            hits += ok;
                        } else if (once) {
                            if (ok) {
                                ++local_c;
                                local += uint32_t(itemA[rk[h]] + (degs ? g.out_info[t].y - degs : pair_b<LOOPS>(x, rc[h].y & 255u, t)));
                            }
                        } else if (ok) {
                            const uint32_t l = rc[h].y & 255u;
                            {
                                const uint32_t av = S[rc[h].y >> 16];
                                if (o1 && pair_adm(x, l, t)) {
                                    ++local_c;
                                    local += FOLD ? uint32_t(itemA[rk[h]] + pair_b<LOOPS>(x, l, t)) : 1u;
                                }
                                if (o2 && pair_adm(x, l, av)) {
                                    ++local_c;
                                    local += FOLD ? uint32_t(pair_a<LOOPS>(x, l, t) + pair_b<LOOPS>(x, l, av)) : 1u;
                                }
                            }
                        }
                    }
                }
                local += uint64_t(hits) * orders;
                local_c += uint64_t(hits) * orders;
                __syncwarp();
            }
            // ---- rows: the core members of the larger sets
            for (unsigned todo = __ballot_sync(kFullMask, cut < hi); todo; todo &= todo - 1) {
                const int l = __ffs(todo) - 1;
                const uint32_t c0 = __shfl_sync(kFullMask, cut, l), ce = __shfl_sync(kFullMask, hi, l);
                const uint32_t lb = __shfl_sync(kFullMask, b, l);
                __syncwarp();
                if (lb != kFullMask) {
                    Sb[lane] = big.bits[size_t(lb) * (kCore / 16) + lane];
                    Tb[lane] = big.bits[size_t(lb) * (kCore / 16) + kCore / 32 + lane];
                    __syncwarp();
                } else {
                    Sb[lane] = 0;
                    Tb[lane] = 0;
                    __syncwarp();
                    for (uint32_t i = c0 + lane; i < ce; i += 32) {
                        const uint32_t u = S[i] - g.core0;
                        atomicOr(&Sb[u >> 5], 1u << (u & 31));
                        if (!ts && pair_adm(x, uint32_t(l), S[i])) atomicOr(&Tb[u >> 5], 1u << (u & 31));
                    }
                    __syncwarp();
                    if (ts) Tb[lane] = Sb[lane];
                    __syncwarp();
                }
                if (lb == kFullMask && ts && kconst) {
                    // a whole set, every member admissible: with n(v) the
                    // members of S in v's row, the pairs' weights add up to
                    // sum B(v) n(v) + (A - B) * pairs, pairs = sum n(v) / 2
                    uint32_t n2 = 0, kap = 0;
                    unsigned long long wsum = 0;
                    const uint32_t q0 = (S[c0] - g.core0) >> 7;  // words below the lowest member are empty
                    for (uint32_t i = c0 + lane; i < ce; i += 32) {
                        const uint32_t v = S[i];
                        const uint4 *rp4 = reinterpret_cast<const uint4 *>(g.core_bits + size_t(v - g.core0) * (kCore / 32));
                        uint32_t n = 0;
                        #pragma unroll 4
                        for (uint32_t q = q0; q < kCore / 128; ++q) {
                            const uint4 r4 = __ldg(rp4 + q), s4 = reinterpret_cast<const uint4 *>(Sb)[q];
                            n += __popc(r4.x & s4.x) + __popc(r4.y & s4.y) + __popc(r4.z & s4.z) + __popc(r4.w & s4.w);
                        }
                        n2 += n;
                        if (TALLY) tb += 8 + 16ull * (kCore / 128 - q0);
                        if (FOLD) {
                            const uint32_t B = pair_b<LOOPS>(x, uint32_t(l), v);
                            wsum += (unsigned long long)((long long)int32_t(B) * n);
                            if (i == c0) kap = pair_a<LOOPS>(x, uint32_t(l), v) - B;
                        }
                    }
                    #pragma unroll
                    for (int o = 16; o; o >>= 1) n2 += __shfl_xor_sync(kFullMask, n2, o);
                    const uint32_t pairs = n2 >> 1;
                    if (FOLD) local += orders * wsum;
                    if (lane == 0) {
                        local += (unsigned long long)(orders * pairs) * (FOLD ? kap : 1u);  // A - B >= 0 where there is a pair
                        local_c += orders * pairs;
                    }
                    continue;
                }
                for (uint32_t i = c0 + lane; i < ce; i += 32) {
                    const uint32_t v = S[i], u = v - g.core0, w0 = u >> 5;
                    const uint32_t above = ~((2u << (u & 31)) - 1u), under = (1u << (u & 31)) - 1u;
                    const uint4 *rp4 = reinterpret_cast<const uint4 *>(g.core_bits + size_t(u) * (kCore / 32));
                    uint32_t upS = 0, dnS = 0, upT = 0, dnT = 0;
                    #pragma unroll 2
                    for (uint32_t q = 0; q < kCore / 128; ++q) {
                        const uint4 r4 = __ldg(rp4 + q);
                        const uint32_t rw[4] = {r4.x, r4.y, r4.z, r4.w};
                        #pragma unroll
                        for (uint32_t k = 0; k < 4; ++k) {
                            const uint32_t j = 4 * q + k;
                            const uint32_t ma = j > w0 ? kFullMask : (j == w0 ? above : 0u);
                            const uint32_t mb = j < w0 ? kFullMask : (j == w0 ? under : 0u);
                            const uint32_t ws = rw[k] & Sb[j];
                            upS += __popc(ws & ma);
                            if (FOLD || !ts || !o1) dnS += __popc(ws & mb);
                            if (!ts) {
                                const uint32_t wt = rw[k] & Tb[j];
                                upT += __popc(wt & ma);
                                dnT += __popc(wt & mb);
                            }
                        }
                    }
                    if (ts) {
                        upT = upS;
                        dnT = dnS;
                    }
                    if (TALLY) tb += 8 + kCore / 8;
                    if (!FOLD && ts && o1) {
                        // every pair once, from its lower row
                        const uint32_t n = o2 ? 2 * upS : upS;
                        local += n;
                        local_c += n;
                    } else {
                        const bool adm = ts || pair_adm(x, uint32_t(l), v);
                        const uint32_t A = pair_a<LOOPS>(x, uint32_t(l), v), B = pair_b<LOOPS>(x, uint32_t(l), v);
                        // A of a vertex with a pair fits 32 bits; B is below
                        // 2^31 or, in a plain fold, -1
                        long long s = 0;
                        if (o1) {
                            s += (long long)A * upT + (adm ? (long long)int32_t(B) * dnS : 0);
                            local_c += upT;
                        }
                        if (o2) {
                            s += (long long)A * dnT + (adm ? (long long)int32_t(B) * upS : 0);
                            local_c += dnT;
                        }
                        local += (unsigned long long)s;
                    }
                }
            }
            __syncwarp();
        }
        __syncwarp();
    }
    local *= times;
    local_c *= times;
    #pragma unroll
    for (int o = 16; o; o >>= 1) {
        local += __shfl_xor_sync(kFullMask, local, o);
        local_c += __shfl_xor_sync(kFullMask, local_c, o);
        if (TALLY) tb += __shfl_xor_sync(kFullMask, tb, o);
    }
    if (lane == 0) {
        if (local) atomicAdd(acc, local);
        if (local_c) atomicAdd(acc_c, local_c);
        if (local_p) atomicAdd(acc_p, local_p);
        if (TALLY && tb) atomicAdd(acc_bytes, tb);
    }
}

// Core members of the deferred parents' sets, one warp per parent.
template <int FOLD>
__global__ void __launch_bounds__(kPW * 32)
k_pair_bits(DevView g, const RunParams *__restrict__ rp, uint32_t p, PairBig big) {
    const unsigned long long n0 = big.n[0];
    const uint32_t nbig = n0 < big.cap ? uint32_t(n0) : big.cap;
    if (!nbig || !g.core_bits) return;
    PAIR_PROLOGUE()
    (void)rec; (void)starts; (void)segs; (void)sege; (void)itemA; (void)S; (void)So;
    for (uint32_t b = blockIdx.x * kPW + warp; b < nbig; b += gridDim.x * kPW) {
        uint32_t moff = 0, s0 = 0, e0 = 0, tmin = 0;
        if (lane == 0) {
            const PairParent pp = pair_parent(g, rp, sP, sC, sF, false, rp->plan.data_loops != 0, p, s_vert, s_par,
                                              big.q[b], 0, col_m, col_off, col_deg, row);
            moff = pp.moff;
            s0 = pp.s0;
            e0 = pp.e0;
            tmin = pp.tmin;
            const uint32_t c0 = lbound(g.adj + moff, e0, g.core0);
            s0 = max(s0, c0);
        }
        moff = __shfl_sync(kFullMask, moff, 0);
        s0 = __shfl_sync(kFullMask, s0, 0);
        e0 = __shfl_sync(kFullMask, e0, 0);
        tmin = __shfl_sync(kFullMask, tmin, 0);
        Sb[lane] = 0;
        Tb[lane] = 0;
        __syncwarp();
        for (uint32_t i = s0 + lane; i < e0; i += 32) {
            const uint32_t v = __ldg(g.adj + moff + i), u = v - g.core0;
            if (pair_in_set(x, 0, tmin, v)) {
                atomicOr(&Sb[u >> 5], 1u << (u & 31));
                if (pair_adm(x, 0, v)) atomicOr(&Tb[u >> 5], 1u << (u & 31));
            }
        }
        __syncwarp();
        big.bits[size_t(b) * (kCore / 16) + lane] = Sb[lane];
        big.bits[size_t(b) * (kCore / 16) + kCore / 32 + lane] = Tb[lane];
        __syncwarp();
    }
}

// ---- edges between two candidate sets ----------------------------------
// When level d = k-2 joins one list of an earlier vertex and the last level
// joins the vertex at d and one earlier vertex (cycles, the house, ladders),
// one parent at level d-1 fixes two sets, C (candidates of d) and T (those of
// the last level but for d's list), and the two levels' matches are the edges
// between them.  L_d is neither stored nor walked entry by entry: its size is
// |C| by list arithmetic, and the edges are found from the smaller set.  A warp takes up
// to 32 parents, one per lane, puts their smaller sets into shared memory and
// walks, for every vertex v there, the other set's window (tested in v's
// table) or v's own neighbours (tested in the other set's list), whichever is
// shorter, 64 a step as in k_level_flat.  Where both sets have kECore or more
// vertices in the dense core, the edges there are popcounts of its bitmap rows
// against the other set's core members.  Sets of more than `split` vertices
// are dealt out in pieces by a second launch.  On a graph whose ids are degree
// ranks, so that d's signature is a bound on the id.
// What it saves is the set-up per entry of L_d: the 5-cycle on 200,003
// vertices / 1M edges has 6.9e9 of them with 1.5 last-level candidates each.
// Whole counts against expanding L_d and counting its entries: that 5-cycle
// 273 -> 45 ms, the house on 100,000 / 500,000 22 -> 18.4 ms, the 4-cycle on
// 10,000 / 40,000 117 -> 101 us.  Bound: instruction issue (45 % of slots), L1
// (79 % of its throughput) and L2 latency.
constexpr uint32_t kECore = 8;    // core members of each set from which they are counted by rows
enum EdgeRow : int { kECOff = 0, kECDeg, kETOff, kETDeg, kEOLo, kEOHi, kEOBase, kEOLen, kESide, kEMatched, kEONear, kECut, kEdgeRows };

__host__ __device__ inline uint32_t edge_words(uint32_t d) {
    return kPS + kPS / 4 + 128 + 32 + kCore / 32 + 32 * (kEdgeRows + d);
}

template <bool ROWS, bool TALLY>
__global__ void __launch_bounds__(kPW * 32, 8)
k_edges(DevView g, const RunParams *__restrict__ rp, uint32_t d, uint32_t turns, const Parents parents, uint32_t phase,
        uint32_t split, uint32_t *__restrict__ cursor, PairBig big, unsigned long long *__restrict__ acc,
        unsigned long long *__restrict__ acc_d, unsigned long long *__restrict__ accb) {
    uint32_t pa, total;
    parents_of(parents, pa, total);
    if (!total) return;
    __shared__ LevelPlan sC, sT;
    __shared__ uint32_t *s_vert[kMaxK];
    __shared__ uint32_t *s_par[kMaxK];
    extern __shared__ __align__(16) uint32_t dyn[];
    {
        const uint32_t words = sizeof(LevelPlan) / 4;
        for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) {
            reinterpret_cast<uint32_t *>(&sC)[i] = reinterpret_cast<const uint32_t *>(&rp->plan.lv[d])[i];
            reinterpret_cast<uint32_t *>(&sT)[i] = reinterpret_cast<const uint32_t *>(&rp->plan.lv[d + 1])[i];
        }
        if (threadIdx.x < kMaxK) {
            s_vert[threadIdx.x] = rp->vert[threadIdx.x];
            s_par[threadIdx.x] = rp->par[threadIdx.x];
        }
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1, le = lt | (1u << lane);
    uint32_t *const wbase = dyn + warp * edge_words(d);
    uint4 *const rec = reinterpret_cast<uint4 *>(wbase);
    uint32_t *const starts = wbase + 128;
    uint32_t *const Ob = starts + 32;                          // core members of one other set
    uint32_t *const S = Ob + kCore / 32;
    uint8_t *const So = reinterpret_cast<uint8_t *>(S + kPS);  // the member's column
    uint32_t *const row = S + kPS + kPS / 4;                   // [EdgeRow][lane]
    uint32_t *const m = row + 32 * kEdgeRows;                  // [position][lane]
    const uint32_t jt = sT.jpos[0] == d ? sT.jpos[1] : sT.jpos[0];  // T's list
    const bool t_above = (sT.gt_mask >> d) & 1u, t_below = (sT.lt_mask >> d) & 1u;  // order between d and the last level
    const uint32_t below = (1u << d) - 1;
    const bool loops = rp->plan.data_loops != 0;
    const bool ordered = t_above || t_below || loops;  // a hit is compared with its vertex
    const bool phase2 = phase == 2;
    uint32_t nbig = 0;
    if (phase2) {
        const unsigned long long n0 = big.n[0];
        nbig = n0 < big.cap ? uint32_t(n0) : big.cap;
        total = nbig ? big.pref[nbig - 1] : 0;
    }
    const uint32_t nturns = turns * gridDim.x * kPW;
    const uint32_t grab = phase2 ? 1u : min(32u, (total + nturns - 1) / nturns);
    const unsigned long long deadline = run_deadline(rp);
    unsigned long long local = 0, local_d = 0, tb = 0;

    while (true) {
        uint32_t start = 0;
        if (lane == 0) start = past_deadline(rp, deadline) ? total : atomicAdd(cursor, grab);
        start = __shfl_sync(kFullMask, start, 0);
        if (start >= total) break;
        uint32_t pos = 0, end = 0;  // the smaller set's candidates left, as adjacency words
        uint32_t far = 0;           // the other set's core members
        if (uint32_t(lane) < grab && start + lane < total) {
            uint32_t q0 = pa + start + lane, ch = 0;
            if (phase2) {
                const uint32_t gi = start + lane;
                uint32_t lo = 0, hi = nbig - 1;  // first b with pref[b] > gi
                while (lo < hi) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (big.pref[mid] > gi) hi = mid; else lo = mid + 1;
                }
                ch = gi - (lo ? big.pref[lo - 1] : 0);
                q0 = big.q[lo];
            }
            uint32_t e = q0;
            for (int j = int(d) - 1; j >= 0; --j) {
                m[32 * j + lane] = s_vert[j][e];
                if (j > 0) e = s_par[j][e];
            }
            // a set's list, value bounds and window
            uint32_t off[2], deg[2], lo[2], hi[2], s0[2], e0[2];
            #pragma unroll
            for (int r = 0; r < 2; ++r) {
                const LevelPlan &L = r ? sT : sC;
                const uint32_t u = m[32 * (r ? jt : uint32_t(sC.jpos[0])) + lane];
                const uint2 inf = g.out_info[u];
                off[r] = inf.x;
                deg[r] = inf.y;
                lo[r] = L.sig_lo;
                hi[r] = kFullMask;
                for (uint32_t k = L.gt_mask & below; k; k &= k - 1) lo[r] = max(lo[r], m[32 * (__ffs(k) - 1) + lane] + 1);
                for (uint32_t k = L.lt_mask & below; k; k &= k - 1) hi[r] = min(hi[r], m[32 * (__ffs(k) - 1) + lane]);
                const uint32_t *l = g.adj + inf.x;
                s0[r] = lo[r] && inf.y && __ldg(l) < lo[r] ? lbound_own(g, false, u, l, inf.y, lo[r], loops) : 0;
                e0[r] = hi[r] != kFullMask ? lbound_own(g, false, u, l, inf.y, hi[r], loops) : inf.y;
                if (e0[r] < s0[r]) e0[r] = s0[r];
            }
            const uint32_t nc = e0[0] - s0[0], nt = e0[1] - s0[1];
            const uint32_t side = nt < nc ? 1u : 0u;  // whose vertices are gone through
            // matched vertices in C's window and list, and in T's where T is
            // the other set
            uint32_t in_c = 0, in_t = 0;
            for (uint32_t j = 0; j < d; ++j) {
                const uint32_t mj = m[32 * j + lane];
                if (mj >= lo[0] && mj < hi[0] && in_list(g, off[0], deg[0], mj)) in_c |= 1u << j;
                if (!side && mj >= lo[1] && mj < hi[1] && in_list(g, off[1], deg[1], mj)) in_t |= 1u << j;
            }
            if (!phase2) {
                local_d += nc - __popc(in_c);  // |C|
                if (TALLY) tb += 8ull * d + 16 + 32ull * d;
            }
            row[32 * kEMatched + lane] = side ? in_c : in_t;
            row[32 * kESide + lane] = side;
            row[32 * kECOff + lane] = off[0];
            row[32 * kECDeg + lane] = deg[0];
            row[32 * kETOff + lane] = off[1];
            row[32 * kETDeg + lane] = deg[1];
            row[32 * kEOLo + lane] = side ? lo[0] : lo[1];
            row[32 * kEOHi + lane] = side ? hi[0] : hi[1];
            row[32 * kEOBase + lane] = side ? off[0] + s0[0] : off[1] + s0[1];
            row[32 * kEOLen + lane] = side ? nc : nt;
            // the other set's entries below the core
            const uint32_t ob = side ? off[0] + s0[0] : off[1] + s0[1], on = side ? nc : nt;
            far = 0;
            if (ROWS && g.core_bits && on >= kECore && nc && nt && __ldg(g.adj + ob + on - kECore) >= g.core0)
                far = on - lbound(g.adj + ob, on, g.core0);
            if (ROWS) row[32 * kEONear + lane] = on - far;
            if (nc && nt) {
                pos = side ? off[1] + s0[1] : off[0] + s0[0];
                end = side ? off[1] + e0[1] : off[0] + e0[0];
            }
            if (phase2) {
                pos = min(pos + ch * kPK, end);
                end = min(pos + kPK, end);
            } else if (end - pos > split) {
                const uint32_t slot = list_place(big, end - pos);
                if (slot != kFullMask) {  // (a full list: this warp counts it)
                    big.q[slot] = q0;
                    big.len[slot] = end - pos;
                    end = pos;
                }
            }
        }
        while (true) {
            // ---- the next round: as many of the sets as fit, a prefix of the lanes
            const uint32_t take = min(end - pos, kPS);
            uint32_t incl = take;
            #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
                if (lane >= o) incl += y;
            }
            const uint32_t len = incl <= kPS ? take : 0u;
            const unsigned live = __ballot_sync(kFullMask, len != 0);
            if (!live) break;
            const uint32_t ftotal = __shfl_sync(kFullMask, incl, 31 - __clz(live));
            if (len) {
                const uint32_t r = __popc(live & lt), excl = incl - len;
                rec[r] = make_uint4(pos - excl, uint32_t(lane), 0, 0);
                starts[r] = excl;
                pos += len;
            }
            __syncwarp();
            uint32_t ns = 0;
            {
                const uint32_t my_start = uint32_t(lane) < uint32_t(__popc(live)) ? starts[lane] : kFullMask;
                uint32_t started = 0;
                for (uint32_t fstep = 0; fstep < ftotal; fstep += 32) {
                    const uint32_t rel = my_start - fstep;
                    const uint32_t bits = __reduce_or_sync(kFullMask, rel < 32u ? 1u << rel : 0u);
                    const uint4 rc = rec[started + __popc(bits & le) - 1];
                    started += __popc(bits);
                    const uint32_t f = fstep + lane, owner = rc.y;
                    bool ok = f < ftotal;
                    const uint32_t v = __ldg(g.adj + (rc.x + min(f, ftotal - 1)));
                    for (uint32_t j = 0; j < d; ++j) ok = ok && v != m[32 * j + owner];
                    const unsigned mk = __ballot_sync(kFullMask, ok);
                    if (ok) {
                        const uint32_t i = ns + __popc(mk & lt);
                        S[i] = v;
                        So[i] = uint8_t(owner);
                    }
                    ns += __popc(mk);
                    if (TALLY && f < ftotal) tb += 4;
                }
            }
            __syncwarp();
            // ---- the lanes' segments of S; from `cut` on (when short of the
            // end) the members are rows of the core
            uint32_t cut = ns, hi = ns;
            if (ROWS && __any_sync(kFullMask, far >= kECore)) {
                uint32_t lo = 0;
                for (uint32_t n = ns; n;) {  // first member whose column is >= lane
                    const uint32_t half = n >> 1;
                    if (So[lo + half] < lane) { lo += half + 1; n -= half + 1; }
                    else n = half;
                }
                hi = __shfl_down_sync(kFullMask, lo, 1);
                if (lane == 31) hi = ns;
                cut = hi;
                if (far >= kECore && hi - lo >= kECore) {
                    uint32_t c0 = lo;
                    for (uint32_t n = hi - lo; n;) {
                        const uint32_t half = n >> 1;
                        if (S[c0 + half] < g.core0) { c0 += half + 1; n -= half + 1; }
                        else n = half;
                    }
                    if (hi - c0 >= kECore) cut = c0;
                }
            }
            if (ROWS) {
                row[32 * kECut + lane] = cut;
                __syncwarp();
            }
            // ---- each vertex of the smaller sets with its possible partners
            for (uint32_t i0 = 0; i0 < ns; i0 += 32) {
                const uint32_t i = i0 + lane;
                uint32_t ilen = 0, ibase = 0, ioff = 0, ideg = 0, ow = 0, mode = 0;
                if (i < ns) {
                    ow = So[i];
                    const uint32_t v = S[i];
                    const uint32_t side = row[32 * kESide + ow];
                    const uint2 inf = g.out_info[v];
                    uint32_t a = 0, b = inf.y;  // the part of v's list that the order allows
                    if (side ? t_below : t_above) a = __ldg(g.bwd_out + v);
                    if (side ? t_above : t_below) b = __ldg(g.bwd_out + v);
                    // a core row's partners here are those below the core,
                    // where they are fewer than v's own neighbours
                    const uint32_t lenV = b - a, near = ROWS ? row[32 * kEONear + ow] : 0u;
                    const bool rowv = ROWS && i >= row[32 * kECut + ow] && near < lenV;
                    if (rowv) So[i] = uint8_t(ow | 128u);
                    const uint32_t lenO = rowv ? near : row[32 * kEOLen + ow];
                    mode = lenV < lenO ? 1u : 0u;
                    ilen = mode ? lenV : lenO;
                    ibase = mode ? inf.x + a : row[32 * kEOBase + ow];
                    ioff = mode ? row[32 * (side ? kECOff : kETOff) + ow] : inf.x;
                    ideg = mode ? row[32 * (side ? kECDeg : kETDeg) + ow] : inf.y;
                    mode |= side << 1;
                    if (TALLY) tb += 8;
                    // the matched vertices among v's partners, taken off here
                    // rather than compared with every hit
                    for (uint32_t k = ilen || rowv ? row[32 * kEMatched + ow] : 0u; k; k &= k - 1) {
                        const uint32_t mj = m[32 * (__ffs(k) - 1) + ow];
                        if (side ? t_below : t_above) { if (mj < v) continue; }
                        if (side ? t_above : t_below) { if (mj > v) continue; }
                        if (in_list(g, inf.x, inf.y, mj)) --local;
                    }
                }
                uint32_t iincl = ilen;
                #pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(kFullMask, iincl, o);
                    if (lane >= o) iincl += y;
                }
                const uint32_t itotal = __shfl_sync(kFullMask, iincl, 31);
                if (!itotal) continue;
                const unsigned ilive = __ballot_sync(kFullMask, ilen != 0);
                if (ilen) {
                    const uint32_t r = __popc(ilive & lt), excl = iincl - ilen;
                    rec[r] = make_uint4(ibase - excl, ow | (mode << 8) | (i << 16), ioff, ideg);
                    starts[r] = excl;
                }
                __syncwarp();
                const uint32_t my_start = uint32_t(lane) < uint32_t(__popc(ilive)) ? starts[lane] : kFullMask;
                uint32_t started = 0;
                for (uint32_t fstep = 0; fstep < itotal; fstep += 64) {
                    uint4 rc[2];
                    uint32_t wv[2], nb[2], bu[2];
                    Bucket bk[2];
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t rel = my_start - (fstep + 32 * h);
                        const uint32_t bits = __reduce_or_sync(kFullMask, rel < 32u ? 1u << rel : 0u);
                        rc[h] = rec[started + __popc(bits & le) - 1];
                        started += __popc(bits);
                        wv[h] = __ldg(g.adj + (rc[h].x + min(fstep + 32 * h + lane, itotal - 1)));
                    }
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        nb[h] = (rc[h].w + 3) >> 2;
                        bu[h] = tab_bucket(nb[h], wv[h]);
                        bk[h] = load_bucket(g.tab, rc[h].z, bu[h]);
                    }
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        bool ok = fstep + 32 * h + lane < itotal;
                        const uint32_t w = wv[h];
                        if (TALLY && ok) tb += 36;
                        if (ok && !bucket_has(bk[h], w)) ok = tab_continue(g.tab, rc[h].z, nb[h], bu[h], bk[h], w);
                        if (ok) {
                            const uint32_t l = rc[h].y & 255u;
                            ok = w >= row[32 * kEOLo + l] && w < row[32 * kEOHi + l];
                            if (ordered) {
                                const uint32_t v = S[rc[h].y >> 16];
                                const bool item_t = (rc[h].y >> 9) & 1u;
                                ok = ok && w != v;  // v lists itself only where there are self-loops
                                if (item_t ? t_below : t_above) ok = ok && w > v;
                                if (item_t ? t_above : t_below) ok = ok && w < v;
                            }
                            local += ok;
                        }
                    }
                }
                __syncwarp();
            }
            // ---- rows: the core members of both sets
            for (unsigned todo = ROWS ? __ballot_sync(kFullMask, cut < hi) : 0u; todo; todo &= todo - 1) {
                const int l = __ffs(todo) - 1;
                const uint32_t c0 = __shfl_sync(kFullMask, cut, l), ce = __shfl_sync(kFullMask, hi, l);
                const uint32_t nf = __shfl_sync(kFullMask, far, l), ob = row[32 * kEOBase + l] + row[32 * kEONear + l];
                const bool item_t = row[32 * kESide + l] != 0;
                const bool up = item_t ? t_below : t_above, down = item_t ? t_above : t_below;
                __syncwarp();
                Ob[lane] = 0;
                __syncwarp();
                for (uint32_t i = lane; i < nf; i += 32) {
                    const uint32_t u = __ldg(g.adj + ob + i) - g.core0;
                    atomicOr(&Ob[u >> 5], 1u << (u & 31));
                }
                __syncwarp();
                const uint32_t q0 = (__ldg(g.adj + ob) - g.core0) >> 7;  // words below the lowest member are empty
                for (uint32_t i = c0 + lane; i < ce; i += 32) {
                    if (!(So[i] & 128u)) continue;  // its own neighbours were walked
                    const uint32_t u = S[i] - g.core0, w0 = u >> 5;
                    const uint4 *rp4 = reinterpret_cast<const uint4 *>(g.core_bits + size_t(u) * (kCore / 32));
                    uint32_t n = 0;
                    if (!ordered) {
                        #pragma unroll 4
                        for (uint32_t q = q0; q < kCore / 128; ++q) {
                            const uint4 r4 = __ldg(rp4 + q), o4 = reinterpret_cast<const uint4 *>(Ob)[q];
                            n += __popc(r4.x & o4.x) + __popc(r4.y & o4.y) + __popc(r4.z & o4.z) + __popc(r4.w & o4.w);
                        }
                    } else {
                        // partners above v, below it, or all but v itself
                        const uint32_t own = 1u << (u & 31), ma = down ? 0u : ~(2 * own - 1), mb = up ? 0u : own - 1;
                        const uint32_t *rw = reinterpret_cast<const uint32_t *>(rp4);
                        for (uint32_t j = 4 * q0; j < kCore / 32; ++j) {
                            const uint32_t msk = j == w0 ? (ma | mb) : (j > w0 ? (down ? 0u : kFullMask) : (up ? 0u : kFullMask));
                            n += __popc(__ldg(rw + j) & Ob[j] & msk);
                        }
                    }
                    local += n;
                    if (TALLY) tb += 4 + kCore / 8;
                }
            }
            __syncwarp();
        }
        __syncwarp();
    }
    #pragma unroll
    for (int o = 16; o; o >>= 1) {
        local += __shfl_xor_sync(kFullMask, local, o);
        local_d += __shfl_xor_sync(kFullMask, local_d, o);
        if (TALLY) tb += __shfl_xor_sync(kFullMask, tb, o);
    }
    if (lane == 0) {
        if (local) atomicAdd(acc, local);
        if (local_d) atomicAdd(acc_d, local_d);
        if (TALLY && tb) atomicAdd(accb, tb);
    }
}

// ---- chunk planner ------------------------------------------------------
// Tile sums of the child bounds of parents [pa, pb).
__global__ void k_tile_sums(const uint32_t *__restrict__ ub, uint32_t pa, uint32_t pb,
                            uint32_t tile, uint64_t *__restrict__ tsum,
                            unsigned long long *__restrict__ tmax) {
    __shared__ unsigned long long red[32];
    const uint32_t ntiles = (pb - pa + tile - 1) / tile;
    for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const uint32_t b = pa + t * tile, e = min(b + tile, pb);
        unsigned long long s = 0;
        for (uint32_t i = b + threadIdx.x; i < e; i += blockDim.x) s += ub[i];
        #pragma unroll
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
        __syncthreads();
        if (threadIdx.x < 32) {
            s = threadIdx.x < blockDim.x / 32 ? red[threadIdx.x] : 0;
            #pragma unroll
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
            if (threadIdx.x == 0) {
                tsum[t] = s;
                atomicMax(tmax, s);
            }
        }
        __syncthreads();
    }
}

// Chunk boundaries (tile indices): tile t opens a chunk when
// floor(prefix(t) / cap_eff) differs from tile t-1's; with cap_eff = cap -
// (max tile sum) every chunk's bound sum stays within cap.  One block.
__global__ void __launch_bounds__(1024)
k_plan(const uint64_t *__restrict__ tsum, uint32_t ntiles, unsigned long long cap_eff,
       uint32_t *__restrict__ bounds, uint32_t *__restrict__ nb_out) {
    __shared__ unsigned long long ws[32];
    __shared__ uint32_t wf[32];
    __shared__ unsigned long long carry;
    __shared__ uint32_t nb;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) { carry = 0; nb = 0; }
    __syncthreads();
    for (uint32_t base = 0; base < ntiles; base += blockDim.x) {
        const uint32_t t = base + threadIdx.x;
        const unsigned long long v = t < ntiles ? tsum[t] : 0;
        // inclusive block scan of v
        unsigned long long x = v;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[warp] = x;
        __syncthreads();
        if (warp == 0) {
            unsigned long long w = lane < int(blockDim.x / 32) ? ws[lane] : 0;
            #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(kFull, w, o);
                if (lane >= o) w += y;
            }
            ws[lane] = w;
        }
        __syncthreads();
        const unsigned long long incl = x + (warp ? ws[warp - 1] : 0) + carry;
        const unsigned long long excl = incl - v;
        bool flag = false;
        if (t < ntiles) {
            if (t == 0) flag = true;
            else {
                const unsigned long long prev_excl = excl - tsum[t - 1];
                flag = (excl / cap_eff) != (prev_excl / cap_eff);
            }
        }
        // ordered compaction of the flags
        const unsigned m = __ballot_sync(kFull, flag);
        if (lane == 0) wf[warp] = __popc(m);
        __syncthreads();
        uint32_t before = 0, tot = 0;
        for (int w = 0; w < int(blockDim.x / 32); ++w) {
            if (w < warp) before += wf[w];
            tot += wf[w];
        }
        if (flag) bounds[nb + before + __popc(m & ((1u << lane) - 1))] = t;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = incl;
        if (threadIdx.x == 0) nb += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        bounds[nb] = ntiles;
        *nb_out = nb;
    }
}

int g_num_sms = 0;
int g_level_blocks[3] = {0, 0, 0};
int g_flat_blocks[3][kFolds] = {};  // blocks of k_level_flat<mode, fold> per SM by registers and threads
int g_fused_blocks[3] = {0, 0, 0};
int g_edge_blocks = 0;  // blocks of k_edges per SM by registers and threads
int g_pair_blocks[3] = {0, 0, 0};  // blocks of k_pairs<fold> per SM by registers and threads
// CUTS_LEVEL_KERNEL=warp selects the warp-per-parent form (A/B comparisons)
bool g_use_flat = true;

int launch_geometry() {
    if (g_num_sms) return CUTS_OK;
    int dev = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev));
    int b = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_level<kExpand>, kWarps * 32, 0));
    g_level_blocks[kExpand] = std::max(1, b) * g_num_sms;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_level<kCountMode>, kWarps * 32, 0));
    g_level_blocks[kCountMode] = std::max(1, b) * g_num_sms;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_level<kBytesMode>, kWarps * 32, 0));
    g_level_blocks[kBytesMode] = std::max(1, b) * g_num_sms;
    auto flat = [&](auto *kernel, int mode, int fold) -> int {
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, kFW * 32, 0));
        g_flat_blocks[mode][fold] = std::max(1, b);
        return CUTS_OK;
    };
    int rc = flat(k_level_flat<kExpand, kNoFold>, kExpand, kNoFold);
    if (!rc) rc = flat(k_level_flat<kCountMode, kNoFold>, kCountMode, kNoFold);
    if (!rc) rc = flat(k_level_flat<kCountMode, kPlainFold>, kCountMode, kPlainFold);
    if (!rc) rc = flat(k_level_flat<kCountMode, kOrbitFold>, kCountMode, kOrbitFold);
    if (!rc) rc = flat(k_level_flat<kCountMode, kPendants>, kCountMode, kPendants);
    if (!rc) rc = flat(k_level_flat<kCountMode, kTwins>, kCountMode, kTwins);
    if (!rc) rc = flat(k_level_flat<kBytesMode, kPlainFold>, kBytesMode, kPlainFold);
    if (rc) return rc;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_fused<kCountMode>, kZW * 32, 0));
    g_fused_blocks[kCountMode] = std::max(1, b) * g_num_sms;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_fused<kBytesMode>, kZW * 32, 0));
    g_fused_blocks[kBytesMode] = std::max(1, b) * g_num_sms;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_pairs<kNoWeights, false, false>, kPW * 32, 0));
    g_pair_blocks[kNoWeights] = std::max(1, b);
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_pairs<kWeights, false, false>, kPW * 32, 0));
    g_pair_blocks[kWeights] = std::max(1, b);
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_pairs<kEvenWeights, false, false>, kPW * 32, 0));
    g_pair_blocks[kEvenWeights] = std::max(1, b);
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_edges<true, false>, kPW * 32, 0));
    g_edge_blocks = std::max(1, b);
    const char *kv = std::getenv("CUTS_LEVEL_KERNEL");
    g_use_flat = !(kv && std::strcmp(kv, "warp") == 0);
    return CUTS_OK;
}

// Dynamic shared memory of one k_level_flat block, and the blocks that fill
// the GPU at that size (227 KB per SM, 1 KB of it per block for the system).
uint32_t flat_smem(int mode, uint32_t lvl, uint32_t nj) {
    return 4 * kFW * flat_words(lvl, nj, mode == kExpand);
}
uint32_t flat_grid(int mode, int fold, uint32_t smem) {
    const uint32_t fixed = 3 * uint32_t(sizeof(LevelPlan)) + 16 * kMaxK + 1024;
    const uint32_t by_smem = 227u * 1024u / (smem + fixed);
    return std::max(1u, std::min(uint32_t(g_flat_blocks[mode][fold]), by_smem)) * uint32_t(g_num_sms);
}

// u32 scratch slots
enum : int { kSlotN0 = 0, kSlotErr = 1, kSlotNb = 2, kSlotOver = 3, kSlotStop = 4, kSlotOut = 8, kSlotCursor = 32, kSlots = 64 };
constexpr int kU64Stamp = 5;  // d_u64 slot: device clock at the start of a budgeted run
constexpr int kU64Scratch = 8;  // d_u64 slots 8..10: counts of the bytes pass (discarded)
constexpr int kU64Pair = 6;     // d_u64 slot: level k-2 size of a pendant-pair count
constexpr int kU64Roots = 7;    // d_u64 slot: sum of the roots' child bounds
constexpr int kU64Big = 11;     // d_u64 slots 11, 12: the fused count's deferred parents
constexpr int kU64Slots = 16;

// Counters of one root slice of a chain (launches queued without the host
// reading level sizes in between).
struct ChainSlice {
    unsigned long long bound[kMaxK];  // child bounds of L_{lvl-1}, by lvl
    unsigned long long big[2];        // the fused count's deferred parents
    uint32_t out_n[kMaxK];
    uint32_t cursor[kMaxK];
};
constexpr uint32_t kChainSlices = 16;  // root slices per chain

// Device scratch and its pinned mirror: the u64 slots, the u32 slots and the
// chain's slices, cleared and read in one piece.
constexpr size_t kCtlHead = sizeof(unsigned long long) * kU64Slots + sizeof(uint32_t) * kSlots;
constexpr size_t kCtlBytes = kCtlHead + sizeof(ChainSlice) * kChainSlices;
ChainSlice *chain_slices(unsigned long long *u64) {
    return reinterpret_cast<ChainSlice *>(reinterpret_cast<char *>(u64) + kCtlHead);
}

}  // namespace

// ---- upload -------------------------------------------------------------

// Allocates a DeviceGraph, builds its layout on the device from CSR arrays
// in host memory (layout.cu) and the engine's scratch.
static int device_graph_build(uint32_t n, const uint64_t *out_off, const uint32_t *out_adj,
                              const uint64_t *in_off, const uint32_t *in_adj, int sym_hint, bool validate,
                              int device, DeviceGraph **out) {
    *out = nullptr;
    CK(cudaSetDevice(device));
    auto *g = new DeviceGraph();
    g->device = device;
    auto fail = [&](cudaError_t e, const char *what) {
        device_graph_free(g);
        return set_error(CUTS_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
    };
    cudaError_t e;
    if ((e = cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking))) return fail(e, "stream");
    {
        // the trie arena and the layout's scratch come from the device's
        // default pool; keep up to 32 GB of freed blocks there, so a graph
        // built after another one reuses its memory instead of mapping anew
        cudaMemPool_t pool = nullptr;
        if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
            uint64_t keep = 32ull << 30;
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        }
    }
    int rc = device_layout(n, out_off, out_adj, in_off, in_adj, sym_hint, validate, *g);
    if (rc) {
        device_graph_free(g);
        return rc;
    }
    if ((e = cudaMalloc(&g->d_u64, kCtlBytes))) return fail(e, "scratch");
    g->d_u32 = reinterpret_cast<uint32_t *>(g->d_u64 + kU64Slots);
    if ((e = cudaMalloc(&g->d_plan, sizeof(RunParams)))) return fail(e, "scratch");
    if ((e = cudaMallocHost(&g->h_u64, kCtlBytes))) return fail(e, "pinned");
    g->h_u32 = reinterpret_cast<uint32_t *>(g->h_u64 + kU64Slots);
    if ((e = cudaMallocHost(&g->h_plan, sizeof(RunParams)))) return fail(e, "pinned");
    if ((e = cudaEventCreate(&g->ev0)) || (e = cudaEventCreate(&g->ev1))) return fail(e, "event");
    if ((e = cudaStreamSynchronize(g->stream))) return fail(e, "upload sync");
    // default arena: proportional to the graph, within [256 MB, 64 GB] and
    // at most 60% of the free memory
    size_t freeb = 0, totb = 0;
    cudaMemGetInfo(&freeb, &totb);
    double want = 384.0 * double(g->arcs) + 64.0 * n;
    want = std::max(want, 256.0 * (1 << 20));
    want = std::min(want, 64.0 * (1ull << 30));
    want = std::min(want, 0.6 * double(freeb));
    g->arena_bytes = size_t(want);
    g->arena_default = g->arena_bytes;
    g->tab_limit = (freeb - std::min(freeb, g->arena_bytes)) / 2;
    // CUTS_TABLES=0 does without the tables' memory (lists are searched)
    const char *tb = std::getenv("CUTS_TABLES");
    if (tb && tb[0] == '0') g->tab_limit = 0;
    *out = g;
    return CUTS_OK;
}

int device_graph_upload(const HostGraph &hg, int device, DeviceGraph **out) {
    return device_graph_build(hg.n, hg.out_off.data(), hg.out_adj.data(),
                              hg.symmetric ? nullptr : hg.in_off.data(), hg.symmetric ? nullptr : hg.in_adj.data(),
                              hg.symmetric ? 1 : 0, false, device, out);
}

int device_graph_from_csr(uint32_t n, const uint64_t *out_off, const uint32_t *out_adj, const uint64_t *in_off,
                          const uint32_t *in_adj, int device, DeviceGraph **out) {
    return device_graph_build(n, out_off, out_adj, in_off, in_adj, -1, true, device, out);
}

void device_graph_free(DeviceGraph *g) {
    if (!g) return;
    cudaSetDevice(g->device);
    if (g->stream) {
        // the arena and the layout's arrays go back to the device's pool,
        // after the work queued on the graph's stream
        if (g->in_info && g->in_info != g->out_info) cudaFreeAsync(g->in_info, g->stream);
        for (void *p : {static_cast<void *>(g->arena), static_cast<void *>(g->out_info),
                        static_cast<void *>(g->adj), static_cast<void *>(g->bwd_out),
                        static_cast<void *>(g->core_bits), static_cast<void *>(g->tab),
                        static_cast<void *>(g->d_orig)})
            if (p) cudaFreeAsync(p, g->stream);
        cudaStreamSynchronize(g->stream);
    }
    cudaFree(g->d_u64);
    cudaFree(g->d_plan);
    cudaFree(g->d_tiles);
    cudaFree(g->d_bounds);
    cudaFree(g->batch_vsorted);
    cudaFree(g->batch_pref);
    cudaFreeHost(g->h_u64);
    cudaFreeHost(g->h_plan);
    cudaFreeHost(g->h_bounds);
    if (g->ev0) cudaEventDestroy(g->ev0);
    if (g->ev1) cudaEventDestroy(g->ev1);
    if (g->stream) cudaStreamDestroy(g->stream);
    delete g;
}

// ---- driver -----------------------------------------------------------------

namespace {

struct Run {
    DeviceGraph &g;
    DevView view;
    RunParams *hp;        // pinned host copy
    RunParams *dp;        // device copy
    uint32_t k;
    uint64_t cap;         // entries per stored level >= 1
    uint32_t grain;
    bool bytes_mode;
    CountResult &res;
    bool dump = false;
    bool profile = false;
    double budget_ms = 0;
    std::chrono::steady_clock::time_point t_start = std::chrono::steady_clock::now();
    std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> marks;
    FILE *dump_file = nullptr;
    const Query *query = nullptr;
    uint64_t dumped = 0;

    int sync() {
        CK(cudaStreamSynchronize(g.stream));
        return CUTS_OK;
    }

    int ensure_tiles(size_t ntiles) {
        if (ntiles + 1 <= g.tiles_cap) return CUTS_OK;
        size_t nc = std::max(ntiles + 1, g.tiles_cap * 2);
        cudaFree(g.d_tiles);
        cudaFree(g.d_bounds);
        cudaFreeHost(g.h_bounds);
        g.d_tiles = nullptr; g.d_bounds = nullptr; g.h_bounds = nullptr; g.tiles_cap = 0;
        CK(cudaMalloc(&g.d_tiles, sizeof(uint64_t) * nc));
        CK(cudaMalloc(&g.d_bounds, sizeof(uint32_t) * nc));
        CK(cudaMallocHost(&g.h_bounds, sizeof(uint32_t) * nc));
        g.tiles_cap = nc;
        return CUTS_OK;
    }

    // Splits parents [pa, pb) of L_{lvl-1} into chunks whose child bounds fit cap.
    int plan_chunks(uint32_t lvl, uint32_t pa, uint32_t pb, std::vector<uint32_t> &cuts) {
        cuts.clear();
        if (uint64_t(pb - pa) * g.max_deg <= cap) { cuts = {pa, pb}; return CUTS_OK; }
        uint64_t tile = std::min<uint64_t>(kTile, cap / (2ull * std::max<uint32_t>(g.max_deg, 1)));
        if (tile == 0)
            return set_error(CUTS_ERR_CAPACITY, "level capacity below twice the maximum degree");
        const uint32_t ntiles = uint32_t((uint64_t(pb - pa) + tile - 1) / tile);
        int rc = ensure_tiles(ntiles);
        if (rc) return rc;
        CK(cudaMemsetAsync(g.d_u64 + 1, 0, sizeof(unsigned long long), g.stream));
        const uint32_t blocks = std::min<uint32_t>(ntiles, uint32_t(g_num_sms) * 16);
        k_tile_sums<<<blocks, 256, 0, g.stream>>>(hp->ub[lvl - 1], pa, pb, uint32_t(tile), g.d_tiles,
                                                 g.d_u64 + 1);
        CK(cudaMemcpyAsync(g.h_u64 + 1, g.d_u64 + 1, sizeof(unsigned long long), cudaMemcpyDeviceToHost, g.stream));
        res.launches++;
        int r2 = sync();
        if (r2) return r2;
        const unsigned long long tmax = g.h_u64[1];
        const unsigned long long cap_eff = cap - tmax;
        k_plan<<<1, 1024, 0, g.stream>>>(g.d_tiles, ntiles, cap_eff, g.d_bounds, g.d_u32 + kSlotNb);
        res.launches++;
        CK(cudaMemcpyAsync(g.h_u32 + kSlotNb, g.d_u32 + kSlotNb, sizeof(uint32_t), cudaMemcpyDeviceToHost, g.stream));
        r2 = sync();
        if (r2) return r2;
        const uint32_t nb = g.h_u32[kSlotNb];
        CK(cudaMemcpyAsync(g.h_bounds, g.d_bounds, sizeof(uint32_t) * (nb + 1), cudaMemcpyDeviceToHost, g.stream));
        r2 = sync();
        if (r2) return r2;
        for (uint32_t c = 0; c <= nb; ++c)
            cuts.push_back(uint32_t(std::min<uint64_t>(pa + uint64_t(g.h_bounds[c]) * tile, pb)));
        return CUTS_OK;
    }

    // A host-known range of parents.
    static Parents known(uint32_t a, uint32_t b) { return Parents{nullptr, a, b, 0, 1, nullptr, 0, nullptr, 0}; }

    // Level `lvl` over the given parents; `most` bounds their number.  A chain
    // launch (cs: its slice's counters on the device) uses counters of its own.
    int launch_level(int mode, uint32_t lvl, const Parents &par, uint32_t most, ChainSlice *cs = nullptr) {
        uint32_t *out_n = cs ? cs->out_n + lvl : g.d_u32 + kSlotOut + lvl;
        uint32_t *cursor = cs ? cs->cursor + lvl : g.d_u32 + kSlotCursor;
        if (!cs) {
            CK(cudaMemsetAsync(cursor, 0, sizeof(uint32_t), g.stream));
            if (mode == kExpand) CK(cudaMemsetAsync(out_n, 0, sizeof(uint32_t), g.stream));
        }
        const uint32_t work = most;
        const uint32_t pa = par.a, pb = par.b;  // the warp-per-parent form: host-known ranges only
        const LevelPlan &L = hp->plan.lv[lvl];
        const bool flat = g_use_flat && L.nj <= uint32_t(kFJ);
        const int fold = mode == kBytesMode   ? kPlainFold
                         : mode == kExpand    ? kNoFold
                         : L.fold2            ? kPendants
                         : L.twin             ? kTwins
                         : !L.fold            ? kNoFold
                         : hp->plan.lv[lvl + 1].ofold ? kOrbitFold
                                                      : kPlainFold;
        const uint32_t smem = flat ? flat_smem(mode, lvl, L.nj) : 0;
        // the flattened form deals out single parents when there are few, but
        // for a closed form, which walks no candidates
        const bool closed = mode == kCountMode && L.closed_form;
        const uint32_t warps_needed = !flat ? (work + grain - 1) / grain : closed ? (work - 1) / 32 + 1 : work;
        const uint32_t wpb = flat ? kFW : kWarps;
        uint32_t blocks = std::min<uint32_t>(flat ? flat_grid(mode, fold, smem) : uint32_t(g_level_blocks[mode]),
                                             (warps_needed + wpb - 1) / wpb);
        blocks = std::max<uint32_t>(blocks, 1);
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        if (profile) {
            CK(cudaEventCreate(&e0));
            CK(cudaEventCreate(&e1));
            CK(cudaEventRecord(e0, g.stream));
        }
        if (flat) {
            auto go = [&](auto *kernel, uint32_t ocap, unsigned long long *a1, unsigned long long *a2,
                          unsigned long long *a3) {
                kernel<<<blocks, kFW * 32, smem, g.stream>>>(view, dp, lvl, flat_turns(g.max_deg), par, cursor, out_n, ocap,
                                                           g.d_u32 + kSlotErr, a1, a2, a3);
            };
            auto count = [&](auto *kernel) { go(kernel, 0, g.d_u64, g.d_u64 + 3, g.d_u64 + kU64Pair); };
            if (mode == kExpand)
                go(k_level_flat<kExpand, kNoFold>, uint32_t(cap), cs && lvl + 1 < uint32_t(kMaxK) ? cs->bound + lvl + 1 : nullptr,
                   nullptr, nullptr);
            else if (mode == kBytesMode) go(k_level_flat<kBytesMode, kPlainFold>, 0, g.d_u64 + 2, nullptr, nullptr);
            else if (fold == kPlainFold) count(k_level_flat<kCountMode, kPlainFold>);
            else if (fold == kOrbitFold) count(k_level_flat<kCountMode, kOrbitFold>);
            else if (fold == kPendants) count(k_level_flat<kCountMode, kPendants>);
            else if (fold == kTwins) count(k_level_flat<kCountMode, kTwins>);
            else count(k_level_flat<kCountMode, kNoFold>);
        } else if (mode == kExpand)
            k_level<kExpand><<<blocks, kWarps * 32, 0, g.stream>>>(view, dp, lvl, pa, pb, grain,
                cursor, out_n, uint32_t(cap), g.d_u32 + kSlotErr, g.d_u64);
        else if (mode == kCountMode)
            k_level<kCountMode><<<blocks, kWarps * 32, 0, g.stream>>>(view, dp, lvl, pa, pb, grain,
                cursor, out_n, 0, g.d_u32 + kSlotErr, g.d_u64);
        else
            k_level<kBytesMode><<<blocks, kWarps * 32, 0, g.stream>>>(view, dp, lvl, pa, pb, grain,
                cursor, out_n, 0, g.d_u32 + kSlotErr, g.d_u64 + 2);
        CK(cudaGetLastError());
        if (profile) {
            CK(cudaEventRecord(e1, g.stream));
            marks.push_back({mode, {e0, e1}});
        }
        res.launches++;
        return CUTS_OK;
    }

    // The fused count of levels p and p+1 over the given parents of L_{p-1}:
    // phase 1 over the parents, then a scan of the parents it deferred and
    // phase 2 over their pieces (k_pairs) or groups (k_fused).
    int launch_fused(int mode, uint32_t p, const Parents &par, uint32_t most, ChainSlice *cs = nullptr) {
        uint32_t *cur1 = cs ? cs->cursor + p : g.d_u32 + kSlotCursor;
        uint32_t *cur2 = cs ? cs->cursor + p + 1 : g.d_u32 + kSlotCursor + 1;
        unsigned long long *bn = cs ? cs->big : g.d_u64 + kU64Big;
        if (!cs) {
            CK(cudaMemsetAsync(cur1, 0, 2 * sizeof(uint32_t), g.stream));
            CK(cudaMemsetAsync(bn, 0, 2 * sizeof(unsigned long long), g.stream));
        }
        // CUTS_FUSE_SPLIT=<n> sets the deferral threshold (tests use small values)
        uint32_t split = g.fuse_split;
        const char *es = std::getenv("CUTS_FUSE_SPLIT");
        if (es) split = uint32_t(std::strtoul(es, nullptr, 10));
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        if (profile) {
            CK(cudaEventCreate(&e0));
            CK(cudaEventCreate(&e1));
            CK(cudaEventRecord(e0, g.stream));
        }
        // counting; the bytes pass of a pair plan runs the same launches with
        // their byte tally on and the counts sent to scratch slots
        const bool tal = mode == kBytesMode;
        unsigned long long *acc = tal ? g.d_u64 + kU64Scratch : g.d_u64;
        unsigned long long *acc_c = tal ? g.d_u64 + kU64Scratch + 1 : g.d_u64 + 3;
        unsigned long long *acc_p = tal ? g.d_u64 + kU64Scratch + 2 : g.d_u64 + 4;
        if (hp->pairs) {
            PairBig pb;
            pb.n = bn;
            pb.cap = hp->fuse_big_cap;
            pb.max_pieces = list_pieces();
            pb.q = hp->fuse_big;
            pb.len = pb.q + pb.cap;
            pb.pref = pb.len + pb.cap;
            pb.bits = pb.pref + pb.cap;
            split = es || g.fuse_split ? std::min(split, kPS) : kPS;
            // parents that are roots (p = 1) have their own list's window for S,
            // so dealing them out in pieces repeats no test, and it keeps a
            // hub's pairs from one warp: 64 there (triangle, 4M / 40M: 512 14.6 ms,
            // 128 12.7 ms, 64 9.3 ms).  Not where the longest list is little more
            // (3 of them; 4 with an order, whose windows are about half of the
            // lists): the second launch and its bitmaps took 40 of 72 us of a root
            // slice (triangle, symmetry breaking, 2,000 vertices / 80,000 edges in
            // 17 slices 1.21 -> 0.60 ms, 5,000 / 250,000 at once 0.21 -> 0.14; 3,000
            // / 300,000 plain, lists of 250, would lose 0.54 -> 0.60)
            const uint32_t few = (hp->plan.lv[p].gt_mask | hp->plan.lv[p].lt_mask ? 4 : 3) * kPK;
            if (p == 1 && (es || g.fuse_split || g.max_deg > few)) split = std::min(split, kPK);
            const LevelPlan &LP = hp->plan.lv[p], &LC = hp->plan.lv[p + 1];
            const int fold = !LC.fold ? kNoWeights
                             : pair_same_set(LP, LC, p) && pair_even(hp->plan.lv[p + 2], p) ? kEvenWeights
                                                                                          : kWeights;
            const uint32_t smem = 4 * kPW * pair_words(p, hp->plan.lv[p].nj);
            const uint32_t fixed = 3 * uint32_t(sizeof(LevelPlan)) + 16 * kMaxK + 1024;
            const uint32_t full = std::max(1u, std::min(uint32_t(g_pair_blocks[fold]), 227u * 1024u / (smem + fixed))) *
                                  uint32_t(g_num_sms);
            const uint32_t blocks = std::max<uint32_t>(1, std::min<uint32_t>(full, (most + kPW - 1) / kPW));
            auto go = [&](auto *kernel, uint32_t grid, uint32_t phase, uint32_t *cur) {
                kernel<<<grid, kPW * 32, smem, g.stream>>>(view, dp, p, par, phase, split, cur, pb, acc, acc_c, acc_p,
                                                          tal ? g.d_u64 + 2 : nullptr);
            };
            auto phase = [&](uint32_t grid, uint32_t ph, uint32_t *cur) {
                // (the byte tally is not timed: one instance, for graphs with and without loops)
                auto pick = [&](auto *none, auto *any, auto *even) {
                    go(fold == kNoWeights ? none : fold == kWeights ? any : even, grid, ph, cur);
                };
                if (tal) pick(k_pairs<kNoWeights, true, true>, k_pairs<kWeights, true, true>, k_pairs<kWeights, true, true>);
                else if (g.loops)
                    pick(k_pairs<kNoWeights, false, true>, k_pairs<kWeights, false, true>, k_pairs<kEvenWeights, false, true>);
                else
                    pick(k_pairs<kNoWeights, false, false>, k_pairs<kWeights, false, false>, k_pairs<kEvenWeights, false, false>);
            };
            phase(blocks, 1, cur1);
            CK(cudaGetLastError());
            res.launches++;
            // (a turn is of `most` parents dealt out as in the kernel, at most)
            const uint32_t turn = std::min(32u, std::max(1u, most / (4 * blocks * kPW)));
            if (pair_defers(p, split, g.max_deg, uint64_t(turn) * g.max_deg)) {
                k_fused_scan<<<1, 1024, 0, g.stream>>>(pb.n, pb.cap, pb.len, kPK, pb.pref);
                k_pair_bits<kNoWeights><<<full, kPW * 32, smem, g.stream>>>(view, dp, p, pb);
                phase(full, 2, cur2);
                CK(cudaGetLastError());
                res.launches += 3;
            }
        } else {
            const uint32_t blocks = std::max<uint32_t>(1, std::min<uint32_t>(uint32_t(g_fused_blocks[mode]),
                                                                             (most + kZW - 1) / kZW));
            if (!es && !split) split = kBigS;
            FusedBig fb;
            fb.n = bn;
            fb.cap = hp->fuse_big_cap;
            fb.gi = hp->fuse_big;
            fb.soff = fb.gi + fb.cap;
            fb.ns = fb.soff + fb.cap;
            fb.pref = fb.ns + fb.cap;
            fb.pool = fb.pref + fb.cap;
            fb.pool_words = hp->fuse_pool_words;
            if (tal) {
                k_fused<kBytesMode><<<blocks, kZW * 32, 0, g.stream>>>(view, dp, p, par, 1, split, cur1,
                    hp->fuse_scratch, hp->fuse_stride, fb, g.d_u64 + 2, nullptr, nullptr);
                CK(cudaGetLastError());
                res.launches++;
            } else {
                k_fused<kCountMode><<<blocks, kZW * 32, 0, g.stream>>>(view, dp, p, par, 1, split, cur1,
                    hp->fuse_scratch, hp->fuse_stride, fb, acc, acc_c, acc_p);
                CK(cudaGetLastError());
                k_fused_scan<<<1, 1024, 0, g.stream>>>(fb.n, fb.cap, fb.ns, 32, fb.pref);
                k_fused<kCountMode><<<uint32_t(g_fused_blocks[kCountMode]), kZW * 32, 0, g.stream>>>(
                    view, dp, p, par, 2, split, cur2, hp->fuse_scratch, hp->fuse_stride, fb, acc, acc_c, acc_p);
                CK(cudaGetLastError());
                res.launches += 3;
            }
        }
        if (profile) {
            CK(cudaEventRecord(e1, g.stream));
            marks.push_back({kCountMode, {e0, e1}});
        }
        return CUTS_OK;
    }

    // Levels d = k-2 and k-1 over the given parents of L_{d-1} as edges between
    // two sets, then the pieces of the sets it listed.
    int launch_edges(int mode, uint32_t d, const Parents &par, uint32_t most, ChainSlice *cs = nullptr) {
        uint32_t *cur1 = cs ? cs->cursor + d : g.d_u32 + kSlotCursor;
        uint32_t *cur2 = cs ? cs->cursor + d + 1 : g.d_u32 + kSlotCursor + 1;
        PairBig pb;
        pb.n = cs ? cs->big : g.d_u64 + kU64Big;
        pb.cap = hp->fuse_big_cap;
        pb.max_pieces = list_pieces();
        pb.q = hp->fuse_big;
        pb.len = pb.q + pb.cap;
        pb.pref = pb.len + pb.cap;
        pb.bits = nullptr;
        if (!cs) {
            CK(cudaMemsetAsync(cur1, 0, 2 * sizeof(uint32_t), g.stream));
            CK(cudaMemsetAsync(pb.n, 0, 2 * sizeof(unsigned long long), g.stream));
        }
        const bool tal = mode == kBytesMode;
        unsigned long long *a1 = tal ? g.d_u64 + kU64Scratch : g.d_u64;
        unsigned long long *ad = tal ? g.d_u64 + kU64Scratch + 1 : g.d_u64 + 4;
        const uint32_t smem = 4 * kPW * edge_words(d);
        const uint32_t fixed = 2 * uint32_t(sizeof(LevelPlan)) + 16 * kMaxK + 1024;
        const uint32_t full = std::max(1u, std::min(uint32_t(g_edge_blocks), 227u * 1024u / (smem + fixed))) *
                              uint32_t(g_num_sms);
        const uint32_t blocks = std::max<uint32_t>(1, std::min<uint32_t>(full, (most + kPW - 1) / kPW));
        const uint32_t split = kPK;
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        if (profile) {
            CK(cudaEventCreate(&e0));
            CK(cudaEventCreate(&e1));
            CK(cudaEventRecord(e0, g.stream));
        }
        auto phase = [&](uint32_t grid, uint32_t ph, uint32_t *cur) {
            auto go = [&](auto *kernel) {
                kernel<<<grid, kPW * 32, smem, g.stream>>>(view, dp, d, flat_turns(g.max_deg), par, ph, split, cur, pb,
                                                          a1, ad, g.d_u64 + 2);
            };
            // core rows pay where lists are longer than the core: 64 mixed
            // queries on 200,000 vertices of up to ~1,500 neighbours 79 -> 61
            // ms (sets of 8 core members on; 24: 69 ms), but the 5-cycle of at
            // most 619 neighbours 48 -> 52 ms for the larger kernel
            if (g.max_deg >= kCore) tal ? go(k_edges<true, true>) : go(k_edges<true, false>);
            else tal ? go(k_edges<false, true>) : go(k_edges<false, false>);
        };
        phase(blocks, 1, cur1);
        CK(cudaGetLastError());
        res.launches++;
        if (g.max_deg > split) {  // else no set can be listed
            k_fused_scan<<<1, 1024, 0, g.stream>>>(pb.n, pb.cap, pb.len, kPK, pb.pref);
            phase(full, 2, cur2);
            CK(cudaGetLastError());
            res.launches += 2;
        }
        if (profile) {
            CK(cudaEventRecord(e1, g.stream));
            marks.push_back({kCountMode, {e0, e1}});
        }
        return CUTS_OK;
    }

    // Sums the profiled launch times per kernel (after a sync).
    void collect_profile() {
        for (auto &m : marks) {
            float t = 0;
            cudaEventElapsedTime(&t, m.second.first, m.second.second);
            if (m.first == kExpand) { res.expand_ms += t; res.expand_launches++; }
            else { res.last_level_ms += t; res.last_level_launches++; }
            cudaEventDestroy(m.second.first);
            cudaEventDestroy(m.second.second);
        }
        marks.clear();
    }

    uint32_t count_level() const {
        if (k >= 4 && hp->plan.lv[k - 3].fold2) return k - 3;
        return k >= 3 && (hp->plan.lv[k - 2].fold || hp->plan.lv[k - 2].twin) ? k - 2 : k - 1;
    }

    // Expands parents [pa, pb) of L_{lvl-1}, depth first by chunks.
    int expand(uint32_t lvl, uint32_t pa, uint32_t pb) {
        if (pb <= pa) return CUTS_OK;
        // the last level is counted; with a folded plan, level k-2 counts both;
        // with a fused plan, the counting kernel runs one level earlier
        const uint32_t count_lvl = count_level();
        if (!dump && k >= 3 && hp->plan.lv[count_lvl].fuse && lvl == count_lvl - 1)
            return launch_fused(bytes_mode ? kBytesMode : kCountMode, lvl, known(pa, pb), pb - pa);
        if (!dump && hp->edges && lvl == count_lvl - 1)
            return launch_edges(bytes_mode ? kBytesMode : kCountMode, lvl, known(pa, pb), pb - pa);
        if (lvl == count_lvl && !dump)
            return launch_level(bytes_mode ? kBytesMode : kCountMode, lvl, known(pa, pb), pb - pa);
        std::vector<uint32_t> cuts;
        int rc = plan_chunks(lvl, pa, pb, cuts);
        if (rc) return rc;
        for (size_t c = 0; c + 1 < cuts.size(); ++c) {
            const uint32_t a = cuts[c], b = cuts[c + 1];
            if (b <= a) continue;
            if (budget_ms > 0 &&
                std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count() >
                    budget_ms)
                return set_error(CUTS_ERR_BUDGET, "time budget exhausted");
            rc = launch_level(kExpand, lvl, known(a, b), b - a);
            if (rc) return rc;
            res.chunks++;
            CK(cudaMemcpyAsync(g.h_u32 + kSlotOut + lvl, g.d_u32 + kSlotOut + lvl, sizeof(uint32_t),
                               cudaMemcpyDeviceToHost, g.stream));
            CK(cudaMemcpyAsync(g.h_u32 + kSlotErr, g.d_u32 + kSlotErr, 3 * sizeof(uint32_t),
                               cudaMemcpyDeviceToHost, g.stream));
            rc = sync();
            if (rc) return rc;
            if (g.h_u32[kSlotOver]) return set_error(CUTS_ERR_BUDGET, "time budget exhausted");
            const uint32_t nout = g.h_u32[kSlotOut + lvl];
            if (g.h_u32[kSlotErr] || nout > cap)
                return set_error(CUTS_ERR_CAPACITY, "level " + std::to_string(lvl) + " overflowed its capacity");
            res.level_sizes[lvl] += nout;
            rc = (dump && lvl + 1 == k) ? write_rows(nout) : expand(lvl + 1, 0, nout);
            if (rc) return rc;
        }
        return CUTS_OK;
    }

    // True when every level of the plan runs in kernels that take their
    // parents' number from the device.
    bool can_chain(uint32_t nshards) const {
        if (dump || bytes_mode || !g_use_flat) return false;
        // (the roots' lists alone do not fit level 1)
        if (hp->stored >= 2 && g.arcs / nshards > cap) return false;
        for (uint32_t i = 1; i <= count_level(); ++i)
            if (hp->plan.lv[i].nj > uint32_t(kFJ)) return false;
        return true;
    }

    // All levels of all root slices queued without waiting: each launch reads
    // its parents' number on the device, so a count costs one wait instead of
    // one per level and slice (the GPU is idle between a level's end and the
    // next launch for a wait and a copy).  4-cycle on 10,000 vertices 174 ->
    // 119 us, twelve 4-6 vertex queries on 3,000 vertices 2.87 -> 2.10 ms.  A level whose children may not fit is left to
    // expand(), which cuts it into chunks.
    int chain(uint32_t chunks);

    // Dump: materialise the nout complete matches of L_{k-1} in pieces and
    // write one ans.txt line per match, pairs in matching order
    // (util.cpp:53-74).
    int write_rows(uint32_t nout);
};

}  // namespace

namespace {

// Rows of complete matches: row r = the path of L_{k-1} entry first + r,
// k words in matching order.
__global__ void k_materialize(const RunParams *__restrict__ rp, uint32_t first, uint32_t nrows,
                              uint32_t *__restrict__ rows) {
    const uint32_t k = rp->plan.k;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += gridDim.x * blockDim.x) {
        uint32_t e = first + r;
        uint32_t *row = rows + size_t(r) * k;
        for (int lv = int(k) - 1; lv >= 0; --lv) {
            row[lv] = rp->vert[lv][e];
            if (lv > 0) e = rp->par[lv][e];
        }
    }
}

constexpr uint32_t kDumpRows = 1u << 22;  // rows materialised per piece

// True when the fused count of levels p and p + 1 runs in k_pairs: a symmetric
// graph (its pairs are unordered) with membership tables, no list of level p + 1 on p itself beyond the pair's, and no plain fold
// whose list or window moves with the vertex at p.  Everything else keeps
// k_fused.  CUTS_FUSE_WALK=0 keeps k_fused always (A/B comparisons).
bool pairs_plan(const DeviceGraph &g, const Plan &plan, uint32_t p) {
    if (!g.symmetric || !g.tab || g.max_deg >= (1u << 31)) return false;
    const LevelPlan &Lc = plan.lv[p + 1];
    const LevelPlan &Lf = plan.lv[p + 2 < plan.k ? p + 2 : p + 1];
    for (uint32_t t = 0; t < Lc.nj; ++t)
        if (((Lc.fuse_extra >> t) & 1u) && Lc.jpos[t] == p) return false;
    if (Lc.fold && !Lf.ofold && (Lf.jpos[0] == p || (((Lf.gt_mask | Lf.lt_mask) >> p) & 1u))) return false;
    const char *w = std::getenv("CUTS_FUSE_WALK");
    return !(w && w[0] == '0');
}

// True when an orbit fold's weights look a vertex below position `upto` up in
// an orbit vertex's list (orbit_base, orbit_weight).
bool orbit_tests(const LevelPlan &F, uint32_t upto, bool loops) {
    if (loops) return true;
    for (uint32_t x = 0; x < upto; ++x)
        if ((F.ofold >> x) & 1u)
            if (~(F.oguar[x] | (1u << x)) & ((1u << upto) - 1)) return true;
    return false;
}

// CUTS_NO_FUSE=1: fusion off process-wide (A/B comparisons)
bool no_fuse_env() {
    const char *nf = std::getenv("CUTS_NO_FUSE");
    return nf && nf[0] == '1';
}

// Carves the arena for `stored` levels and uploads the run parameters.
int prepare(DeviceGraph &g, const Query &q, uint32_t flags, uint32_t stored, RunParams *&hp,
            RunParams *&dp, uint64_t &cap) {
    const uint32_t k = q.k;
    hp = static_cast<RunParams *>(g.h_plan);
    std::memset(hp, 0, sizeof(RunParams));
    int rc = build_plan(q, g.symmetric, flags, hp->plan);
    if (rc) return rc;
    // the arena before the membership tables: these do without memory
    if (!g.arena) {
        cudaError_t e = cudaMallocAsync(&g.arena, g.arena_bytes, g.stream);
        if (e != cudaSuccess) {
            g.arena = nullptr;
            return set_error(CUTS_ERR_NOMEM, "arena allocation failed: " + std::string(cudaGetErrorString(e)));
        }
    }
    const bool counting = stored == k - 1;
    const bool env_nofuse = no_fuse_env();
    if (k >= 3 && hp->plan.lv[k - 1].ofold) {
        // the orbit fold needs its weight evaluated by the flattened or the
        // fused counting kernel, in 32 bits; otherwise break Q's symmetry
        const bool fused = hp->plan.lv[k - 2].fuse && !env_nofuse;
        const bool flat = g_use_flat && hp->plan.lv[k - 2].nj <= uint32_t(kFJ);
        const bool fits = uint64_t(__builtin_popcount(hp->plan.lv[k - 1].ofold)) *
                              std::max<uint32_t>(g.max_deg, 1) < (1ull << 32);
        if (!counting || !(fused || flat) || !fits) {
            rc = build_plan(q, g.symmetric, flags | CUTS_FLAG_NO_ORBIT_FOLD, hp->plan);
            if (rc) return rc;
        }
    }
    hp->plan.data_loops = g.loops ? 1u : 0u;
    if (k >= 4 && hp->plan.lv[k - 3].fold2) {
        // the pendant pair is counted by the flattened kernel at level k-3;
        // where that kernel does not run, plan without it
        if (!counting || !g_use_flat || hp->plan.lv[k - 3].nj > uint32_t(kFJ)) {
            rc = build_plan(q, g.symmetric, flags | CUTS_FLAG_NO_PAIR_FOLD |
                                                (hp->plan.lv[k - 1].ofold ? 0u : CUTS_FLAG_NO_ORBIT_FOLD),
                            hp->plan);
            if (rc) return rc;
            hp->plan.data_loops = g.loops ? 1u : 0u;
        } else {
            stored = k - 3;  // levels k-3.. are counted, not stored
        }
    }
    if (k >= 3 && hp->plan.lv[k - 2].fold) {
        // the folded count runs in the flattened or the fused kernel only
        const bool fused_here = hp->plan.lv[k - 2].fuse != 0;
        if (!fused_here && (!g_use_flat || hp->plan.lv[k - 2].nj > uint32_t(kFJ))) hp->plan.lv[k - 2].fold = 0;
        else if (counting) stored = k - 2;  // level k-2 is counted, not stored
    }
    if (k >= 4 && hp->plan.lv[k - 2].twin) {
        // twins are counted by the flattened kernel at level k-2
        if (counting && g_use_flat && hp->plan.lv[k - 2].nj <= uint32_t(kFJ)) stored = k - 2;
        else hp->plan.lv[k - 2].twin = 0;
    }
    // the counted level and, when fused, the one before it are not stored
    const uint32_t cl = (k >= 3 && hp->plan.lv[k - 2].fold) ? k - 2 : k - 1;
    if (k >= 3 && !hp->plan.lv[k - 2].fold) hp->plan.lv[k - 2].fuse = 0;
    if (!counting || env_nofuse)
        for (uint32_t i = 0; i < k; ++i) hp->plan.lv[i].fuse = 0;
    const bool fuse = counting && k >= 3 && hp->plan.lv[cl].fuse;
    if (fuse) stored = cl - 1;
    // levels k-2 and k-1 as edges between two candidate sets, where the id
    // bounds stand for k-2's signature (degree-ranked ids) and the lists have
    // tables; not where the caller wants level k-2 materialised
    bool edges = counting && !fuse && edges_counted(flags) && g_use_flat && g.ranked && edges_shape(hp->plan);
    if (edges) {
        if ((rc = device_tables(g))) return rc;
        edges = g.tab != nullptr;
    }
    hp->edges = edges ? 1u : 0u;
    if (edges) stored = k - 2;
    // on a symmetric graph with degree-ranked ids the vertices of degree d or
    // more are a suffix of the ids: the signature is a compare of ids, not a
    // gather of the candidate's degree
    if (g.symmetric && g.ranked)
        for (uint32_t i = 1; i < k; ++i) {
            LevelPlan &L = hp->plan.lv[i];
            if (!L.check_sig) continue;
            const uint32_t d = std::max(L.qin, L.qout);
            L.sig_lo = g.n - uint32_t(d < g.stats.out_ge.size() ? g.stats.out_ge[d] : 0);
            L.check_sig = 0;
        }
    // membership tables, for the levels that test candidates in other lists
    // or matched vertices in a list that a closed form counts (a graph whose
    // counts are edges and stars does without: their build is 0.3 ms for 20M
    // arcs, an edge count 0.1)
    bool tests = false;
    // positions below upto that L's list may hold for all the plan knows
    auto unknown = [&](const LevelPlan &L, uint32_t guar, uint32_t upto) {
        const uint32_t known = guar | (g.loops ? 0u : 1u << L.jpos[0]);
        return (~known & ((1u << upto) - 1)) != 0;
    };
    for (uint32_t i = 1; i < k && i <= stored; ++i) {
        const LevelPlan &L = hp->plan.lv[i];
        if (fuse && i >= stored) break;
        tests = tests || L.nj >= 2;
        if (!counting) continue;
        const LevelPlan &F = hp->plan.lv[k - 1];
        if (i == k - 1 && L.closed_form) tests = tests || unknown(L, L.guar_mask, i);
        else if (L.fold2) tests = tests || unknown(hp->plan.lv[i + 1], hp->plan.lv[i + 1].guar1, i + 1) || unknown(F, F.guar_mask, i + 1);
        else if (L.fold && F.ofold) tests = tests || orbit_tests(F, i, g.loops);
        else if (L.fold) tests = tests || unknown(F, F.guar_mask, i + 1);
    }
    if ((tests || (fuse && g.symmetric)) && (rc = device_tables(g))) return rc;
    hp->pairs = fuse && pairs_plan(g, hp->plan, cl - 1);
    hp->stored = stored;
    // before a fused count of levels p = cl - 1 and cl, the entries of
    // level p - 1 record where their vertex sits in its list
    hp->pos_lvl = (fuse && cl >= 3) ? cl - 2 : 0xffffffffu;
    // L_0: vert + ub (n entries each); L_1..L_{stored-1}: vert + par + ub
    const uint64_t n = g.n;
    const uint64_t l0_bytes = ((8 * n + 255) / 256) * 256 + 256;
    // fused kernel: one scratch row per resident warp, as long as the longest list
    uint64_t fuse_bytes = 0, big_bytes = 0;
    if (fuse && hp->pairs) {
        // deferred parents: index, length and prefix sum, and two core bitmaps
        // each; a parent beyond the list's capacity is counted where it is found
        const uint64_t per = 3 + kCore / 16;
        hp->fuse_big_cap = uint32_t(std::max<uint64_t>(64, std::min<uint64_t>(1u << 17, g.arena_bytes / 64 / (4 * per))));
        big_bytes = (4 * per * hp->fuse_big_cap + 255) / 256 * 256;
        fuse_bytes = big_bytes;
    } else if (edges) {
        // listed sets: parent, length and prefix sum each (beyond the list's
        // capacity a set is counted where it is found)
        hp->fuse_big_cap = uint32_t(std::max<uint64_t>(64, std::min<uint64_t>(1u << 18, g.arena_bytes / 64 / 12)));
        big_bytes = (12ull * hp->fuse_big_cap + 255) / 256 * 256;
        fuse_bytes = big_bytes;
    } else if (fuse) {
        hp->fuse_stride = ((std::max<uint32_t>(g.max_deg, 1) + 31) / 32) * 32;
        fuse_bytes = uint64_t(g_fused_blocks[kCountMode] > g_fused_blocks[kBytesMode] ? g_fused_blocks[kCountMode]
                                                                                      : g_fused_blocks[kBytesMode]) *
                     kZW * hp->fuse_stride * 4;
        // deferred parents: four arrays of cap words and a pool of saved
        // candidate sets (1/32 of the arena, 1M..16M words)
        hp->fuse_big_cap = 1u << 17;
        const uint64_t pool = std::min<uint64_t>(16ull << 20, std::max<uint64_t>(1ull << 20, g.arena_bytes / 128));
        hp->fuse_pool_words = uint32_t(std::max<uint64_t>(pool, 2ull * hp->fuse_stride));
        big_bytes = 256 + 16ull * hp->fuse_big_cap + 4ull * hp->fuse_pool_words;
        big_bytes = (big_bytes + 255) / 256 * 256;
        fuse_bytes += big_bytes;
    }
    cap = 0;
    if (g.arena_bytes < l0_bytes + fuse_bytes)
        return set_error(CUTS_ERR_NOMEM, "arena smaller than the root level and scratch");
    if (fuse || edges) {
        char *const end = static_cast<char *>(g.arena) + (g.arena_bytes & ~uint64_t(255));
        hp->fuse_scratch = reinterpret_cast<uint32_t *>(end - fuse_bytes);
        hp->fuse_big = reinterpret_cast<uint32_t *>(end - big_bytes);
    }
    if (stored >= 2) {
        cap = (g.arena_bytes - l0_bytes - fuse_bytes) / (12ull * (stored - 1));
        cap = std::min<uint64_t>(cap, (1ull << 31) - 64);
        if (g.level_cap_req) cap = std::min<uint64_t>(cap, g.level_cap_req);
        cap &= ~uint64_t(63);
        if (cap < 2ull * std::max<uint32_t>(g.max_deg, 1))
            return set_error(CUTS_ERR_CAPACITY, "level capacity below twice the maximum degree");
    }
    char *base = static_cast<char *>(g.arena);
    hp->vert[0] = reinterpret_cast<uint32_t *>(base);
    hp->ub[0] = reinterpret_cast<uint32_t *>(base + ((4 * n + 255) / 256) * 256);
    hp->par[0] = nullptr;
    char *cur = base + l0_bytes;
    for (uint32_t i = 1; i < stored; ++i) {
        hp->vert[i] = reinterpret_cast<uint32_t *>(cur); cur += 4 * cap;
        hp->par[i] = reinterpret_cast<uint32_t *>(cur); cur += 4 * cap;
        hp->ub[i] = reinterpret_cast<uint32_t *>(cur); cur += 4 * cap;
    }
    hp->budget_ns = 0;
    hp->stamp = g.d_u64 + kU64Stamp;
    hp->over = g.d_u32 + kSlotOver;
    dp = static_cast<RunParams *>(g.d_plan);
    CK(cudaMemcpyAsync(dp, hp, sizeof(RunParams), cudaMemcpyHostToDevice, g.stream));
    return CUTS_OK;
}

// Level 0 into L_0; returns |L_0|.  For a chain of `slices` root slices it is
// only queued (|L_0| stays on the device), the slices' counters cleared.
int run_roots(DeviceGraph &g, Run &run, uint32_t shard, uint32_t nshards, uint32_t &n0, uint32_t slices = 0) {
    CK(cudaMemsetAsync(g.d_u64, 0, kCtlHead + sizeof(ChainSlice) * std::min(slices, kChainSlices), g.stream));
    n0 = 0;
    if (!g.n) return CUTS_OK;
    const uint32_t threads = 256;
    const uint32_t blocks = std::min<uint32_t>((g.n + threads - 1) / threads, uint32_t(g_num_sms) * 8);
    k_roots<<<blocks, threads, 0, g.stream>>>(run.view, run.dp, shard, nshards, g.d_u32 + kSlotN0, g.d_u64 + kU64Roots);
    CK(cudaGetLastError());
    run.res.launches++;
    if (slices) return CUTS_OK;  // a chain reads the number on the device
    CK(cudaMemcpyAsync(g.h_u32 + kSlotN0, g.d_u32 + kSlotN0, sizeof(uint32_t), cudaMemcpyDeviceToHost, g.stream));
    int rc = run.sync();
    if (rc) return rc;
    n0 = g.h_u32[kSlotN0];
    return CUTS_OK;
}

// Root slices, as the reference's trunks (host_funcs.cu:66-72).
int run_slices(Run &run, uint32_t n0, uint32_t chunks) {
    const uint32_t slice = uint32_t((uint64_t(n0) - 1) / chunks + 1);
    for (uint32_t s = 0; s < chunks; ++s) {
        const uint64_t a = uint64_t(s) * slice;
        if (a >= n0) break;
        int rc = run.expand(1, uint32_t(a), uint32_t(std::min<uint64_t>(a + slice, n0)));
        if (rc) return rc;
    }
    return CUTS_OK;
}

int Run::chain(uint32_t chunks) {
    const uint32_t cl = count_level();
    const bool fused = k >= 3 && hp->plan.lv[cl].fuse;
    const uint32_t last = fused || hp->edges ? cl - 1 : cl;  // level of the counting launch
    // bounds on the levels' sizes, for the launches' grids
    std::vector<uint64_t> most(last + 1, 0);
    most[0] = g.n;
    for (uint32_t i = 1; i < last; ++i) most[i] = std::min<uint64_t>(cap, most[i - 1] * std::max<uint32_t>(g.max_deg, 1));
    ChainSlice *const ds = chain_slices(g.d_u64), *const hs = chain_slices(g.h_u64);
    int rc = CUTS_OK;
    for (uint32_t s0 = 0; s0 < chunks;) {
        const uint32_t ns = std::min(chunks - s0, kChainSlices);
        if (s0) CK(cudaMemsetAsync(ds, 0, sizeof(ChainSlice) * ns, g.stream));
        for (uint32_t i = 0; i < ns; ++i) {
            for (uint32_t lvl = 1; lvl <= last; ++lvl) {
                const bool exp = lvl < last;
                Parents par{lvl == 1 ? g.d_u32 + kSlotN0 : ds[i].out_n + lvl - 1, 0, 0, lvl == 1 ? s0 + i : 0,
                            lvl == 1 ? chunks : 1,
                            !exp ? nullptr : lvl == 1 ? g.d_u64 + kU64Roots : ds[i].bound + lvl, cap,
                            g.d_u32 + kSlotStop, ((i + 1) << 8) | lvl};
                const uint32_t m = uint32_t(std::min<uint64_t>(lvl == 1 ? most[0] / chunks + 1 : most[lvl - 1], UINT32_MAX));
                if (!exp && fused) rc = launch_fused(kCountMode, lvl, par, m, ds + i);
                else if (!exp && hp->edges) rc = launch_edges(kCountMode, lvl, par, m, ds + i);
                else rc = launch_level(exp ? kExpand : kCountMode, lvl, par, m, ds + i);
                if (rc) return rc;
            }
        }
        CK(cudaEventRecord(g.ev1, g.stream));
        CK(cudaMemcpyAsync(g.h_u64, g.d_u64, kCtlHead + sizeof(ChainSlice) * ns, cudaMemcpyDeviceToHost, g.stream));
        if ((rc = sync())) return rc;
        const uint32_t n0 = g.h_u32[kSlotN0], stop = g.h_u32[kSlotStop];
        res.level_sizes[0] = n0;
        const uint32_t done = stop ? (stop >> 8) - 1 : ns;  // slices before the one that stopped
        for (uint32_t i = 0; i < std::min(done + 1, ns); ++i)
            for (uint32_t lvl = 1; lvl < (i < done ? last : (stop & 255u)); ++lvl) {
                res.level_sizes[lvl] += hs[i].out_n[lvl];
                res.chunks++;
            }
        if (g.h_u32[kSlotOver]) return set_error(CUTS_ERR_BUDGET, "time budget exhausted");
        if (g.h_u32[kSlotErr]) return set_error(CUTS_ERR_CAPACITY, "a level overflowed its capacity");
        if (!n0) break;
        if (!stop) {
            s0 += ns;
            if (uint64_t(s0) * ((n0 - 1) / chunks + 1) >= n0) break;  // the remaining slices are empty
            continue;
        }
        // slice s0 + done from level `lvl` on in chunks, and the slices after
        // it one by one: queued again, each that does not fit would cost the
        // empty launches of the slices behind it (the 4-cycle on 5,000 vertices
        // in 1,000 slices, capacity 16,384 entries: 299 ms, 46 this way)
        const uint32_t lvl = stop & 255u, per = (n0 - 1) / chunks + 1;
        if (lvl > 1 && (rc = expand(lvl, 0, hs[done].out_n[lvl - 1]))) return rc;
        for (uint64_t s = s0 + done + (lvl > 1); s < chunks && s * per < n0; ++s)
            if ((rc = expand(1, uint32_t(s * per), uint32_t(std::min<uint64_t>((s + 1) * per, n0))))) return rc;
        CK(cudaEventRecord(g.ev1, g.stream));
        CK(cudaMemcpyAsync(g.h_u64, g.d_u64, kCtlHead, cudaMemcpyDeviceToHost, g.stream));
        return sync();
    }
    return CUTS_OK;
}

}  // namespace

int Run::write_rows(uint32_t nout) {
    const uint32_t k = this->k;
    const std::vector<uint32_t> &order = query->order;
    uint32_t *d_rows = nullptr, *h_rows = nullptr;
    const uint32_t piece = std::min<uint32_t>(nout, kDumpRows);
    CK(cudaMalloc(&d_rows, sizeof(uint32_t) * size_t(piece) * k));
    cudaError_t e = cudaMallocHost(&h_rows, sizeof(uint32_t) * size_t(piece) * k);
    if (e != cudaSuccess) {
        cudaFree(d_rows);
        return set_error(CUTS_ERR_NOMEM, "pinned dump buffer");
    }
    std::vector<char> text;
    int rc = CUTS_OK;
    for (uint32_t first = 0; first < nout && rc == CUTS_OK; first += piece) {
        const uint32_t nr = std::min(piece, nout - first);
        k_materialize<<<std::max<uint32_t>(1, std::min<uint32_t>((nr + 255) / 256, 4096)), 256, 0, g.stream>>>(
            dp, first, nr, d_rows);
        res.launches++;
        if ((e = cudaMemcpyAsync(h_rows, d_rows, sizeof(uint32_t) * size_t(nr) * k, cudaMemcpyDeviceToHost,
                                 g.stream)) != cudaSuccess ||
            (e = cudaStreamSynchronize(g.stream)) != cudaSuccess) {
            rc = set_error(CUTS_ERR_CUDA, std::string("dump copy: ") + cudaGetErrorString(e));
            break;
        }
        // text, formatted in parallel: each thread a contiguous block of
        // rows into its own part of the buffer, written in row order
        const size_t per_row = size_t(k) * 24 + 1;
        text.resize(size_t(nr) * per_row + 16);
        const int nth = std::max(1, std::min(omp_get_max_threads(), int((nr + 4095) / 4096)));
        std::vector<size_t> used(size_t(nth), 0);
        #pragma omp parallel for schedule(static, 1) num_threads(nth)
        for (int t = 0; t < nth; ++t) {
            const uint32_t r0 = uint32_t(uint64_t(nr) * t / nth), r1 = uint32_t(uint64_t(nr) * (t + 1) / nth);
            char *const b0 = text.data() + size_t(r0) * per_row;
            char *w = b0, *const end = text.data() + size_t(r1) * per_row;
            for (uint32_t r = r0; r < r1; ++r) {
                const uint32_t *row = h_rows + size_t(r) * k;
                for (uint32_t j = 0; j < k; ++j) {
                    *w++ = '(';
                    w = std::to_chars(w, end, order[j]).ptr;
                    *w++ = ',';
                    w = std::to_chars(w, end, g.orig.empty() ? row[j] : g.orig[row[j]]).ptr;
                    *w++ = ')';
                }
                *w++ = '\n';
            }
            used[size_t(t)] = size_t(w - b0);
        }
        for (int t = 0; t < nth && rc == CUTS_OK; ++t) {
            const char *b0 = text.data() + size_t(uint64_t(nr) * t / nth) * per_row;
            if (std::fwrite(b0, 1, used[size_t(t)], dump_file) != used[size_t(t)])
                rc = set_error(CUTS_ERR_IO, std::string("short write to the dump file: ") + std::strerror(errno));
        }
        dumped += nr;
    }
    cudaFree(d_rows);
    cudaFreeHost(h_rows);
    return rc;
}

bool edges_counted(uint32_t flags) { return !(flags & CUTS_FLAG_NO_FUSE) && !no_fuse_env(); }

int device_count(DeviceGraph &g, const Query &q, const CountOptions &opt, CountResult &res) {
    res = CountResult();
    if (opt.chunks == 0) return set_error(CUTS_ERR_ARG, "chunks must be >= 1");
    if (opt.nshards == 0 || opt.shard >= opt.nshards) return set_error(CUTS_ERR_ARG, "bad shard");
    CK(cudaSetDevice(g.device));
    int rc = launch_geometry();
    if (rc) return rc;
    const uint32_t k = q.k;
    RunParams *hp = nullptr, *dp = nullptr;
    uint64_t cap = 0;
    const bool had_tables = g.tab != nullptr;
    rc = prepare(g, q, opt.flags, k - 1, hp, dp, cap);
    if (rc) return rc;
    Run run{g, graph_view(g), hp, dp, k, cap, 4, false, res};
    run.profile = opt.profile;
    run.budget_ms = opt.budget_ms;
    if (opt.budget_ms > 0) {  // the kernels' own deadline (device time from k_roots)
        hp->budget_ns = (unsigned long long)(opt.budget_ms * 1e6);
        CK(cudaMemcpyAsync(dp, hp, sizeof(RunParams), cudaMemcpyHostToDevice, g.stream));
    }
    // the time starts here, or with the tables that this count had built
    if (had_tables || !g.tab) CK(cudaEventRecord(g.ev0, g.stream));
    uint32_t n0 = 0;
    if (k >= 2 && g.n && run.can_chain(opt.nshards)) {
        rc = run_roots(g, run, opt.shard, opt.nshards, n0, opt.chunks);
        if (rc) return rc;
        rc = run.chain(opt.chunks);
        if (rc) return rc;
        n0 = g.h_u32[kSlotN0];
    } else {
        rc = run_roots(g, run, opt.shard, opt.nshards, n0);
        if (rc) return rc;
        res.level_sizes[0] = n0;
        if (k >= 2 && n0 > 0) {
            rc = run_slices(run, n0, opt.chunks);
            if (rc) return rc;
        }
        CK(cudaEventRecord(g.ev1, g.stream));
        CK(cudaMemcpyAsync(g.h_u64, g.d_u64, kCtlHead, cudaMemcpyDeviceToHost, g.stream));
        rc = run.sync();
        if (rc) return rc;
    }
    run.collect_profile();
    CK(cudaEventElapsedTime(&res.ms, g.ev0, g.ev1));
    if (g.h_u32[kSlotOver]) return set_error(CUTS_ERR_BUDGET, "time budget exhausted");
    const uint64_t raw = k >= 2 ? uint64_t(g.h_u64[0]) : 0;
    res.level_sizes[k - 1] = k >= 2 ? raw : n0;
    if (k >= 4 && hp->plan.lv[k - 3].fold2) {  // level k-3 counted both pendant levels
        res.level_sizes[k - 3] = g.h_u64[3];
        res.level_sizes[k - 2] = g.h_u64[kU64Pair];
    }
    if (k >= 3 && (hp->plan.lv[k - 2].fold || hp->plan.lv[k - 2].twin)) {
        res.level_sizes[k - 2] = g.h_u64[3];
    }
    if (k >= 3) {
        const uint32_t cl = hp->plan.lv[k - 2].fold ? k - 2 : k - 1;
        if (hp->plan.lv[cl].fuse || hp->edges)  // the level before the counted one, counted with it
            res.level_sizes[cl - 1] = g.h_u64[4];
    }
    res.count = raw * hp->plan.aut;
    if (opt.want_bytes && k >= 2 && n0 > 0) {
        // untimed second pass: algorithmic bytes of the last-level kernel
        CountResult tmp;
        if (hp->budget_ns) {  // the bytes pass runs to the end
            hp->budget_ns = 0;
            CK(cudaMemcpyAsync(dp, hp, sizeof(RunParams), cudaMemcpyHostToDevice, g.stream));
        }
        Run r2{g, run.view, hp, dp, k, cap, 4, true, tmp};
        CK(cudaMemsetAsync(g.d_u64 + 2, 0, sizeof(unsigned long long), g.stream));
        rc = run_slices(r2, n0, opt.chunks);
        if (rc) return rc;
        CK(cudaMemcpyAsync(g.h_u64 + 2, g.d_u64 + 2, sizeof(unsigned long long), cudaMemcpyDeviceToHost, g.stream));
        rc = r2.sync();
        if (rc) return rc;
        res.last_level_bytes = g.h_u64[2];
    }
    return CUTS_OK;
}

int device_dump(DeviceGraph &g, const Query &q, const char *path, uint64_t *lines, uint32_t shard,
                uint32_t nshards) {
    if (nshards == 0 || shard >= nshards) return set_error(CUTS_ERR_ARG, "bad shard");
    CK(cudaSetDevice(g.device));
    int rc = launch_geometry();
    if (rc) return rc;
    const uint32_t k = q.k;
    FILE *f = std::fopen(path, "wb");
    if (!f) return set_error(CUTS_ERR_IO, std::string("cannot write ") + path);
    std::unique_ptr<FILE, int (*)(FILE *)> hold(f, std::fclose);
    if (lines) *lines = 0;
    if (k < 2) return CUTS_OK;  // the reference dumps nothing for a 1-vertex query
    RunParams *hp = nullptr, *dp = nullptr;
    uint64_t cap = 0;
    rc = prepare(g, q, CUTS_FLAG_NO_CLOSED_FORM, k, hp, dp, cap);
    if (rc) return rc;
    if ((rc = host_orig(g))) return rc;
    CountResult res;
    Run run{g, graph_view(g), hp, dp, k, cap, 4, false, res};
    run.dump = true;
    run.dump_file = f;
    run.query = &q;
    uint32_t n0 = 0;
    rc = run_roots(g, run, shard, nshards, n0);
    if (rc) return rc;
    if (n0 > 0) {
        rc = run_slices(run, n0, 1);
        if (rc) return rc;
    }
    if (lines) *lines = run.dumped;
    return CUTS_OK;
}

}  // namespace cuts
