// layout.cu -- the data graph's device layout, built on the device.
//
// The caller's CSR (host memory, the reference's format after parsing:
// graph.cpp:29-57 builds the same out/in lists) is copied to the device as
// is; validation, the symmetry check, the degree ranking of vertex ids, the
// padded layout and the per-list sort all run there, so a resident graph
// costs one host-to-device copy plus a few milliseconds of kernels instead
// of host passes over every arc.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_segmented_sort.cuh>

#include "device_util.cuh"
#include "engine.hpp"

namespace cuts {
namespace {

constexpr uint32_t kPad = 0xffffffffu;

__device__ __forceinline__ uint32_t padded(uint32_t len) { return (len + 3u) & ~3u; }

// Walks every vertex's list: body(v, thread, threads) by one warp per vertex,
// or, for lists of more than kLongList entries, by the whole block after its
// warps are through with theirs.  One warp per vertex alone leaves a
// 20,000-entry hub's 625 dependent steps as the launch's tail: the symmetry
// check of 1M vertices / 20M arcs took 4.06 ms that way, 0.77 ms this way.
// len(v) gives the list's length.
constexpr uint32_t kLongList = 512;
constexpr uint32_t kLongQueue = 512;

template <class Len, class Body>
__device__ __forceinline__ void per_list(uint32_t n, Len len, Body body) {
    __shared__ uint32_t q[kLongQueue];
    __shared__ uint32_t qn;
    if (threadIdx.x == 0) qn = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += warps) {
        uint32_t slot = kLongQueue;
        if (len(v) > kLongList) {
            if (lane == 0) slot = atomicAdd(&qn, 1u);
            slot = __shfl_sync(kFullMask, slot, 0);
            if (slot < kLongQueue && lane == 0) q[slot] = v;
        }
        if (slot >= kLongQueue) body(v, lane, 32u);
    }
    __syncthreads();
    const uint32_t nq = min(qn, kLongQueue);
    for (uint32_t i = 0; i < nq; ++i) body(q[i], threadIdx.x, blockDim.x);
}

// The lane whose part of a warp's concatenated sequence holds element w
// (incl: inclusive scan of the lanes' lengths).
__device__ __forceinline__ uint32_t run_owner(uint32_t incl, uint32_t w) {
    uint32_t owner = 0;
    #pragma unroll
    for (int step = 16; step; step >>= 1) {
        const uint32_t probe = __shfl_sync(kFullMask, incl, int(owner + step - 1));
        if (probe <= w) owner += step;
    }
    return min(owner, 31u);
}

// Offsets monotone and within the arc count; every list strictly increasing
// with ids below n.  flag |= 1 (offsets) or 2 (lists).
__global__ void k_validate(uint32_t n, uint64_t m, const uint64_t *__restrict__ off,
                           const uint32_t *__restrict__ adj, uint32_t *__restrict__ flag) {
    bool bad = false;
    per_list(
        n,
        [&](uint32_t v) {
            const uint64_t a = off[v], b = off[v + 1];
            if (b < a || b > m) return 0u;
            return uint32_t(min(b - a, uint64_t(0xffffffffu)));
        },
        [&](uint32_t v, uint32_t t, uint32_t nt) {
            const uint64_t a = off[v], b = off[v + 1];
            if (b < a || b > m) {
                if (t == 0) atomicOr(flag, 1u);
                return;
            }
            for (uint64_t x = a + t; x < b; x += nt) {
                const uint32_t id = adj[x];
                if (id >= n || (x > a && id <= adj[x - 1])) bad = true;
            }
        });
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 2u);
}

// flag |= 1 where the two arrays differ.
template <class T>
__global__ void k_differ(uint64_t cnt, const T *__restrict__ a, const T *__restrict__ b,
                         uint32_t *__restrict__ flag) {
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < cnt; i += uint64_t(gridDim.x) * blockDim.x)
        if (a[i] != b[i]) atomicOr(flag, 1u);
}

// Every arc u -> v has its reverse.  Order the vertices by (degree, id).
// With no repeated arc (the lists were checked strictly increasing),
// reversal maps the arcs that go down in that order one-to-one into the
// arcs that go up, once every down arc's reverse is found; the two sets then
// have equal sizes exactly when every up arc's reverse exists too.  So only
// a down arc u -> v is searched for, as u in v's list -- the shorter of the
// two: a hub's list is never searched -- and the arcs going up and down are
// counted into updown[0] / updown[1] (a self-loop is its own reverse).
__global__ void k_symmetric(uint32_t n, const uint64_t *__restrict__ off, const uint32_t *__restrict__ adj,
                            uint32_t *__restrict__ flag, unsigned long long *__restrict__ updown) {
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long up = 0, down = 0;
    auto len = [&](uint32_t u) { return uint32_t(off[u + 1] - off[u]); };
    per_list(n, len, [&](uint32_t u, uint32_t t, uint32_t nt) {
        const uint64_t a = off[u], b = off[u + 1];
        const uint64_t du = b - a;
        for (uint64_t x = a + t; x < b; x += nt) {
            const uint32_t v = adj[x];
            if (v == u) continue;
            const uint64_t lo0 = off[v], hi0 = off[v + 1], dv = hi0 - lo0;
            if (!(dv < du || (dv == du && v < u))) {
                ++up;
                continue;
            }
            ++down;
            uint64_t lo = lo0, hi = hi0;
            while (lo < hi) {
                const uint64_t mid = (lo + hi) >> 1;
                if (adj[mid] < u) lo = mid + 1; else hi = mid;
            }
            if (lo == hi0 || adj[lo] != u) atomicOr(flag, 1u);
        }
    });
    for (int sh = 16; sh; sh >>= 1) {
        up += __shfl_xor_sync(0xffffffffu, up, sh);
        down += __shfl_xor_sync(0xffffffffu, down, sh);
    }
    if (lane == 0 && (up | down)) {
        atomicAdd(updown, up);
        atomicAdd(updown + 1, down);
    }
}

// Sort keys (degree << 32 | vertex): ascending degree, then id.
__global__ void k_keys(uint32_t n, const uint64_t *__restrict__ ooff, const uint64_t *__restrict__ ioff,
                       unsigned long long *__restrict__ keys) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        uint64_t d = ooff[v + 1] - ooff[v];
        if (ioff) d += ioff[v + 1] - ioff[v];
        keys[v] = (d << 32) | v;
    }
}

// orig[d] = the vertex of rank d; rank[v] = its rank.
__global__ void k_ranks(uint32_t n, const unsigned long long *__restrict__ sorted, uint32_t *__restrict__ orig,
                        uint32_t *__restrict__ rank) {
    for (uint32_t d = blockIdx.x * blockDim.x + threadIdx.x; d < n; d += gridDim.x * blockDim.x) {
        const uint32_t v = uint32_t(sorted[d] & 0xffffffffull);
        orig[d] = v;
        rank[v] = d;
    }
}

// Padded length of device vertex d's list (entry n = 0, for the scan's total).
__global__ void k_plen(uint32_t n, const uint32_t *__restrict__ orig, const uint64_t *__restrict__ off,
                       unsigned long long *__restrict__ plen) {
    for (uint32_t d = blockIdx.x * blockDim.x + threadIdx.x; d <= n; d += gridDim.x * blockDim.x) {
        if (d == n) { plen[d] = 0; continue; }
        const uint32_t v = orig ? orig[d] : d;
        plen[d] = padded(uint32_t(off[v + 1] - off[v]));
    }
}

// info[d] = {base + start, length}; segment bounds for the sort.
__global__ void k_info(uint32_t n, const uint32_t *__restrict__ orig, const uint64_t *__restrict__ off,
                       const unsigned long long *__restrict__ start, uint32_t base, uint2 *__restrict__ info,
                       uint32_t *__restrict__ seg_b, uint32_t *__restrict__ seg_e) {
    for (uint32_t d = blockIdx.x * blockDim.x + threadIdx.x; d < n; d += gridDim.x * blockDim.x) {
        const uint32_t v = orig ? orig[d] : d;
        const uint32_t len = uint32_t(off[v + 1] - off[v]);
        const uint32_t s = base + uint32_t(start[d]);
        info[d] = make_uint2(s, len);
        if (seg_b) {
            seg_b[d] = s;
            seg_e[d] = s + len;
        }
    }
}

// Device vertices' lists, ids mapped through rank (when given), and the
// padding: a warp takes 32 consecutive vertices and spreads their words over
// its lanes, four chains of reads (list entry, rank) in flight per lane; lists
// of more than kLongList entries are queued for k_fill_long.  20M arcs: 0.56
// ms with one warp per vertex, 0.28 ms this way.
__global__ void __launch_bounds__(256)
k_fill(uint32_t n, const uint32_t *__restrict__ orig, const uint32_t *__restrict__ rank,
       const uint64_t *__restrict__ off, const uint32_t *__restrict__ src, const uint2 *__restrict__ info,
       uint32_t *__restrict__ dst, uint32_t *__restrict__ queue, uint32_t *__restrict__ queued) {
    const int lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t d0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; d0 < n; d0 += warps * 32) {
        const uint32_t d = d0 + lane;
        const uint2 inf = d < n ? info[d] : make_uint2(0, 0);
        const unsigned long long a = d < n ? off[orig ? orig[d] : d] : 0ull;
        const bool longl = inf.y > kLongList;
        if (longl) queue[atomicAdd(queued, 1u)] = d;
        const uint32_t words = longl ? 0u : padded(inf.y);
        uint32_t incl = words;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(kFullMask, incl, 31);
        for (uint32_t w0 = 0; w0 < total; w0 += 128) {
            uint32_t x[4], to[4];
            #pragma unroll
            for (int h = 0; h < 4; ++h) {
                const uint32_t w = w0 + 32 * h + lane, owner = run_owner(incl, w);
                const uint32_t ow = __shfl_sync(kFullMask, words, int(owner)), oi = __shfl_sync(kFullMask, incl, int(owner));
                const uint32_t at = w - (oi - ow);  // place in its list
                to[h] = __shfl_sync(kFullMask, inf.x, int(owner)) + at;
                const uint32_t len = __shfl_sync(kFullMask, inf.y, int(owner));
                const unsigned long long oa = __shfl_sync(kFullMask, a, int(owner));
                x[h] = w < total && at < len ? src[oa + at] : kPad;
            }
            if (rank) {
                #pragma unroll
                for (int h = 0; h < 4; ++h)
                    if (x[h] != kPad) x[h] = rank[x[h]];
            }
            #pragma unroll
            for (int h = 0; h < 4; ++h)
                if (w0 + 32 * h + lane < total) dst[to[h]] = x[h];
        }
    }
}

// The queued lists, one block each.
__global__ void __launch_bounds__(512)
k_fill_long(const uint32_t *__restrict__ orig, const uint32_t *__restrict__ rank, const uint64_t *__restrict__ off,
            const uint32_t *__restrict__ src, const uint2 *__restrict__ info, uint32_t *__restrict__ dst,
            const uint32_t *__restrict__ queue, const uint32_t *__restrict__ queued) {
    const uint32_t nq = *queued;
    for (uint32_t i = blockIdx.x; i < nq; i += gridDim.x) {
        const uint32_t d = queue[i];
        const uint64_t a = off[orig ? orig[d] : d];
        const uint2 inf = info[d];
        #pragma unroll 2
        for (uint32_t j = threadIdx.x; j < padded(inf.y); j += blockDim.x) {
            uint32_t x = kPad;
            if (j < inf.y) {
                x = src[a + j];
                if (rank) x = rank[x];
            }
            dst[inf.x + j] = x;
        }
    }
}

// The padding after each sorted list.
__global__ void k_pad(uint32_t n, const uint2 *__restrict__ info, uint32_t *__restrict__ adj) {
    for (uint32_t d = blockIdx.x * blockDim.x + threadIdx.x; d < n; d += gridDim.x * blockDim.x) {
        const uint2 inf = info[d];
        for (uint32_t j = inf.y; j < padded(inf.y); ++j) adj[inf.x + j] = kPad;
    }
}

// flag |= 1 when some vertex lists itself.
__global__ void k_loops(uint32_t n, const uint2 *__restrict__ info, const uint32_t *__restrict__ adj,
                        uint32_t *__restrict__ flag) {
    for (uint32_t d = blockIdx.x * blockDim.x + threadIdx.x; d < n; d += gridDim.x * blockDim.x) {
        const uint2 inf = info[d];
        if (contains(adj + inf.x, inf.y, d)) atomicOr(flag, 1u);
    }
}

// bwd[d] = entries of d's list below d (a lower-bound search per vertex).
__global__ void k_bwd(uint32_t n, const uint2 *__restrict__ info, const uint32_t *__restrict__ adj,
                      uint32_t *__restrict__ bwd) {
    for (uint32_t d = blockIdx.x * blockDim.x + threadIdx.x; d < n; d += gridDim.x * blockDim.x) {
        const uint2 inf = info[d];
        bwd[d] = lbound(adj + inf.x, inf.y, d);
    }
}

// Dense core rows: one warp per core vertex d, its list entries u >= core0
// other than d itself set bit u - core0 of row d - core0 (rows are zeroed
// before).
__global__ void k_core_bits(uint32_t n, uint32_t core0, const uint2 *__restrict__ info,
                            const uint32_t *__restrict__ adj, uint32_t *__restrict__ bits) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t words = kCore / 32;
    for (uint32_t d = core0 + (blockIdx.x * blockDim.x + threadIdx.x) / 32; d < n;
         d += (gridDim.x * blockDim.x) / 32) {
        const uint2 inf = info[d];
        const uint32_t *l = adj + inf.x;
        for (uint32_t i = lbound(l, inf.y, core0) + lane; i < inf.y; i += 32) {
            const uint32_t u = l[i] - core0;
            if (u != d - core0) atomicOr(bits + size_t(d - core0) * words + (u >> 5), 1u << (u & 31));
        }
    }
}

// Puts key x into the table of a list of len entries at `base` (global or
// shared memory).  At most len of the 2 len or more slots are taken, so a free
// one exists.
__device__ __forceinline__ void tab_insert(uint32_t *base, uint32_t len, uint32_t x) {
    const uint32_t nb = (len + 3) >> 2;
    uint32_t b = tab_bucket(nb, x);
    for (uint32_t tries = 0; tries < nb; ++tries) {
        for (uint32_t i = 0; i < 8; ++i)
            if (atomicCAS(base + 8 * size_t(b) + i, kTabEmpty, x) == kTabEmpty) return;
        b = b + 1 == nb ? 0 : b + 1;
    }
}

// Membership tables of the lists of vertices [0, h0): consecutive vertices'
// lists, and so their tables, lie one after the other, so a warp builds the
// tables of up to kTabWords list words at a time in shared memory and writes
// them out whole -- 4 B read and 8 B written per entry, the atomics in shared
// memory (built by compare-and-swap in global memory they took 2.3 ms for 20M
// entries, 0.28 ms with the hub kernels below).  A longer list (ids not
// degree-ranked) is queued for k_tables_queue.
constexpr uint32_t kTabWords = 1024;
constexpr int kTabWarps = 4;

__global__ void __launch_bounds__(kTabWarps * 32)
k_tables(uint32_t h0, const uint2 *__restrict__ info, const uint32_t *__restrict__ adj, uint32_t *__restrict__ tab,
         uint32_t *__restrict__ queue, uint32_t *__restrict__ queued) {
    __shared__ uint4 sh[kTabWarps][kTabWords / 2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint4 *const t4 = sh[warp];
    uint32_t *const t = reinterpret_cast<uint32_t *>(t4);
    const uint32_t warps = gridDim.x * kTabWarps;
    for (uint32_t v0 = (blockIdx.x * kTabWarps + warp) * 32; v0 < h0; v0 += warps * 32) {
        const uint32_t v = v0 + lane;
        const uint2 inf = v < h0 ? info[v] : make_uint2(0, 0);
        uint32_t left = padded(inf.y);  // words of this lane's list not built yet
        while (true) {
            // the lanes whose lists fit together, from the first one left on
            uint32_t incl = left;
            #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
                if (lane >= o) incl += y;
            }
            const unsigned todo = __ballot_sync(kFullMask, left != 0);
            if (!todo) break;
            const int first = __ffs(todo) - 1;
            const uint32_t off0 = __shfl_sync(kFullMask, inf.x, first);
            const unsigned sel = __ballot_sync(kFullMask, left != 0 && incl <= kTabWords);
            if (!sel) {  // the first one alone is too long
                if (lane == first) {
                    queue[atomicAdd(queued, 1u)] = v;
                    left = 0;
                }
                continue;
            }
            const bool mine = (sel >> lane) & 1u;
            const uint32_t words = __shfl_sync(kFullMask, incl, 31 - __clz(sel));
            for (uint32_t i = lane; i < words / 2; i += 32) t4[i] = make_uint4(kTabEmpty, kTabEmpty, kTabEmpty, kTabEmpty);
            __syncwarp();
            // word w of the run belongs to the last selected list that starts
            // at or before it; the padding is skipped
            for (uint32_t w0 = 0; w0 < words; w0 += 128) {
                uint32_t x[4];  // four reads in flight per lane
                #pragma unroll
                for (int h = 0; h < 4; ++h) x[h] = w0 + 32 * h + lane < words ? __ldg(adj + off0 + w0 + 32 * h + lane) : kPad;
                #pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const uint32_t w = w0 + 32 * h + lane, owner = run_owner(incl, w);
                    const uint32_t off = __shfl_sync(kFullMask, inf.x, int(owner));
                    const uint32_t len = __shfl_sync(kFullMask, inf.y, int(owner));
                    if (x[h] != kPad) tab_insert(t + 2 * (off - off0), len, x[h]);
                }
            }
            __syncwarp();
            uint4 *const out = reinterpret_cast<uint4 *>(tab + 2 * size_t(off0));
            for (uint32_t i = lane; i < words / 2; i += 32) out[i] = t4[i];
            __syncwarp();
            if (mine) left = 0;
        }
    }
}

// The same for hubs, one block per list of [h0, h1) with its table of 8 B per
// entry in dynamic shared memory.
__global__ void __launch_bounds__(1024)
k_tables_hub(uint32_t h0, uint32_t h1, const uint2 *__restrict__ info, const uint32_t *__restrict__ adj,
             uint32_t *__restrict__ tab) {
    extern __shared__ __align__(16) uint32_t t[];
    uint4 *const t4 = reinterpret_cast<uint4 *>(t);
    for (uint32_t v = h0 + blockIdx.x; v < h1; v += gridDim.x) {
        const uint2 inf = info[v];
        const uint32_t quads = padded(inf.y) / 2;
        for (uint32_t i = threadIdx.x; i < quads; i += blockDim.x)
            t4[i] = make_uint4(kTabEmpty, kTabEmpty, kTabEmpty, kTabEmpty);
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < inf.y; i += blockDim.x) tab_insert(t, inf.y, __ldg(adj + inf.x + i));
        __syncthreads();
        uint4 *const out = reinterpret_cast<uint4 *>(tab + 2 * size_t(inf.x));
        for (uint32_t i = threadIdx.x; i < quads; i += blockDim.x) out[i] = t4[i];
        __syncthreads();
    }
}

// The queued lists, one block each, in place (20M arcs in the host's order,
// lists of up to 20,000: first count 4 ms over a later one with one warp per
// such list, 1.3 this way; lists of up to 300,000: 12 and 0.7).
__global__ void __launch_bounds__(1024)
k_tables_queue(const uint2 *__restrict__ info, const uint32_t *__restrict__ adj, uint32_t *__restrict__ tab,
               const uint32_t *__restrict__ queue, const uint32_t *__restrict__ queued) {
    const uint32_t nq = *queued;
    for (uint32_t i = blockIdx.x; i < nq; i += gridDim.x) {
        const uint2 inf = info[queue[i]];
        uint32_t *const base = tab + 2 * size_t(inf.x);
        for (uint32_t j = threadIdx.x; j < 2 * padded(inf.y); j += blockDim.x) base[j] = kTabEmpty;
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < inf.y; j += blockDim.x) tab_insert(base, inf.y, __ldg(adj + inf.x + j));
    }
}

// Hubs whose table does not fit shared memory: in global memory (cleared
// before), one warp per 512 entries of a list.
__global__ void __launch_bounds__(256)
k_tables_long(uint32_t h0, uint32_t n, uint32_t chunks, const uint2 *__restrict__ info,
              const uint32_t *__restrict__ adj, uint32_t *__restrict__ tab) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t(gridDim.x) * blockDim.x) >> 5, tasks = uint64_t(n - h0) * chunks;
    for (uint64_t t = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; t < tasks; t += warps) {
        const uint2 inf = info[h0 + uint32_t(t / chunks)];
        const uint32_t a = uint32_t(t % chunks) * 512;
        if (a >= inf.y) continue;
        const uint32_t b = min(a + 512, inf.y);
        for (uint32_t i = a + lane; i < b; i += 32) tab_insert(tab + 2 * size_t(inf.x), inf.y, __ldg(adj + inf.x + i));
    }
}

// Device buffers of one build, stream-ordered from the device's memory pool
// (reused across builds instead of mapped and unmapped each time), released
// on every exit.
struct Scratch {
    cudaStream_t s;
    std::vector<void *> p;
    explicit Scratch(cudaStream_t st) : s(st) {}
    ~Scratch() {
        for (void *x : p) cudaFreeAsync(x, s);
        cudaStreamSynchronize(s);
    }
    template <class T>
    cudaError_t get(T **out, size_t count) {
        *out = nullptr;
        if (!count) count = 1;
        cudaError_t e = cudaMallocAsync(reinterpret_cast<void **>(out), sizeof(T) * count, s);
        if (e == cudaSuccess) p.push_back(*out);
        return e;
    }
};

}  // namespace

#define LCK(x)                                                                                   \
    do {                                                                                         \
        cudaError_t e_ = (x);                                                                    \
        if (e_ != cudaSuccess)                                                                   \
            return set_error(CUTS_ERR_CUDA, std::string("graph layout: ") + cudaGetErrorString(e_)); \
    } while (0)

int device_layout(uint32_t n, const uint64_t *out_off, const uint32_t *out_adj, const uint64_t *in_off,
                  const uint32_t *in_adj, int sym_hint, bool validate, DeviceGraph &g) {
    if (!out_off || (n > 0 && !out_adj && out_off[n] > 0)) return set_error(CUTS_ERR_ARG, "null CSR array");
    if (in_adj && !in_off) return set_error(CUTS_ERR_ARG, "in_adj without in_off");
    if (in_off && !in_adj && n > 0 && in_off[n] > 0) return set_error(CUTS_ERR_ARG, "in_off without in_adj");
    if (out_off[0] != 0 || (in_off && in_off[0] != 0)) return set_error(CUTS_ERR_ARG, "CSR offsets must start at 0");
    const uint64_t m = out_off[n];
    if (in_off && in_off[n] != m) return set_error(CUTS_ERR_ARG, "in/out arc counts differ");
    cudaStream_t s = g.stream;
    const uint32_t grid = std::max<uint32_t>(1, std::min<uint32_t>((n + 255) / 256, 148u * 16));
    Scratch sc(s);
    uint64_t *d_ooff = nullptr, *d_ioff = nullptr;
    uint32_t *d_oadj = nullptr, *d_iadj = nullptr, *d_flag = nullptr;
    LCK(sc.get(&d_ooff, size_t(n) + 1));
    LCK(sc.get(&d_oadj, m));
    LCK(sc.get(&d_flag, 1));
    LCK(cudaMemcpyAsync(d_ooff, out_off, sizeof(uint64_t) * (size_t(n) + 1), cudaMemcpyHostToDevice, s));
    if (m) LCK(cudaMemcpyAsync(d_oadj, out_adj, sizeof(uint32_t) * m, cudaMemcpyHostToDevice, s));
    if (in_off) {
        LCK(sc.get(&d_ioff, size_t(n) + 1));
        LCK(sc.get(&d_iadj, m));
        LCK(cudaMemcpyAsync(d_ioff, in_off, sizeof(uint64_t) * (size_t(n) + 1), cudaMemcpyHostToDevice, s));
        if (m) LCK(cudaMemcpyAsync(d_iadj, in_adj, sizeof(uint32_t) * m, cudaMemcpyHostToDevice, s));
    }
    // host-side tables, while the copies and the first kernels run: the
    // largest degree, degree tails, padded words.  An offset pair that the
    // validation below will refuse counts as an empty list, and so does a list
    // of more than n entries (not strictly sorted below n): the tails have an
    // entry per degree.
    auto host_deg = [&](const uint64_t *off, uint32_t v) {
        return off[v + 1] >= off[v] && off[v + 1] <= m && off[v + 1] - off[v] <= n ? uint32_t(off[v + 1] - off[v]) : 0u;
    };
    const uint64_t *const ioff_host = in_off ? in_off : out_off;  // without in-lists: symmetric, or refused below
    uint32_t maxd = 0;
    uint64_t w0 = 0, w1 = 0;
    #pragma omp parallel for reduction(max : maxd) reduction(+ : w0, w1) schedule(static)
    for (int64_t v = 0; v < int64_t(n); ++v) {
        const uint32_t o = host_deg(out_off, uint32_t(v)), i = in_off ? host_deg(in_off, uint32_t(v)) : o;
        maxd = std::max(maxd, std::max(o, i));
        w0 += (uint64_t(o) + 3) & ~uint64_t(3);
        w1 += (uint64_t(i) + 3) & ~uint64_t(3);
    }
    const uint64_t words_of[2] = {w0, w1};
    DegreeStats st;
    st.n = n;
    st.out_ge.assign(size_t(maxd) + 2, 0);
    st.in_ge.assign(size_t(maxd) + 2, 0);
    // per-thread histograms while they are small (two of 8 B x (maxd + 2)
    // per thread: 1 MB at the bound); one pass otherwise
    #pragma omp parallel if (maxd < (1u << 16))
    {
        std::vector<uint64_t> lo(size_t(maxd) + 2, 0), li(size_t(maxd) + 2, 0);
        #pragma omp for schedule(static) nowait
        for (int64_t v = 0; v < int64_t(n); ++v) {
            lo[host_deg(out_off, uint32_t(v))]++;
            li[host_deg(ioff_host, uint32_t(v))]++;
        }
        #pragma omp critical
        for (size_t d = 0; d < lo.size(); ++d) {
            st.out_ge[d] += lo[d];
            st.in_ge[d] += li[d];
        }
    }
    for (int64_t d = int64_t(maxd); d >= 0; --d) {
        st.out_ge[d] += st.out_ge[d + 1];
        st.in_ge[d] += st.in_ge[d + 1];
    }
    uint32_t h_flag = 0;
    auto read_flag = [&]() -> int {
        LCK(cudaMemcpyAsync(&h_flag, d_flag, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        LCK(cudaStreamSynchronize(s));
        return CUTS_OK;
    };
    int rc = CUTS_OK;
    if (validate && n) {
        LCK(cudaMemsetAsync(d_flag, 0, sizeof(uint32_t), s));
        const uint32_t vgrid = std::max<uint32_t>(1, std::min<uint32_t>((n + 7) / 8, 148u * 16));
        k_validate<<<vgrid, 256, 0, s>>>(n, m, d_ooff, d_oadj, d_flag);
        if (in_off) k_validate<<<vgrid, 256, 0, s>>>(n, m, d_ioff, d_iadj, d_flag);
        LCK(cudaGetLastError());
        if ((rc = read_flag())) return rc;
        if (h_flag & 1) return set_error(CUTS_ERR_ARG, "CSR offsets not monotone");
        if (h_flag & 2) return set_error(CUTS_ERR_ARG, "CSR list not strictly sorted or out of range");
    }
    // symmetry: given, compared with the in-lists, or checked arc by arc
    bool symmetric = sym_hint == 1;
    unsigned long long *d_updown = nullptr, h_updown[2] = {0, 0};
    if (sym_hint < 0) {
        LCK(cudaMemsetAsync(d_flag, 0, sizeof(uint32_t), s));
        if (in_off) {
            k_differ<uint64_t><<<grid, 256, 0, s>>>(uint64_t(n) + 1, d_ooff, d_ioff, d_flag);
            const uint32_t g2 = uint32_t(std::max<uint64_t>(1, std::min<uint64_t>((m + 255) / 256, 148u * 16)));
            if (m) k_differ<uint32_t><<<g2, 256, 0, s>>>(m, d_oadj, d_iadj, d_flag);
        } else if (n) {
            LCK(sc.get(&d_updown, 2));
            LCK(cudaMemsetAsync(d_updown, 0, 2 * sizeof(unsigned long long), s));
            k_symmetric<<<std::max<uint32_t>(1, std::min<uint32_t>((n + 7) / 8, 148u * 16)), 256, 0, s>>>(
                n, d_ooff, d_oadj, d_flag, d_updown);
            LCK(cudaMemcpyAsync(h_updown, d_updown, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
        }
        LCK(cudaGetLastError());
        if ((rc = read_flag())) return rc;
        symmetric = h_flag == 0 && h_updown[0] == h_updown[1];
        if (!in_off && !symmetric)
            return set_error(CUTS_ERR_ARG, "in-lists omitted but the graph is not symmetric");
    }
    if (!symmetric && !in_off) return set_error(CUTS_ERR_ARG, "directed graph without in-lists");
    const uint64_t *ioff_used = symmetric ? nullptr : d_ioff;

    // degree ranks (CUTS_NO_RELABEL=1 keeps host ids); the per-list sort
    // indexes words with int, so a layout of 2^31 words or more keeps them too
    uint64_t pre_words = words_of[0] + (symmetric ? 0 : words_of[1]);
    const char *nr = std::getenv("CUTS_NO_RELABEL");
    const bool relabel = !(nr && nr[0] == '1') && n > 1 && pre_words < (uint64_t(1) << 31);
    uint32_t *d_orig = nullptr, *d_rank = nullptr;
    if (relabel) {
        unsigned long long *k0 = nullptr, *k1 = nullptr;
        LCK(sc.get(&k0, n));
        LCK(sc.get(&k1, n));
        LCK(cudaMallocAsync(reinterpret_cast<void **>(&g.d_orig), sizeof(uint32_t) * n, s));
        d_orig = g.d_orig;
        LCK(sc.get(&d_rank, n));
        k_keys<<<grid, 256, 0, s>>>(n, d_ooff, ioff_used, k0);
        LCK(cudaGetLastError());
        size_t tb = 0;
        LCK(cub::DeviceRadixSort::SortKeys(nullptr, tb, k0, k1, int(n), 0, 64, s));
        void *tmp = nullptr;
        LCK(sc.get(reinterpret_cast<char **>(&tmp), tb));
        LCK(cub::DeviceRadixSort::SortKeys(tmp, tb, k0, k1, int(n), 0, 64, s));
        k_ranks<<<grid, 256, 0, s>>>(n, k1, d_orig, d_rank);
        LCK(cudaGetLastError());
    }
    // padded offsets: out-lists, then in-lists of a directed graph
    unsigned long long *plen = nullptr, *pstart = nullptr;
    LCK(sc.get(&plen, size_t(n) + 1));
    LCK(sc.get(&pstart, size_t(n) + 1));
    size_t sb = 0;
    LCK(cub::DeviceScan::ExclusiveSum(nullptr, sb, plen, pstart, int(n) + 1, s));
    void *scan_tmp = nullptr;
    LCK(sc.get(reinterpret_cast<char **>(&scan_tmp), sb));
    uint64_t words[2] = {0, 0};
    const int dirs = symmetric ? 1 : 2;
    std::vector<unsigned long long *> starts(dirs);
    for (int dir = 0; dir < dirs; ++dir) {
        const uint64_t *off = dir ? d_ioff : d_ooff;
        k_plen<<<grid, 256, 0, s>>>(n, d_orig, off, plen);
        LCK(cudaGetLastError());
        unsigned long long *st = nullptr;
        LCK(sc.get(&st, size_t(n) + 1));
        LCK(cub::DeviceScan::ExclusiveSum(scan_tmp, sb, plen, st, int(n) + 1, s));
        unsigned long long tot = 0;
        LCK(cudaMemcpyAsync(&tot, st + n, sizeof(tot), cudaMemcpyDeviceToHost, s));
        LCK(cudaStreamSynchronize(s));
        words[dir] = tot;
        starts[dir] = st;
    }
    const uint64_t total = std::max<uint64_t>(words[0] + words[1], 4);
    if (total >= (uint64_t(1) << 32)) return set_error(CUTS_ERR_LIMIT, "padded adjacency exceeds 2^32 words");

    // device-resident arrays of the graph (owned by g from here on)
    // the graph's own arrays come from the device's default pool too (freed
    // with cudaFreeAsync by device_graph_free), so a rebuilt graph reuses them
    LCK(cudaMallocAsync(reinterpret_cast<void **>(&g.out_info), sizeof(uint2) * std::max<uint32_t>(n, 1), s));
    if (symmetric) g.in_info = g.out_info;
    else LCK(cudaMallocAsync(reinterpret_cast<void **>(&g.in_info), sizeof(uint2) * std::max<uint32_t>(n, 1), s));
    LCK(cudaMallocAsync(reinterpret_cast<void **>(&g.adj), sizeof(uint32_t) * total, s));
    LCK(cudaMemsetAsync(g.adj, 0xff, sizeof(uint32_t) * total, s));
    uint32_t *seg_b = nullptr, *seg_e = nullptr, *fill = g.adj;
    if (relabel) {
        LCK(sc.get(&seg_b, size_t(n) * dirs));
        LCK(sc.get(&seg_e, size_t(n) * dirs));
        LCK(sc.get(&fill, total));
    }
    uint32_t *d_queue = nullptr;
    LCK(sc.get(&d_queue, n));
    for (int dir = 0; dir < dirs; ++dir) {
        const uint64_t *off = dir ? d_ioff : d_ooff;
        const uint32_t *src = dir ? d_iadj : d_oadj;
        uint2 *info = dir ? g.in_info : g.out_info;
        const uint32_t base = dir ? uint32_t(words[0]) : 0u;
        k_info<<<grid, 256, 0, s>>>(n, d_orig, off, starts[dir], base, info,
                                    seg_b ? seg_b + size_t(dir) * n : nullptr,
                                    seg_e ? seg_e + size_t(dir) * n : nullptr);
        if (n) {
            LCK(cudaMemsetAsync(d_flag, 0, sizeof(uint32_t), s));  // here: lists queued
            k_fill<<<std::max<uint32_t>(1, std::min<uint32_t>((n + 255) / 256, 148u * 8)), 256, 0, s>>>(
                n, d_orig, d_rank, off, src, info, fill, d_queue, d_flag);
            if (maxd > kLongList) k_fill_long<<<148 * 4, 512, 0, s>>>(d_orig, d_rank, off, src, info, fill, d_queue, d_flag);
        }
        LCK(cudaGetLastError());
    }
    if (relabel && m) {
        // each list, now in device ids, sorted into the final array
        size_t tb = 0;
        const int segs = int(n) * dirs;
        LCK(cub::DeviceSegmentedSort::SortKeys(nullptr, tb, fill, g.adj, int(total), segs, seg_b, seg_e, s));
        void *tmp = nullptr;
        LCK(sc.get(reinterpret_cast<char **>(&tmp), tb));
        LCK(cub::DeviceSegmentedSort::SortKeys(tmp, tb, fill, g.adj, int(total), segs, seg_b, seg_e, s));
        for (int dir = 0; dir < dirs; ++dir)
            k_pad<<<grid, 256, 0, s>>>(n, dir ? g.in_info : g.out_info, g.adj);
        LCK(cudaGetLastError());
    }
    LCK(cudaMemsetAsync(d_flag, 0, sizeof(uint32_t), s));
    if (n) k_loops<<<grid, 256, 0, s>>>(n, g.out_info, g.adj, d_flag);
    LCK(cudaGetLastError());
    if ((rc = read_flag())) return rc;
    g.loops = h_flag != 0;
    // per-vertex counts of list entries below the vertex (windows that start
    // or end at a list's own vertex need no search)
    LCK(cudaMallocAsync(reinterpret_cast<void **>(&g.bwd_out), sizeof(uint32_t) * std::max<uint32_t>(n, 1) * (symmetric ? 1 : 2), s));
    g.bwd_in = symmetric ? g.bwd_out : g.bwd_out + n;
    if (n) {
        k_bwd<<<grid, 256, 0, s>>>(n, g.out_info, g.adj, g.bwd_out);
        if (!symmetric) k_bwd<<<grid, 256, 0, s>>>(n, g.in_info, g.adj, g.bwd_in);
    }
    LCK(cudaGetLastError());
    if (symmetric && n) {
        // the dense core: the kCore highest ids (the hubs under the degree
        // ranking), as an adjacency bitmap
        g.core0 = n > kCore ? n - kCore : 0;
        const size_t words = size_t(kCore) * (kCore / 32);
        LCK(cudaMallocAsync(reinterpret_cast<void **>(&g.core_bits), words * sizeof(uint32_t), s));
        LCK(cudaMemsetAsync(g.core_bits, 0, words * sizeof(uint32_t), s));
        k_core_bits<<<(kCore * 32 + 255) / 256, 256, 0, s>>>(n, g.core0, g.out_info, g.adj, g.core_bits);
        LCK(cudaGetLastError());
    }
    g.adj_words = total;
    g.symmetric = symmetric;
    g.n = n;
    g.arcs = m;

    g.max_deg = maxd;
    g.stats = std::move(st);
    g.ranked = relabel;
    return CUTS_OK;
}

// The id map on the host (dumps), fetched once.
int host_orig(DeviceGraph &g) {
    if (!g.ranked || !g.orig.empty()) return CUTS_OK;
    std::vector<uint32_t> orig(g.n);
    LCK(cudaMemcpyAsync(orig.data(), g.d_orig, sizeof(uint32_t) * g.n, cudaMemcpyDeviceToHost, g.stream));
    LCK(cudaStreamSynchronize(g.stream));
    g.orig.swap(orig);
    return CUTS_OK;
}

// Degrees by device id on the host (the batched engine's task table), fetched
// once.
int host_degrees(DeviceGraph &g) {
    if (!g.h_out_deg.empty() || !g.n) return CUTS_OK;
    std::vector<uint2> info(g.n);
    std::vector<uint32_t> deg[2];
    for (int dir = 0; dir < (g.symmetric ? 1 : 2); ++dir) {
        LCK(cudaMemcpyAsync(info.data(), dir ? g.in_info : g.out_info, sizeof(uint2) * g.n, cudaMemcpyDeviceToHost,
                            g.stream));
        LCK(cudaStreamSynchronize(g.stream));
        deg[dir].resize(g.n);
        #pragma omp parallel for schedule(static)
        for (int64_t d = 0; d < int64_t(g.n); ++d) deg[dir][size_t(d)] = info[size_t(d)].y;
    }
    g.h_in_deg = g.symmetric ? deg[0] : std::move(deg[1]);
    g.h_out_deg = std::move(deg[0]);
    return CUTS_OK;
}

// Builds the tables at `tab`, on g.stream.
static int build_tables(DeviceGraph &g, uint32_t *tab) {
    cudaStream_t s = g.stream;
    const int dirs = g.symmetric ? 1 : 2;
    // ids are degree ranks (unless relabelling is off: then every list goes
    // to the first kernel, which queues the long ones), so no list of the vertices below n - c has more
    // than L entries, c being at least the number of vertices of degree above
    // L; out- plus in-degree above L needs one of them above L / 2
    auto longer = [&](uint64_t L) {
        if (!g.ranked) return g.n;
        auto above = [&](const std::vector<uint64_t> &ge, uint64_t d) { return d + 1 < ge.size() ? uint64_t(ge[d + 1]) : 0; };
        const uint64_t c = g.symmetric ? above(g.stats.out_ge, L) : above(g.stats.out_ge, L / 2) + above(g.stats.in_ge, L / 2);
        return g.n - uint32_t(std::min<uint64_t>(c, g.n));
    };
    // classes of list lengths: 32 vertices per warp; one block per list with 8,
    // 32 and 192 KB of shared memory; in place.  The first ends at 128: with
    // 1,024, 32 neighbouring lists of 500 were a warp's 16 rounds and the build's
    // tail (20M arcs: build 0.71 ms, 0.28 this way; the first count on 30,000
    // vertices / 100,000 edges 315 us, 245 this way)
    constexpr uint32_t kShort = 128, kMid = 4096, kBig = 24576;
    const uint32_t h0 = longer(kShort), hm = longer(kTabWords), h1 = longer(kMid), h2 = longer(kBig);
    LCK(cudaFuncSetAttribute(k_tables_hub, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kBig * 8)));
    std::unique_ptr<Scratch> sc;  // (its end waits for the stream)
    uint32_t *queued = nullptr, *queue = nullptr;  // lists too long for k_tables
    if (!g.ranked && g.max_deg > kTabWords) {
        sc = std::make_unique<Scratch>(s);
        LCK(sc->get(&queued, size_t(g.n) + 1));
        queue = queued + 1;
    }
    for (int dir = 0; dir < dirs; ++dir) {
        const uint2 *info = dir ? g.in_info : g.out_info;
        if (queue) LCK(cudaMemsetAsync(queued, 0, sizeof(uint32_t), s));
        k_tables<<<std::max<uint32_t>(1, std::min<uint32_t>((h0 + 127) / 128, 148u * 7)), kTabWarps * 32, 0, s>>>(
            h0, info, g.adj, tab, queue, queued);
        if (queue) k_tables_queue<<<148 * 2, 1024, 0, s>>>(info, g.adj, tab, queue, queued);
        if (hm > h0) k_tables_hub<<<std::min<uint32_t>(hm - h0, 148u * 16), 128, kTabWords * 8, s>>>(h0, hm, info, g.adj, tab);
        if (h1 > hm) k_tables_hub<<<std::min<uint32_t>(h1 - hm, 148u * 6), 256, kMid * 8, s>>>(hm, h1, info, g.adj, tab);
        if (h2 > h1) k_tables_hub<<<std::min<uint32_t>(h2 - h1, 148u), 1024, kBig * 8, s>>>(h1, h2, info, g.adj, tab);
        if (h2 < g.n) {
            // their words are the last ones of this direction's lists
            std::vector<uint2> hubs(g.n - h2);
            LCK(cudaMemcpyAsync(hubs.data(), info + h2, sizeof(uint2) * hubs.size(), cudaMemcpyDeviceToHost, s));
            LCK(cudaStreamSynchronize(s));
            const uint2 first = hubs[0];
            uint64_t words = 0;
            for (const uint2 &h : hubs) words += (uint64_t(h.y) + 3) & ~uint64_t(3);
            LCK(cudaMemsetAsync(tab + 2 * size_t(first.x), 0xff, 8 * words, s));
            k_tables_long<<<148 * 8, 256, 0, s>>>(h2, g.n, (g.max_deg + 511) / 512, info, g.adj, tab);
        }
        LCK(cudaGetLastError());
    }
    return CUTS_OK;
}

int device_tables(DeviceGraph &g) {
    if (g.tab_tried) return CUTS_OK;
    g.tab_tried = true;
    if (!g.n || !g.arcs) return CUTS_OK;
    const size_t bytes = sizeof(uint32_t) * 2 * size_t(g.adj_words);
    if (bytes > g.tab_limit) return CUTS_OK;
    uint32_t *tab = nullptr;
    if (cudaMallocAsync(reinterpret_cast<void **>(&tab), bytes, g.stream) != cudaSuccess) {
        cudaGetLastError();
        return CUTS_OK;
    }
    // the graph has them once they are queued whole: a table built in part has
    // no end to a search's chain of full buckets
    struct Hold {
        DeviceGraph &g;
        uint32_t *tab;
        ~Hold() {
            if (tab) cudaFreeAsync(tab, g.stream);
        }
    } hold{g, tab};
    LCK(cudaEventRecord(g.ev0, g.stream));  // the device time of the count that builds them includes the build
    const int rc = build_tables(g, tab);
    if (rc) return rc;
    hold.tab = nullptr;
    g.tab = tab;
    return CUTS_OK;
}

}  // namespace cuts
