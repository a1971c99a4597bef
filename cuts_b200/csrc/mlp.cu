// mlp.cu -- the learned matching-order cost model: a small MLP (FP32 at its interface, FP64 inside)
// (in -> H -> H -> 1, ReLU) trained and evaluated by hand-written kernels.
//
// It predicts log(1 + |L_i|), the size of trie level i, from per-step
// features of a candidate order; the order search (order_search.cpp) sums
// the predictions into a work estimate and keeps the cheapest order.
//
// Training is full-batch or mini-batch Adam on the mean squared error: two
// launches per step (k_mlp, k_mlp_adam).  Callers give and get FP32; the
// weights, the optimiser's state and all sums are kept in FP64, so a training
// run follows the exact one (a ReLU that flips on a rounding error changes the
// steps after it: with FP32 sums runs of 48 steps ended up to 8e-6 from it,
// with FP64 3e-8, for 1.73 ms instead of 1.38 for such a fit).  Sizes are tiny (in <= 32, H = 64), so a
// step is a few microseconds of CUDA-core work bound by shared-memory latency
// and launches; tensor cores would mean less precision.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "mlp.hpp"

namespace cuts {

#define MCK(call)                                                                      \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess)                                                         \
            return set_error(CUTS_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

namespace {

constexpr int kH = MLP_HIDDEN;
constexpr int kMaxIn = MLP_MAX_IN;
constexpr int kThreads = 256;
constexpr int kRows = 32;              // samples per tile
constexpr int kS = kH + 2;             // row stride of the 64-wide tiles in shared memory

// parameter layout: W1[H][in] b1[H] W2[H][H] b2[H] W3[H] b3
__host__ __device__ inline int n_params(int in) { return kH * in + kH + kH * kH + kH + kH + 1; }

struct Layout {
    int w1, b1, w2, b2, w3, b3, total;
};
__host__ __device__ inline Layout layout(int in) {
    Layout L;
    L.w1 = 0;
    L.b1 = L.w1 + kH * in;
    L.w2 = L.b1 + kH;
    L.b2 = L.w2 + kH * kH;
    L.w3 = L.b2 + kH;
    L.b3 = L.w3 + kH;
    L.total = L.b3 + 1;
    return L;
}

// Forward (and, with GRAD, backward) over samples [0, n) in tiles of kRows,
// grid-strided.  A block keeps the weights and one tile's activations in
// shared memory and computes 2 rows x 4 units per thread; the gradient is
// accumulated over the block's tiles in registers (a 4 x 4 tile of dW2, 4 x 2
// of dW1, one bias or W3 entry per thread) and written once per block to
// part[block][param], which k_mlp_adam / k_mlp_reduce sum in a fixed order in
// FP64.  lossp[block] = the block's sum of squared errors.  No atomics: the
// form with one shared-memory atomic per sample and weight took 260 us for
// 4,096 rows of 16 features (forward and backward), this one 18 us (both ncu,
// cold caches); a fit of 48 such steps and a prediction of 6,000 rows, copies
// included, 13.33 -> 1.39 ms in FP32 and 1.73 ms in FP64.  Rows of the tiles
// are padded to 66 values, so 16-byte reads of 8 consecutive rows (W2 by unit)
// hit 8 different bank groups.
template <bool GRAD>
__global__ void __launch_bounds__(kThreads, 1)
k_mlp(const double *__restrict__ params, int in, const float *__restrict__ X, const float *__restrict__ T, int n,
      float *__restrict__ Y, double *__restrict__ part, double *__restrict__ lossp) {
    extern __shared__ __align__(16) double sm[];
    const Layout L = layout(in);
    const int s1 = in | 1;                 // odd row stride of W1: units on different banks
    double *W2 = sm;                        // [H][kS]
    double *h1 = W2 + kH * kS;              // [kRows][kS]
    double *h2 = h1 + kRows * kS;           // [kRows][kS]: layer 2, then dL/d(layer 2)
    double *d1 = h2 + kRows * kS;           // [kRows][kS]: dL/d(layer 1)
    double *B1 = d1 + kRows * kS;           // [H]
    double *B2 = B1 + kH, *W3 = B2 + kH;
    double *dy = W3 + kH;                   // [kRows]
    double *x = dy + kRows;                 // [kRows][in]
    double *W1 = x + kRows * kMaxIn;        // [H][s1]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    for (int i = tid; i < kH * kH; i += kThreads) W2[(i / kH) * kS + i % kH] = params[L.w2 + i];
    for (int i = tid; i < kH * in; i += kThreads) W1[(i / in) * s1 + i % in] = params[L.w1 + i];
    if (tid < kH) {
        B1[tid] = params[L.b1 + tid];
        B2[tid] = params[L.b2 + tid];
        W3[tid] = params[L.w3 + tid];
    }
    const double b3 = params[L.b3];
    const double inv_n = 1.0 / double(max(n, 1));
    double g2[4][4] = {}, g1[4][2] = {}, gv = 0.0;
    double lsum = 0.0;
    for (int base = blockIdx.x * kRows; base < n; base += gridDim.x * kRows) {
        const int rows = min(kRows, n - base);
        __syncthreads();  // the weights are in; the previous tile is done with
        for (int i = tid; i < kRows * in; i += kThreads) x[i] = i < rows * in ? double(X[size_t(base) * in + i]) : 0.0;
        __syncthreads();
        double acc[2][4], z2[2][4];
        // layer 1: units tx + 16 q of rows ty, ty + 16
        #pragma unroll
        for (int q = 0; q < 4; ++q) acc[0][q] = acc[1][q] = B1[tx + 16 * q];
        for (int f = 0; f < in; ++f) {
            const double xa = x[ty * in + f], xb = x[(ty + 16) * in + f];
            #pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double w = W1[(tx + 16 * q) * s1 + f];
                acc[0][q] += w * xa;
                acc[1][q] += w * xb;
            }
        }
        #pragma unroll
        for (int r = 0; r < 2; ++r)
            #pragma unroll
            for (int q = 0; q < 4; ++q)
                h1[(ty + 16 * r) * kS + tx + 16 * q] = ty + 16 * r < rows ? fmax(acc[r][q], 0.0) : 0.0;
        __syncthreads();
        // layer 2
        #pragma unroll
        for (int q = 0; q < 4; ++q) acc[0][q] = acc[1][q] = B2[tx + 16 * q];
        #pragma unroll 4
        for (int i = 0; i < kH; i += 2) {
            const double2 a = *reinterpret_cast<const double2 *>(h1 + ty * kS + i);
            const double2 b = *reinterpret_cast<const double2 *>(h1 + (ty + 16) * kS + i);
            #pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double2 w = *reinterpret_cast<const double2 *>(W2 + (tx + 16 * q) * kS + i);
                acc[0][q] += w.x * a.x;
                acc[0][q] += w.y * a.y;
                acc[1][q] += w.x * b.x;
                acc[1][q] += w.y * b.y;
            }
        }
        // output: the 16 threads of a row reduce w3 . h2
        #pragma unroll
        for (int r = 0; r < 2; ++r) {
            double o = 0.0;
            #pragma unroll
            for (int q = 0; q < 4; ++q) {
                z2[r][q] = fmax(acc[r][q], 0.0);
                o += W3[tx + 16 * q] * z2[r][q];
            }
            #pragma unroll
            for (int d = 8; d; d >>= 1) o += __shfl_xor_sync(0xffffffffu, o, d);
            const int row = ty + 16 * r;
            const bool valid = row < rows;
            const double y = o + b3;
            double e = 0.0;
            if (valid && T) e = y - double(T[base + row]);
            const double de = 2.0 * e * inv_n;
            if (tx == 0) {
                if (valid && Y) Y[base + row] = float(y);
                if (valid) lsum += e * e;
                if (GRAD) dy[row] = de;
            }
            if (GRAD)
                #pragma unroll
                for (int q = 0; q < 4; ++q) h2[row * kS + tx + 16 * q] = valid ? z2[r][q] : 0.0;
        }
        if constexpr (GRAD) {
            __syncthreads();
            // dW3 and db3, before layer 2's values make room for its gradient
            if (tid >= 128 && tid < 192) {
                for (int r = 0; r < kRows; ++r) gv += dy[r] * h2[r * kS + tid - 128];
            } else if (tid == 192) {
                for (int r = 0; r < kRows; ++r) gv += dy[r];
            }
            __syncthreads();
            #pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int row = ty + 16 * r;
                const double de = dy[row];
                #pragma unroll
                for (int q = 0; q < 4; ++q)
                    h2[row * kS + tx + 16 * q] = row < rows && z2[r][q] > 0.0 ? de * W3[tx + 16 * q] : 0.0;
            }
            __syncthreads();
            // dL/d(layer 1): units 4 tx .. 4 tx + 3 of rows ty, ty + 16
            double e1[2][4] = {};
            #pragma unroll 4
            for (int j = 0; j < kH; ++j) {
                const double2 w0 = *reinterpret_cast<const double2 *>(W2 + j * kS + 4 * tx);
                const double2 w1 = *reinterpret_cast<const double2 *>(W2 + j * kS + 4 * tx + 2);
                const double a = h2[ty * kS + j], b = h2[(ty + 16) * kS + j];
                e1[0][0] += w0.x * a; e1[0][1] += w0.y * a; e1[0][2] += w1.x * a; e1[0][3] += w1.y * a;
                e1[1][0] += w0.x * b; e1[1][1] += w0.y * b; e1[1][2] += w1.x * b; e1[1][3] += w1.y * b;
            }
            #pragma unroll
            for (int r = 0; r < 2; ++r)
                #pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int at = (ty + 16 * r) * kS + 4 * tx + q;
                    d1[at] = h1[at] > 0.0 ? e1[r][q] : 0.0;
                }
            // dW2[4 ty + a][4 tx + b] over the tile's rows
            #pragma unroll 2
            for (int r = 0; r < kRows; ++r) {
                const double2 d0 = *reinterpret_cast<const double2 *>(h2 + r * kS + 4 * ty);
                const double2 dd1 = *reinterpret_cast<const double2 *>(h2 + r * kS + 4 * ty + 2);
                const double2 hh0 = *reinterpret_cast<const double2 *>(h1 + r * kS + 4 * tx);
                const double2 hh1 = *reinterpret_cast<const double2 *>(h1 + r * kS + 4 * tx + 2);
                const double dd[4] = {d0.x, d0.y, dd1.x, dd1.y}, hh[4] = {hh0.x, hh0.y, hh1.x, hh1.y};
                #pragma unroll
                for (int a = 0; a < 4; ++a)
                    #pragma unroll
                    for (int b = 0; b < 4; ++b) g2[a][b] += dd[a] * hh[b];
            }
            __syncthreads();
            // dW1[4 ty + a][tx + 16 c], and the two bias gradients
            for (int r = 0; r < kRows; ++r) {
                const double2 d0 = *reinterpret_cast<const double2 *>(d1 + r * kS + 4 * ty);
                const double2 dd1 = *reinterpret_cast<const double2 *>(d1 + r * kS + 4 * ty + 2);
                #pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int f = tx + 16 * c;
                    if (f < in) {
                        const double v = x[r * in + f];
                        g1[0][c] += d0.x * v; g1[1][c] += d0.y * v; g1[2][c] += dd1.x * v; g1[3][c] += dd1.y * v;
                    }
                }
            }
            if (tid < 128) {
                const double *src = tid < 64 ? d1 + tid : h2 + tid - 64;
                for (int r = 0; r < kRows; ++r) gv += src[r * kS];
            }
        }
    }
    if constexpr (GRAD) {
        double *out = part + size_t(blockIdx.x) * L.total;
        #pragma unroll
        for (int a = 0; a < 4; ++a) {
            #pragma unroll
            for (int b = 0; b < 4; ++b) out[L.w2 + (4 * ty + a) * kH + 4 * tx + b] = g2[a][b];
            #pragma unroll
            for (int c = 0; c < 2; ++c)
                if (tx + 16 * c < in) out[L.w1 + (4 * ty + a) * in + tx + 16 * c] = g1[a][c];
        }
        if (tid < 64) out[L.b1 + tid] = gv;
        else if (tid < 128) out[L.b2 + tid - 64] = gv;
        else if (tid < 192) out[L.w3 + tid - 128] = gv;
        else if (tid == 192) out[L.b3] = gv;
    }
    if (lossp) {
        // tx == 0 threads (lanes 0 and 16 of each warp) hold the sums
        __shared__ double lred[kThreads / 16];
        if (tx == 0) lred[ty] = lsum;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int i = 0; i < kThreads / 16; ++i) s += lred[i];
            lossp[blockIdx.x] = s;
        }
    }
}

// Sum of the blocks' partial gradients, 32 parameters x 8 groups of blocks
// per thread block, in FP64 and in a fixed order; the group-0 threads return
// it.  Each thread reads nparts / 8 values, independent loads in flight.
__device__ __forceinline__ double partial_sum(const double *__restrict__ part, int nparts, int total, int i) {
    __shared__ double red[8][33];
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
    double s = 0.0;
    if (i < total) {
        #pragma unroll 8
        for (int b = grp; b < nparts; b += 8) s += part[size_t(b) * total + i];
    }
    red[grp][lane] = s;
    __syncthreads();
    s = 0.0;
    if (grp == 0)
        for (int q = 0; q < 8; ++q) s += red[q][lane];
    return s;
}

__global__ void __launch_bounds__(256)
k_mlp_reduce(const double *__restrict__ part, int nparts, int total, float *__restrict__ g) {
    const int i = blockIdx.x * 32 + (threadIdx.x & 31);
    const double v = partial_sum(part, nparts, total, i);
    if (threadIdx.x < 32 && i < total) g[i] = float(v);
}

// Adam (Kingma & Ba 2015) with bias correction, on the summed partials.
__global__ void __launch_bounds__(256)
k_mlp_adam(double *__restrict__ p, const double *__restrict__ part, int nparts, double *__restrict__ m,
           double *__restrict__ v, int total, double lr, double b1, double b2, double eps, double c1, double c2) {
    const int i = blockIdx.x * 32 + (threadIdx.x & 31);
    const double gi = partial_sum(part, nparts, total, i);
    if (threadIdx.x < 32 && i < total) {
        const double mi = b1 * m[i] + (1.0 - b1) * gi;
        const double vi = b2 * v[i] + (1.0 - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrt(vi / c2) + eps);
    }
}

size_t smem_bytes(int in) {
    return sizeof(double) * (size_t(kH) * kS + 3 * size_t(kRows) * kS + 3 * kH + kRows + kRows * kMaxIn +
                            size_t(kH) * (in | 1));
}

}  // namespace

int mlp_param_count(int in) { return n_params(in); }

int Mlp::create(int in_dim, uint64_t seed, int dev) {
    if (in_dim < 1 || in_dim > kMaxIn) return set_error(CUTS_ERR_ARG, "mlp input dim out of range");
    in = in_dim;
    device = dev;
    MCK(cudaSetDevice(device));
    const int np = n_params(in);
    // blocks of the training kernel, at most: one per SM
    MCK(cudaDeviceGetAttribute(&max_blocks, cudaDevAttrMultiProcessorCount, device));
    // params, adam m, adam v, the loss partials, and the gradient as callers see it
    MCK(cudaMalloc(&d_params, sizeof(double) * (size_t(np) * 3 + max_blocks) + sizeof(float) * np));
    d_m = d_params + np;
    d_v = d_m + np;
    d_loss = d_v + np;
    d_grad = reinterpret_cast<float *>(d_loss + max_blocks);
    // He-uniform initialisation from a splitmix64 stream
    std::vector<float> h(np, 0.f);
    const Layout L = layout(in);
    uint64_t ctr = splitmix64(seed ^ 0x4d4c50ull);
    auto uni = [&](float lim) { return float((u01(splitmix64(ctr++)) * 2.0 - 1.0) * lim); };
    for (int i = 0; i < kH * in; ++i) h[L.w1 + i] = uni(std::sqrt(6.f / in));
    for (int i = 0; i < kH * kH; ++i) h[L.w2 + i] = uni(std::sqrt(6.f / kH));
    for (int i = 0; i < kH; ++i) h[L.w3 + i] = uni(std::sqrt(6.f / kH));
    const int rc = set_params(h.data());
    if (rc) return rc;
    MCK(cudaFuncSetAttribute(k_mlp<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_bytes(kMaxIn))));
    MCK(cudaFuncSetAttribute(k_mlp<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_bytes(kMaxIn))));
    step = 0;
    return CUTS_OK;
}

void Mlp::destroy() {
    if (d_params) {
        cudaSetDevice(device);
        cudaFree(d_params);
        release();
    }
    d_params = d_m = d_v = d_loss = nullptr;
    d_grad = nullptr;
}

// Below 2 MB from the runtime's allocator, which has such blocks at hand (first
// fit of 500 rows x 2 epochs 0.13 ms, from the pool 0.37).  Larger ones from
// the device's pool where it holds that much unused, as after a graph (4,096
// rows, one step: 0.10 ms, from the runtime 0.42 to 0.5; the form with
// shared-memory atomics, which had no partials, 0.38 to 0.42); a pool that has
// to grow is not asked, for its first growth in a process takes 6 ms.
int Mlp::Room::alloc(int device, size_t bytes) {
    pooled = false;
    cudaMemPool_t pool = nullptr;
    uint64_t held = 0, used = 0;
    if (bytes >= (size_t(2) << 20)) {
        MCK(cudaDeviceGetDefaultMemPool(&pool, device));
        MCK(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held));
        MCK(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used));
        pooled = held >= used + bytes;
    }
    if (pooled) MCK(cudaMallocAsync(&p, bytes, cudaStreamLegacy));
    else MCK(cudaMalloc(&p, bytes));
    return CUTS_OK;
}

void Mlp::Room::free() {
    if (!p) return;
    if (pooled) cudaFreeAsync(p, cudaStreamLegacy);
    else cudaFree(p);
    p = nullptr;
}

void Mlp::release() {
    part.free();
    samples.free();
    d_part = nullptr;
    d_X = nullptr;
    cap_rows = part_blocks = 0;
}

// Room for the partial gradients of `blocks` blocks and for `rows` staged
// samples, kept for later calls: one allocation where both have to grow, for a
// model's first fit is usually its only one.  Where one of the two outgrows its
// room the other stays: a fit of 672 rows, then a prediction of 937, gives the
// samples a small block of their own (0.05 ms; with the partials allocated anew
// 0.75).
int Mlp::reserve(int rows, int blocks) {
    const bool more_part = blocks > part_blocks, more_rows = rows > cap_rows;
    if (!more_part && !more_rows) return CUTS_OK;
    const bool inside = d_X && !samples.p;  // the samples lie behind the partials
    const size_t part_bytes = sizeof(double) * size_t(n_params(in)) * size_t(std::max(blocks, part_blocks));
    const size_t x_bytes = sizeof(float) * size_t(std::max(rows, cap_rows)) * (in + 2);
    int rc;
    if (!more_part || (!more_rows && !inside)) {
        Room &r = more_part ? part : samples;
        if (more_part) d_part = nullptr, part_blocks = 0;
        else d_X = nullptr, cap_rows = 0;
        r.free();
        if ((rc = r.alloc(device, more_part ? part_bytes : x_bytes))) return rc;
        if (more_part) d_part = static_cast<double *>(part.p), part_blocks = blocks;
        else d_X = static_cast<float *>(samples.p), cap_rows = rows;
        return CUTS_OK;
    }
    rows = std::max(rows, cap_rows);
    release();
    if ((rc = part.alloc(device, part_bytes + x_bytes))) return rc;
    d_part = static_cast<double *>(part.p);
    d_X = reinterpret_cast<float *>(static_cast<char *>(part.p) + part_bytes);
    cap_rows = rows;
    part_blocks = blocks;
    return CUTS_OK;
}

// Stages n samples, with room for `blocks` blocks' partial gradients.
int Mlp::upload(const float *X, const float *T, int n, int blocks) {
    const int rc = reserve(n, blocks);
    if (rc) return rc;
    MCK(cudaMemcpy(d_X, X, sizeof(float) * size_t(n) * in, cudaMemcpyHostToDevice));
    if (T) MCK(cudaMemcpy(d_X + size_t(cap_rows) * in, T, sizeof(float) * n, cudaMemcpyHostToDevice));
    return CUTS_OK;
}

int Mlp::grid_for(int n) const { return std::max(1, std::min((n + kRows - 1) / kRows, max_blocks)); }

// Mean of the blocks' sums of squared errors.
int Mlp::read_loss(int blocks, int n, float *loss) {
    std::vector<double> h(static_cast<size_t>(blocks));
    MCK(cudaMemcpy(h.data(), d_loss, sizeof(double) * size_t(blocks), cudaMemcpyDeviceToHost));
    double l = 0;
    for (double v : h) l += v;
    *loss = float(l / double(std::max(n, 1)));
    return CUTS_OK;
}

int Mlp::loss_grad(const float *X, const float *T, int n, float *loss, float *grad_out) {
    MCK(cudaSetDevice(device));
    const int np = n_params(in), blocks = grid_for(n);
    int rc = upload(X, T, n, blocks);
    if (rc) return rc;
    k_mlp<true><<<blocks, kThreads, smem_bytes(in)>>>(d_params, in, d_X, d_X + size_t(cap_rows) * in, n, nullptr,
                                                     d_part, d_loss);
    k_mlp_reduce<<<(np + 31) / 32, 256>>>(d_part, blocks, np, d_grad);
    MCK(cudaGetLastError());
    float l = 0;
    if ((rc = read_loss(blocks, n, &l))) return rc;
    if (loss) *loss = l;
    if (grad_out) MCK(cudaMemcpy(grad_out, d_grad, sizeof(float) * np, cudaMemcpyDeviceToHost));
    return CUTS_OK;
}

int Mlp::train(const float *X, const float *T, int n, int epochs, int batch, float lr,
               float *final_loss) {
    MCK(cudaSetDevice(device));
    if (batch <= 0 || batch > n) batch = n;
    int rc = upload(X, T, n, grid_for(batch));
    if (rc) return rc;
    const int np = n_params(in);
    const double b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;  // the FP32 values, as lr
    const float *dT = d_X + size_t(cap_rows) * in;
    for (int e = 0; e < epochs; ++e) {
        for (int s0 = 0; s0 < n; s0 += batch) {
            const int nb = std::min(batch, n - s0), blocks = grid_for(nb);
            k_mlp<true><<<blocks, kThreads, smem_bytes(in)>>>(d_params, in, d_X + size_t(s0) * in, dT + s0, nb, nullptr,
                                                             d_part, nullptr);
            ++step;
            const double c1 = 1.0 - std::pow(b1, double(step)), c2 = 1.0 - std::pow(b2, double(step));
            k_mlp_adam<<<(np + 31) / 32, 256>>>(d_params, d_part, blocks, d_m, d_v, np, lr, b1, b2, eps, c1, c2);
        }
    }
    MCK(cudaGetLastError());
    if (final_loss) {
        const int blocks = grid_for(n);
        k_mlp<false><<<blocks, kThreads, smem_bytes(in)>>>(d_params, in, d_X, dT, n, nullptr, nullptr, d_loss);
        MCK(cudaGetLastError());
        if ((rc = read_loss(blocks, n, final_loss))) return rc;
    }
    MCK(cudaDeviceSynchronize());
    return CUTS_OK;
}

int Mlp::predict(const float *X, int n, float *Y) {
    MCK(cudaSetDevice(device));
    int rc = upload(X, nullptr, n, 0);
    if (rc) return rc;
    float *dY = d_X + size_t(cap_rows) * in;  // reuse the target slot
    k_mlp<false><<<grid_for(n), kThreads, smem_bytes(in)>>>(d_params, in, d_X, nullptr, n, dY, nullptr, nullptr);
    MCK(cudaGetLastError());
    MCK(cudaMemcpy(Y, dY, sizeof(float) * n, cudaMemcpyDeviceToHost));
    return CUTS_OK;
}

int Mlp::get_params(float *out) {
    MCK(cudaSetDevice(device));
    std::vector<double> h(size_t(n_params(in)));
    MCK(cudaMemcpy(h.data(), d_params, sizeof(double) * h.size(), cudaMemcpyDeviceToHost));
    for (size_t i = 0; i < h.size(); ++i) out[i] = float(h[i]);
    return CUTS_OK;
}

int Mlp::set_params(const float *p) {
    MCK(cudaSetDevice(device));
    const size_t np = size_t(n_params(in));
    std::vector<double> h(p, p + np);
    h.resize(np * 3, 0.0);  // and the optimiser's state
    MCK(cudaMemcpy(d_params, h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice));
    step = 0;
    return CUTS_OK;
}

}  // namespace cuts
