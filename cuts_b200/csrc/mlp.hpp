// mlp.hpp -- MLP cost model for the learned matching order.
#pragma once
#include <cstddef>
#include <cstdint>

#include "host.hpp"

#define MLP_HIDDEN 64
#define MLP_MAX_IN 32

namespace cuts {

int mlp_param_count(int in);

// in -> 64 -> 64 -> 1 with ReLU, parameters resident on one GPU.
struct Mlp {
    int in = 0;
    int device = 0;
    // weights and Adam's moments in FP64 (FP32 at the interface)
    double *d_params = nullptr, *d_m = nullptr, *d_v = nullptr;
    float *d_grad = nullptr;
    double *d_part = nullptr;   // [part_blocks][params]: partial gradients of one step
    int part_blocks = 0;
    double *d_loss = nullptr;   // [max_blocks]: partial sums of squared errors
    int max_blocks = 1;
    float *d_X = nullptr;  // staged samples: X rows, then targets / outputs
    int cap_rows = 0;
    int64_t step = 0;

    int create(int in_dim, uint64_t seed, int dev);
    void destroy();
    // mean squared error and its gradient w.r.t. every parameter
    int loss_grad(const float *X, const float *T, int n, float *loss, float *grad);
    // Adam over mini-batches of `batch` rows (0 = full batch) for `epochs`
    int train(const float *X, const float *T, int n, int epochs, int batch, float lr,
              float *final_loss);
    int predict(const float *X, int n, float *Y);
    int get_params(float *out);
    int set_params(const float *p);

  private:
    // device memory from the runtime's allocator, or from the pool where large
    struct Room {
        void *p = nullptr;
        bool pooled = false;
        int alloc(int device, size_t bytes);
        void free();
    };
    Room part, samples;  // samples: unused while d_X lies behind the partials
    int upload(const float *X, const float *T, int n, int blocks);
    int grid_for(int n) const;
    int reserve(int rows, int blocks);
    void release();
    int read_loss(int blocks, int n, float *loss);
};

}  // namespace cuts
