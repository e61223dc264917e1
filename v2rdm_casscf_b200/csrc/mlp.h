// Launchers of the learned warm start's MLP kernels (mlp.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace v2g {

// A layer: C[M x N] = A[M x K] W^T + bias (ReLU), W (N x K) in BF16; FP32
// arithmetic, deterministic, like everything here.
void mlp_layer(int M, int N, int K, const float* A, const __nv_bfloat16* W, const float* bias, bool relu, float* C,
               cudaStream_t s);
// dx[M x N] = dy[M x K] W (W: K x N), zero where gate <= 0 (the ReLU of the layer below)
void mlp_input_grad(int M, int N, int K, const float* dy, const __nv_bfloat16* W, const float* gate, float* dx,
                    cudaStream_t s);
// Slice k of mlp_slices(rows): its partial dW (out x in) = dy^T x at dw + k * stride,
// its partial db (column sums of dy) at db + k * stride
int mlp_slices(int rows);
void mlp_weight_grad(int rows, int out, int in, const float* dy, const float* x, float* dw, float* db, int64_t stride,
                     cudaStream_t s);
// g[i] = sum over slices of part[k * n + i]
void mlp_sum_slices(int64_t n, int slices, const float* part, float* g, cudaStream_t s);
// d = 2 (out - t) scale; partial[block] = sum (out - t)^2 (mlp_mse_blocks() blocks)
int mlp_mse_blocks();
void mlp_mse(int64_t n, const float* out, const float* t, float scale, float* d, double* partial, cudaStream_t s);
// one Adam step (step >= 1) on w with gradient g, moments m and v; w16 = bf16(w)
void mlp_adam(int64_t n, float* w, const float* g, float* m, float* v, __nv_bfloat16* w16, float lr, int step,
              cudaStream_t s);
void mlp_to_bf16(int64_t n, const float* w, __nv_bfloat16* w16, cudaStream_t s);

}  // namespace v2g
