// Kernels of the learned warm start's pair-wise MLP: FP32 arithmetic with
// BF16 weights for inference and training (FP32 master weights, Adam).
//
// Every dense layer is C = op(A) op(B) (+ bias) (ReLU) on row-major FP32 /
// BF16 matrices, tiled 64 x 64 x 16 with 256 threads and a 4 x 4 block of C
// per thread.  The weight gradient dW = dY^T X (a reduction over all rows) is
// the same kernel with op(A) transposed, cut into slices of rows whose partial
// products are added in slice order, so every sum runs in a fixed order (no
// atomics) and training is deterministic.
#include <cuda_bf16.h>

#include "kernels.cuh"
#include "mlp.h"

namespace v2g {

namespace {

constexpr int kT = 64, kK = 16;
constexpr int kLd = kT + 4;  // rows of a chunk stay 16-byte aligned

template <class TB>
__device__ __forceinline__ float to_f(TB v);
template <>
__device__ __forceinline__ float to_f<float>(float v) {
    return v;
}
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) {
    return __bfloat162float(v);
}

// C[M x N] = op(A)[M x K] op(B)[K x N] (+ bias[n]) (ReLU) (zero where
// gate[m, n] <= 0); op(A)(m, k) = transA ? A[k * lda + m] : A[m * lda + k], same
// for B.  Slice blockIdx.z of the K range (kper rows each) writes its partial
// product to C + blockIdx.z * cstride, and with colsum the sums over its k of
// op(A)(m, k) to colsum + blockIdx.z * cstride (the bias gradient beside the
// weight gradient, from the chunks already in shared memory).
//
// Bound: FP32 FMA where the grid fills the GPU, latency below.  A thread holds
// 4 x 4 neighbouring elements, so a K step is two 16-byte shared loads for 16
// FMAs (4-byte ones of rows 16 apart before), and the next chunk's global loads
// are under way meanwhile.  Loss and gradient of 4,096 rows through the C ABI on a
// B200: 2.68 -> 0.46 ms, most of it copies now; gradient error against 64 bits
// 7.9e-7 -> 9.3e-8 (shorter sums).
template <class TB>
__global__ void __launch_bounds__(256) mlp_gemm_kernel(int M, int N, int K, const float* __restrict__ A, int lda,
                                                       bool transA, const TB* __restrict__ B, int ldb, bool transB,
                                                       const float* __restrict__ bias, int relu,
                                                       const float* __restrict__ gate, float* __restrict__ C, int ldc,
                                                       int kper, int64_t cstride, float* __restrict__ colsum) {
    __shared__ __align__(16) float As[2][kK][kLd];
    __shared__ __align__(16) float Bs[2][kK][kLd];
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int m0 = blockIdx.y * kT, n0 = blockIdx.x * kT;
    const int kb = blockIdx.z * kper, ke = min(K, kb + kper);
    C += blockIdx.z * cstride;
    float ra[4], rb[4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = threadIdx.x + 256 * u;
            const int mm = transA ? i % kT : i / kK, kk = transA ? i / kT : i % kK;
            const int m = m0 + mm, k = k0 + kk;
            ra[u] = m < M && k < ke ? (transA ? A[(int64_t)k * lda + m] : A[(int64_t)m * lda + k]) : 0.f;
            const int nn = transB ? i / kK : i % kT, kq = k0 + (transB ? i % kK : i / kT);
            const int n = n0 + nn;
            rb[u] = n < N && kq < ke ? to_f<TB>(transB ? B[(int64_t)n * ldb + kq] : B[(int64_t)kq * ldb + n]) : 0.f;
        }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = threadIdx.x + 256 * u;
            As[buf][transA ? i / kT : i % kK][transA ? i % kT : i / kK] = ra[u];
            Bs[buf][transB ? i % kK : i / kT][transB ? i / kK : i % kT] = rb[u];
        }
    };
    float acc[4][4] = {};
    float cs = 0.f;
    fetch(kb);
    stash(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = kb; k0 < ke; k0 += kK) {
        const bool more = k0 + kK < ke;
        if (more) fetch(k0 + kK);
#pragma unroll
        for (int kk = 0; kk < kK; kk++) {
            const float4 a = *reinterpret_cast<const float4*>(&As[buf][kk][4 * ty]);
            const float4 b = *reinterpret_cast<const float4*>(&Bs[buf][kk][4 * tx]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        if (colsum && blockIdx.x == 0 && threadIdx.x < kT)
            for (int kk = 0; kk < kK; kk++) cs += As[buf][kk][threadIdx.x];
        if (more) {
            stash(buf ^ 1);
            __syncthreads();
            buf ^= 1;
        }
    }
    if (colsum && blockIdx.x == 0 && threadIdx.x < kT && m0 + (int)threadIdx.x < M)
        colsum[blockIdx.z * cstride + m0 + threadIdx.x] = cs;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = m0 + 4 * ty + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + 4 * tx + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[n];
            if (relu) v = fmaxf(v, 0.f);
            if (gate && !(gate[(int64_t)m * ldc + n] > 0.f)) v = 0.f;
            C[(int64_t)m * ldc + n] = v;
        }
    }
}

// g[i] = sum over slices of part[s * n + i], in slice order
__global__ void sum_slices_kernel(int64_t n, int slices, const float* __restrict__ part, float* __restrict__ g) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float s = 0.f;
#pragma unroll 8
        for (int k = 0; k < slices; k++) s += part[k * n + i];
        g[i] = s;
    }
}

// mean squared error: d = (out - t) * scale, per-block partial sums of d^2 / scale
__global__ void mse_kernel(int64_t n, const float* __restrict__ out, const float* __restrict__ t, float scale,
                           float* __restrict__ d, double* __restrict__ partial) {
    __shared__ double sh[256];
    double s = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float e = out[i] - t[i];
        d[i] = 2.f * e * scale;
        s += (double)e * e;
    }
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

// Adam (Kingma and Ba 2015) on the FP32 master weights, then the BF16 copy
__global__ void adam_kernel(int64_t n, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, __nv_bfloat16* __restrict__ w16, float lr, float b1, float b2,
                            float c1, float c2, float eps) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        w[i] = wi;
        w16[i] = __float2bfloat16_rn(wi);
    }
}

__global__ void to_bf16_kernel(int64_t n, const float* __restrict__ w, __nv_bfloat16* __restrict__ w16) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        w16[i] = __float2bfloat16_rn(w[i]);
}

inline int grid1(int64_t n) {
    int64_t g = (n + 255) / 256;
    return (int)(g < 1 ? 1 : (g > 148 * 8 ? 148 * 8 : g));
}

}  // namespace

void mlp_layer(int M, int N, int K, const float* A, const __nv_bfloat16* W, const float* bias, bool relu, float* C,
               cudaStream_t s) {
    dim3 grid((N + kT - 1) / kT, (M + kT - 1) / kT);
    mlp_gemm_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(M, N, K, A, K, false, W, K, true, bias, relu, nullptr, C, N, K,
                                                        0, nullptr);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void mlp_input_grad(int M, int N, int K, const float* dy, const __nv_bfloat16* W, const float* gate, float* dx,
                    cudaStream_t s) {
    dim3 grid((N + kT - 1) / kT, (M + kT - 1) / kT);
    mlp_gemm_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(M, N, K, dy, K, false, W, N, false, nullptr, 0, gate, dx, N, K,
                                                        0, nullptr);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

// One slice per 256 rows, up to 32: the weight gradients of the 224-wide layers
// are 16 tiles, and one CTA per tile over 4,096 rows took 721 us a product.
int mlp_slices(int rows) { return rows <= 256 ? 1 : (rows >= 32 * 256 ? 32 : (rows + 255) / 256); }

void mlp_weight_grad(int rows, int out, int in, const float* dy, const float* x, float* dw, float* db, int64_t stride,
                     cudaStream_t s) {
    const int slices = mlp_slices(rows), kper = (rows + slices - 1) / slices;
    dim3 grid((in + kT - 1) / kT, (out + kT - 1) / kT, slices);
    mlp_gemm_kernel<float><<<grid, 256, 0, s>>>(out, in, rows, dy, out, true, x, in, false, nullptr, 0, nullptr, dw, in,
                                                kper, stride, db);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void mlp_sum_slices(int64_t n, int slices, const float* part, float* g, cudaStream_t s) {
    sum_slices_kernel<<<grid1(n), 256, 0, s>>>(n, slices, part, g);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

int mlp_mse_blocks() { return 148; }

void mlp_mse(int64_t n, const float* out, const float* t, float scale, float* d, double* partial, cudaStream_t s) {
    mse_kernel<<<mlp_mse_blocks(), 256, 0, s>>>(n, out, t, scale, d, partial);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void mlp_adam(int64_t n, float* w, const float* g, float* m, float* v, __nv_bfloat16* w16, float lr, int step,
              cudaStream_t s) {
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    adam_kernel<<<grid1(n), 256, 0, s>>>(n, w, g, m, v, w16, lr, b1, b2, c1, c2, 1e-8f);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void mlp_to_bf16(int64_t n, const float* w, __nv_bfloat16* w16, cudaStream_t s) {
    to_bf16_kernel<<<grid1(n), 256, 0, s>>>(n, w, w16);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

}  // namespace v2g
