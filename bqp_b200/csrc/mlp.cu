// The gravity surrogate's tensor-core building blocks: the BF16 GEMM of
// tc_gemm.cuh behind a launcher (C = A B^T, FP32 out).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "launch.h"
#include "tc_gemm.cuh"

namespace bqp {

// Split z of gridDim.z takes k from kz z to kz (z + 1) and writes its own C.
__global__ void __launch_bounds__(tc::kThreads, 1)
    k_gemm_bf16(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ B, float* __restrict__ C,
                int N, int K, int kz, int* err) {
    const int m0 = blockIdx.x * tc::kBM, n0 = blockIdx.y * tc::kBN;
    const int k0 = blockIdx.z * kz, k1 = min(K, k0 + kz);
    float* Cz = C + (size_t)blockIdx.z * gridDim.x * tc::kBM * N;
    tc::gemm_tile(A, B, K, k0, k1, m0, n0, err, [&](int row, int col0, const float* v) {
        float4* dst = reinterpret_cast<float4*>(Cz + (size_t)row * N + col0);
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    });
}

// out = the sum of S matrices of n4 float4, pairs first
__global__ void k_sum_splits(int S, int64_t n4, const float4* __restrict__ part, float4* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n4) return;
    float4 a[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int s = 0; s < S; s += 4)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (s + q < S) {
                const float4 v = part[(size_t)(s + q) * n4 + i];
                a[q].x += v.x;
                a[q].y += v.y;
                a[q].z += v.z;
                a[q].w += v.w;
            }
    out[i] = make_float4((a[0].x + a[1].x) + (a[2].x + a[3].x), (a[0].y + a[1].y) + (a[2].y + a[3].y),
                         (a[0].z + a[1].z) + (a[2].z + a[3].z), (a[0].w + a[1].w) + (a[2].w + a[3].w));
}

// The reduction is split where the tiles alone leave most SMs idle: a weight
// gradient is 256 x 256 over a whole batch, two tiles of 128 stages for 8,192
// rows (643 us a product, one after the other; 16 us in 32 splits of four).
int gemm_splits(int64_t M, int64_t N, int64_t K) {
    const int64_t tiles = (M / tc::kBM) * (N / tc::kBN), stages = K / tc::kBK;
    int64_t s = stages / 4;
    if (s > kGemmSplitsMax) s = kGemmSplitsMax;
    if (s * tiles > device_sm_count()) s = device_sm_count() / tiles;
    return (int)(s < 1 ? 1 : s);
}

cudaError_t launch_gemm_bf16_split(int64_t M, int64_t N, int64_t K, const void* A, const void* B, float* C,
                                   float* part, int* err, cudaStream_t st) {
    const int S = gemm_splits(M, N, K);
    if (S == 1) return launch_gemm_bf16(M, N, K, A, B, C, err, st);
    cudaError_t e = cudaFuncSetAttribute(k_gemm_bf16, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::kSmemBytes);
    if (e != cudaSuccess) return e;
    const int stages = (int)(K / tc::kBK), per = (stages + S - 1) / S, used = (stages + per - 1) / per;
    const dim3 grid((unsigned)(M / tc::kBM), (unsigned)(N / tc::kBN), (unsigned)used);
    k_gemm_bf16<<<grid, tc::kThreads, tc::kSmemBytes, st>>>(reinterpret_cast<const __nv_bfloat16*>(A),
                                                             reinterpret_cast<const __nv_bfloat16*>(B), part, (int)N,
                                                             (int)K, per * tc::kBK, err);
    const int64_t n4 = M * N / 4;
    k_sum_splits<<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(used, n4, reinterpret_cast<const float4*>(part),
                                                               reinterpret_cast<float4*>(C));
    return cudaGetLastError();
}

cudaError_t launch_gemm_bf16(int64_t M, int64_t N, int64_t K, const void* A, const void* B, float* C, int* err,
                             cudaStream_t st) {
    if (M <= 0 || N <= 0 || K <= 0) return cudaSuccess;
    if (M % tc::kBM || N % tc::kBN || K % tc::kBK) return cudaErrorInvalidValue;
    if (((uintptr_t)A | (uintptr_t)B | (uintptr_t)C) & 15u) return cudaErrorInvalidValue;
    if (M / tc::kBM > 65535 * 1024ll || N / tc::kBN > 65535) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(k_gemm_bf16, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::kSmemBytes);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)(M / tc::kBM), (unsigned)(N / tc::kBN));
    k_gemm_bf16<<<grid, tc::kThreads, tc::kSmemBytes, st>>>(reinterpret_cast<const __nv_bfloat16*>(A),
                                                             reinterpret_cast<const __nv_bfloat16*>(B), C, (int)N,
                                                             (int)K, (int)K, err);
    return cudaGetLastError();
}

}  // namespace bqp
