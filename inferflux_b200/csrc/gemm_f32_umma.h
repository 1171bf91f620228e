// The float32 product on the tensor cores, for the library's own callers (gemm_f32.cu).
#pragma once
#include <cuda_runtime.h>

// Whether a product's shape goes to the tensor cores (from N, K and W's alignment alone, never from M, so that a row is
// summed the same way in every batch).
bool gemm_f32_umma_takes(const float* W, int N, int K);

// As ifx_gemm_f32, for shapes that gemm_f32_umma_takes.  scratch: gemm_f32_umma_scratch(M, K) bytes, 16-byte aligned (none
// up to 64 rows).
long long gemm_f32_umma_scratch(int M, int K);
int gemm_f32_umma(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda, long long ldc,
                  void* scratch, int w_fixed, int* error_flag, cudaStream_t stream);
