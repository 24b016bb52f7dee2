// The float32 products over rows that start on 16 bytes (gemm_f32.cu).
#pragma once
#include "common.cuh"

// Whether the kernels take these operands: K and the rows' distance multiples of four values, both matrices on 16 bytes.  (The number of rows
// has no say: the general kernel sums in another order, and a row alone has the result that it has among others.)
bool gemm_f32_takes(const float* A, int64_t lda, const float* W, int K);
// C[M,N] = A[M,K] W^T, epi as in gemm_simt.cu; 0 on success.
int gemm_f32(const float* A, int64_t lda, const float* W, float* C, int64_t ldc, int M, int N, int K, int epi, cudaStream_t stream);
