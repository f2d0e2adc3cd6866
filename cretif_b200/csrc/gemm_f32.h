// The 32-bit product's fast bodies (gemm_f32.cu), for the launchers of gemm_simt.cu.
#pragma once

#include <cuda_runtime.h>

namespace cretif {

// Whether gemm_f32 takes these operands (alignment, the grid's limits).
bool gemm_f32_takes(const void* A, const void* W, int M, int N, int K, int lda, int ldw);

// C[M,N] (+)= A[M,K] · W[N,K]^T; returns a status like the launchers.
int gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
             int accumulate, cudaStream_t st);

}  // namespace cretif
