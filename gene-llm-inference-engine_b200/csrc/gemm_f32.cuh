// The tiled 32-bit matrix product (gemm_f32.cu), reached through gi_gemm_simt.
#pragma once

#include "common.cuh"

namespace gi {

// Whether the operands have the form that gemm_f32 reads.
bool gemm_f32_takes(const float* A, const float* W, int M, int N, int K, int lda, int ldw);
// C[M,N] (+)= A[M,K] * W[N,K]^T, row strides in elements.
int gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int accumulate, int w_constant, cudaStream_t st);

}  // namespace gi
