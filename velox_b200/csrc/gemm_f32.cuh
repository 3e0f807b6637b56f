// The float32 products, for the entry points that take several element types (gemm_simt.cu).
#pragma once
#include <cuda_runtime.h>

// Multiply-adds on the CUDA cores.
int vx_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc, int batch,
                long long sa, long long sw, long long sc, int w_ready, cudaStream_t stream);
// The tensor cores, every operand in three bfloat16 parts.  `error` (may be null): set if a wait for the tensor core runs out.
int vx_gemm_f32_tc(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc, int batch,
                   long long sa, long long sw, long long sc, int w_ready, int* error, cudaStream_t stream);
// Whether a product of these sizes takes the tensor cores.
extern "C" int vx_gemm_f32_takes_tc(int N, int K);
