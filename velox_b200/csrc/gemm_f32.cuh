// The float32 product, for the entry points that take several element types (gemm_simt.cu).
#pragma once
#include <cuda_runtime.h>

int vx_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc, int batch,
                long long sa, long long sw, long long sc, int w_ready, cudaStream_t stream);
