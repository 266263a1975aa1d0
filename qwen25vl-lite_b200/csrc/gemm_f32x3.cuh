// The 32-bit product on tensor cores (gemm_f32x3.cu), as gemm_f32.cu calls it.
#pragma once

#include "common.cuh"

// Whole lines of 32 k; below 256 k the FMA kernels' shorter start counts for more (gemm_f32.cu).
static inline bool f32x3_takes(int K) { return K >= 256 && K % 32 == 0; }
// W aligned for TMA; A too where M <= F32X3_FEW, else `scratch` holds f32x3_scratch(M, N, K) bytes.
#define F32X3_FEW 16
size_t f32x3_scratch(int M, int N, int K);
extern thread_local int f32x3_launches;
int launch_f32x3_few(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                     bool early, int* err, cudaStream_t s);
int launch_f32x3_many(const float* A, const float* W, const float* bias, float* C, void* scratch, int M, int N, int K, int lda, int ldw, int ldc,
                      bool early, int* err, cudaStream_t s);
