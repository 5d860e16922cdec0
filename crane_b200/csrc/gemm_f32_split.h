// The 32-bit product on the tensor cores (gemm_f32_split.cu), for the dispatch of gemm_simt.cu.
#pragma once
#include <cuda_runtime.h>

// Rows of whole 16-byte pieces.
bool crane_f32_split_takes(const float* A, const float* W, int M, int N, int K, long long lda, long long ldw);
// part_stride > 0: C is the partial sums of crane_f32_slices(N, K) slices, part_stride elements apart; their sum in order has the
// same bits as the result that part_stride 0 writes.  err: the device-side error word, or null (a product whose waits ran out is NaN).
int crane_f32_split(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda,
                    long long ldw, long long ldc, long long part_stride, int* err, cudaStream_t st);
