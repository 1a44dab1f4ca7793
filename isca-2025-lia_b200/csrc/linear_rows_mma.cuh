// Projections of a few rows, or to a few columns, on mma.sync (linear_rows_mma.cu): as the GEMM's plan sees them, as plain projections with strides, and as gates.
#pragma once
#include "common.cuh"

bool gemm_rows_takes(int M, int N, int K);
// (W as lia_gemm_bf16 takes it: no work in flight on the stream writes it; the others are told so by `resident`)
int gemm_rows(const void* A, const void* W, void* C, int M, int N, int K, cudaStream_t stream);
// rows of bf16 numbers that are whole 16-byte vectors
bool linear_rows_takes(const void* A, long long lda, long long sA, const void* W, long long ldw, long long sW, int M, int K);
int linear_rows(const void* A, long long lda, long long sA, const void* W, long long ldw, long long sW, void* C, int c_f32, long long ldc, long long sC, int M, int N, int K,
                int batch, float scale, int resident, cudaStream_t stream);
// lia_linear_small
int linear_rows_gates(const void* A, long long lda, const void* W, const float* bias, float* out, int M, int N, int K, int mode, float cap, int resident,
                      cudaStream_t stream);
