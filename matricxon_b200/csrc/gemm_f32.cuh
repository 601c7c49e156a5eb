// The float products of the 32-bit path: the order in which every kernel forms a sum, and the entry of gemm_f32.cu.
#pragma once

#include <cuda_runtime.h>

constexpr int F32_PIECES = 4;         // chains of a sum over K: (p0 + p1) + (p2 + p3)
// Up to here the kernel that streams the weights, in groups of 16 rows: 32 rows of the four products of a 3B layer
// take it 0.38 ms, 33 rows take the tiles 0.59 ms.
constexpr int F32_FEW_ROWS = 32;

// Length of a piece of K: a quarter, in whole steps of the kernels' loops (the last pieces may be short or empty).
__host__ __device__ inline int f32_piece(int K) { return ((K + F32_PIECES - 1) / F32_PIECES + 31) / 32 * 32; }

// Whether gemm_f32.cu takes these operands (16-byte reads, and enough of K); it gives the same bits as the general kernel.
extern "C" int mx_gemm_f32_pays(int M, int N, int K);
bool mx_gemm_f32_takes(const float* A, int lda, const float* W, int ldw, int M, int N, int K);
int mx_gemm_f32(const float* A, int lda, const float* W, int ldw, const float* bias, const float* residual, float* out,
                int ldo, int M, int N, int K, int mode, cudaStream_t stream);
