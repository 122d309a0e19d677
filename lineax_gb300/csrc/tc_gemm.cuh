// Host-side launcher of the tcgen05 TF32 GEMM (tc_gemm.cu) for other
// translation units: C = alpha * A Bᵀ + beta * C, A m×k, B n×k (K-major).
#pragma once

#include "common.cuh"

namespace lxgb {
// beside: the kernel before it on the stream lets its successor start at once and
// touches nothing of this product, which then runs beside it and ends no earlier:
// kBesidePanel on the SMs that a panel's cluster leaves, kBesideRow on all (a block
// row, whose CTAs are short and leave one by one).  Without the persistent kernel
// the product runs after the other.
constexpr int kBesidePanel = 1, kBesideRow = 2;
int gemm_tf32_nt(int M, int N, int K, const float* A, int64_t lda, const float* B, int64_t ldb,
                 float* C, int64_t ldc, float alpha, float beta, int* err, cudaStream_t st,
                 int beside = 0);
// 3xTF32 when Al and Bl (the lo parts) are given, plain TF32 otherwise.
int gemm_tf32_nt_split(int M, int N, int K, const float* A, const float* Al, int64_t lda,
                       const float* B, const float* Bl, int64_t ldb, float* C, int64_t ldc,
                       float alpha, float beta, int* err, cudaStream_t st, int beside = 0);
// C = alpha A Aᵀ + beta C on the tiles holding C's lower triangle (M×M),
// 3xTF32 when Al is given; the full product when tiles cannot be skipped.
int gemm_tf32_nt_split_lower(int M, int K, const float* A, const float* Al, int64_t lda, float* C,
                             int64_t ldc, float alpha, float beta, int* err, cudaStream_t st);
// One block row of the FP32 LU between its panel and the trailing update
// (ir.cu): the panel's interchanges on the other columns, U12 = L11^{-1} A12 in
// place, and the update's operands with 64 entries per row or column: U12ᵀ in
// b0 (FP32, precision 0; BF16, precision 2) or b0, b1 (hi, lo; precision 1),
// L21 likewise in a0, a1 (precision 1 and 2).
int lu32_block_row(int precision, int n, int j0, int nb, float* lu, const int32_t* piv, void* a0,
                   void* a1, void* b0, void* b1, cudaStream_t st);
// Split-K products C_s = A[:, K_s] B[:, K_s]ᵀ (K_s: splits ranges of chunk
// elements, chunk % 32 == 0), C_s at C + s * M * ldc, in one launch.
int gemm_tf32_nt_splitk(int M, int N, int K, const float* A, int64_t lda, const float* B,
                        int64_t ldb, float* C, int64_t ldc, int chunk, int splits, int* err,
                        cudaStream_t st);
// BF16 operands (kind::f16, FP32 accumulation); A and B hold __nv_bfloat16.
int gemm_bf16_nt(int M, int N, int K, const void* A, int64_t lda, const void* B, int64_t ldb,
                 float* C, int64_t ldc, float alpha, float beta, int* err, cudaStream_t st,
                 int beside = 0);
}
