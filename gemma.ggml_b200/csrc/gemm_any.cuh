// gemm_any.cuh — products of fp32 matrices, and of bf16 matrices of any shape, on the tensor cores
#pragma once

#include <stdint.h>

struct ggb_moe_groups;

// Up to here along K a product is for the kernels of multiply-adds (dense.cu): their few steps take no longer than bringing up a tensor-core tile
// (65 x 65: 8.4 against 10.5 us, fp32 128 x 128: 10.5 against 11.5), and a chain this short is as exact as sums that the tensor cores truncate
// (K = 65: 5e-8 against 7e-8).
constexpr int64_t kShortK = 128;

// c (fp32, [T][ldc]) = a w^T, or (c_act) act(a w^T) in the matrices' type
int ggb_gemm_any(int dt, const void *w, int64_t N, int64_t K, const void *a, int64_t lda, int64_t T, float *c, int64_t ldc, void *c_act = nullptr, int act = 0);

// the grouped form, bf16: w [n_exp][N][K], n slots in all, c rows in sorted-slot order; K a multiple of 64, lda of 8, w and a on 16 bytes
int ggb_gemm_any_grouped(const void *w, int64_t N, int64_t K, const void *a, int64_t lda, int64_t n, int n_exp, float *c, int64_t ldc, void *c_act, int act,
                         const ggb_moe_groups &grp);
