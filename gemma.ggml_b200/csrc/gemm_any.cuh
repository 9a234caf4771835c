// gemm_any.cuh — products of fp32 matrices, and of bf16 matrices of any shape, on the tensor cores
#pragma once

#include <stdint.h>

// c (fp32, [T][ldc]) = a w^T, or (c_act) act(a w^T) in the matrices' type
int ggb_gemm_any(int dt, const void *w, int64_t N, int64_t K, const void *a, int64_t lda, int64_t T, float *c, int64_t ldc, void *c_act = nullptr, int act = 0);
