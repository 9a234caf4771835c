// prefill_attention.cuh — attention of a prompt on the tensor cores; ggb_op_attn_prefill picks between it and the CUDA-core kernels
#pragma once

#include <stdint.h>

// 16 tokens and more that see enough keys, key sizes that are whole 128-byte rows, aligned buffers, a context whose scores would fit the tiles' shared memory
bool ggb_attn_prefill_fits(const float *q, const void *kcache, const void *vcache, int64_t T, int pos0, int H, int Hkv, int d, const float *out, const void *out_bf16);
int ggb_attn_prefill_tiles(const float *q, const void *kcache, const void *vcache, int64_t T, int pos0, int H, int Hkv, int d, float *out, void *out_bf16);
