// kquants.cu — the formats the reference's own offload kernels target.
//   Q4_K x Q8_K   ref: src/kernals.cl:48-111  (matrix_multiply_q4_K :166-214)
//   Q6_K x Q8_K   ref: src/kernals.cl:114-156 ([UPSTREAM] ggml's QK_K = 256 layout; the reference's copy indexes
//                 the block as QK_K = 64 and reads an uninitialised aux8 tail - its host never launches it,
//                 src/hpc.cpp:254-257 - so the pinned behaviour is ggml's scalar vec_dot)
//   F16 x F16     ref: src/kernals.cl:158-164 (double accumulator)
//   quantize_row_q8_K  [UPSTREAM] ggml INIT stage of mul_mat for K-quant weights (block at src/kernals.cl:29-34)
//
// The reference runs one work-item per output with a private aux8[256] and a serial loop.  Here a warp owns an
// output row and a super-block is spread over the warp: lane L holds the 8 consecutive aux8 elements 8L..8L+7, so
// element l of the lane IS the reference's lane-sum index (aux32[l], sums[l], l = e mod 8).  The integer part
// (aux32[l] = sum over the super-block of scale * q8 * a, sumi = sum bsums * mins) is exact in any order and is
// reduced with a folding butterfly (9 shuffles for the eight sums); the fp32 part keeps the reference's order: eight
// chains sums[l] += d * aux32[l] advanced super-block by super-block, sumf -= dmin * sumi, then sumf += sums[0..7].
// Results are bit-identical to the scalar code (tests compare bits with oracle/_ref, the reference's own source).
//
// That form takes weights and activations as they come, in ggml's AoS blocks (144 / 210 / 292 B).  Weights that stay on the device are
// re-laid out once and multiplied by integer tensor cores (below: packed form).
#include <algorithm>

#include "common.cuh"

namespace {

constexpr int kQK = 256;
constexpr int kQ4K = 144, kQ6K = 210, kQ8K = 292;
constexpr int kWarps = 8;

__device__ __forceinline__ uint32_t ld_u32(const uint8_t *p) { return *reinterpret_cast<const uint32_t *>(p); }
__device__ __forceinline__ uint32_t ld_u16(const uint8_t *p) { return *reinterpret_cast<const uint16_t *>(p); }
// 8 bytes from a 2-byte aligned address
__device__ __forceinline__ void ld8_a2(const uint8_t *p, uint32_t &lo, uint32_t &hi) {
    lo = ld_u16(p) | (ld_u16(p + 2) << 16);
    hi = ld_u16(p + 4) | (ld_u16(p + 6) << 16);
}
__device__ __forceinline__ int sx8(uint32_t w, int i) { return (int)(int8_t)(w >> (8 * i)); }

// v[0..7] per lane -> sum over the warp of v[l], returned in every lane of the group {4l .. 4l+3}
__device__ __forceinline__ int fold8(int (&v)[8], int lane) {
    int w4[4], w2[2];
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int send = b4 ? v[k] : v[4 + k];
        const int keep = b4 ? v[4 + k] : v[k];
        w4[k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int send = b3 ? w4[k] : w4[2 + k];
        const int keep = b3 ? w4[2 + k] : w4[k];
        w2[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    int w = (b2 ? w2[1] : w2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? w2[0] : w2[1], 4);
    w += __shfl_xor_sync(0xffffffffu, w, 2);
    w += __shfl_xor_sync(0xffffffffu, w, 1);
    return w; // l = 4*bit4 + 2*bit3 + bit2 = lane >> 2
}

__device__ __forceinline__ int warp_sum_i32(int v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// the eight chains live in lane groups; the final "for l: sumf += sums[l]" reads them in order
__device__ __forceinline__ float finish_lanes(float sumf, float sums) {
#pragma unroll
    for (int l = 0; l < 8; l++) sumf = __fadd_rn(sumf, __shfl_sync(0xffffffffu, sums, 4 * l));
    return sumf;
}

__device__ __forceinline__ float dot_q4_K(const uint8_t *x, const uint8_t *y, int nb, int lane) {
    float sums = 0.0f, sumf = 0.0f;
    const int c = lane >> 3, hi = lane & 4, j = lane >> 2;
#pragma unroll 1
    for (int i = 0; i < nb; i++, x += kQ4K, y += kQ8K) {
        const uint32_t dd = ld_u32(x);
        uint32_t u0 = ld_u32(x + 4), u1 = ld_u32(x + 8), u2 = ld_u32(x + 12);
        // 6-bit scales / mins (src/kernals.cl:75-80)
        const uint32_t u3 = ((u2 >> 4) & 0x0f0f0f0fu) | (((u1 >> 6) & 0x03030303u) << 4);
        const uint32_t uaux = u1 & 0x3f3f3f3fu;
        u1 = (u2 & 0x0f0f0f0fu) | (((u0 >> 6) & 0x03030303u) << 4);
        u2 = uaux;
        u0 &= 0x3f3f3f3fu;
        const int scale = (int)(((j < 4 ? u0 : u1) >> (8 * (j & 3))) & 0xff);
        const uint8_t *q4 = x + 16 + 32 * c + 8 * (lane & 3);
        uint32_t w0 = ld_u32(q4), w1 = ld_u32(q4 + 4);
        if (hi) { w0 >>= 4; w1 >>= 4; }
        w0 &= 0x0f0f0f0fu;
        w1 &= 0x0f0f0f0fu;
        const uint32_t a0 = ld_u32(y + 4 + 8 * lane), a1 = ld_u32(y + 8 + 8 * lane);
        int v[8];
#pragma unroll
        for (int l = 0; l < 4; l++) {
            v[l] = scale * (sx8(a0, l) * (int)((w0 >> (8 * l)) & 0xff));
            v[4 + l] = scale * (sx8(a1, l) * (int)((w1 >> (8 * l)) & 0xff));
        }
        const int aux = fold8(v, lane);
        // sumi = sum_j bsums[j] * mins[j / 2]
        int sm = 0;
        if (lane < 16) {
            const int bs = (int)(int16_t)ld_u16(y + 260 + 2 * lane);
            const int mj = lane >> 1;
            sm = bs * (int)(((mj < 4 ? u2 : u3) >> (8 * (mj & 3))) & 0xff);
        }
        const int sumi = warp_sum_i32(sm);
        const float yd = __uint_as_float(ld_u32(y));
        const float d = __fmul_rn(half_bits_to_float((uint16_t)(dd & 0xffff)), yd);
        const float dmin = __fmul_rn(half_bits_to_float((uint16_t)(dd >> 16)), yd);
        sums = __fadd_rn(sums, __fmul_rn(d, (float)aux));
        sumf = __fsub_rn(sumf, __fmul_rn(dmin, (float)sumi));
    }
    return finish_lanes(sumf, sums);
}

__device__ __forceinline__ float dot_q6_K(const uint8_t *x, const uint8_t *y, int nb, int lane) {
    float sums = 0.0f;
    const int c = lane >> 4, quarter = (lane >> 2) & 3, l0 = 8 * (lane & 3);
#pragma unroll 1
    for (int i = 0; i < nb; i++, x += kQ6K, y += kQ8K) {
        uint32_t q0, q1, h0, h1;
        ld8_a2(x + 64 * c + 32 * (quarter & 1) + l0, q0, q1);
        ld8_a2(x + 128 + 32 * c + l0, h0, h1);
        if (quarter & 2) { q0 >>= 4; q1 >>= 4; }
        q0 &= 0x0f0f0f0fu;
        q1 &= 0x0f0f0f0fu;
        h0 = ((h0 >> (2 * quarter)) & 0x03030303u) << 4;
        h1 = ((h1 >> (2 * quarter)) & 0x03030303u) << 4;
        q0 |= h0;
        q1 |= h1;
        const int scale = (int)(int8_t)x[192 + (lane >> 1)];
        const uint32_t a0 = ld_u32(y + 4 + 8 * lane), a1 = ld_u32(y + 8 + 8 * lane);
        int v[8];
#pragma unroll
        for (int l = 0; l < 4; l++) {
            v[l] = scale * (sx8(a0, l) * ((int)((q0 >> (8 * l)) & 0xff) - 32));
            v[4 + l] = scale * (sx8(a1, l) * ((int)((q1 >> (8 * l)) & 0xff) - 32));
        }
        const int aux = fold8(v, lane);
        const float d = __fmul_rn(half_bits_to_float((uint16_t)ld_u16(x + 208)), __uint_as_float(ld_u32(y)));
        sums = __fadd_rn(sums, __fmul_rn(d, (float)aux));
    }
    return finish_lanes(0.0f, sums);
}

// fp16 x fp16 products are exact in fp32 and in double; the double sum is insensitive to its order at the
// precision the final rounding to fp32 keeps (same argument as attention.cu)
__device__ __forceinline__ float dot_f16(const uint8_t *x, const uint8_t *y, int64_t n, int lane) {
    const __half2 *x2 = reinterpret_cast<const __half2 *>(x), *y2 = reinterpret_cast<const __half2 *>(y);
    const __half *xh = reinterpret_cast<const __half *>(x), *yh = reinterpret_cast<const __half *>(y);
    double acc = 0.0;
    if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 3) == 0) {
        for (int64_t i = lane; i < n / 2; i += 32) {
            const float2 a = __half22float2(x2[i]), b = __half22float2(y2[i]);
            acc = __fma_rn((double)a.x, (double)b.x, acc);
            acc = __fma_rn((double)a.y, (double)b.y, acc);
        }
        if ((n & 1) && lane == 0)
            acc = __fma_rn((double)__half2float(xh[n - 1]), (double)__half2float(yh[n - 1]), acc);
    } else { // odd row pitch: 2-byte loads
        for (int64_t i = lane; i < n; i += 32)
            acc = __fma_rn((double)__half2float(xh[i]), (double)__half2float(yh[i]), acc);
    }
    return __double2float_rn(warp_sum_f64(acc));
}

// grid (ceil(rows / 8), T)
template <int TYPE>
__global__ void __launch_bounds__(kWarps * 32)
raw_matvec_kernel(const uint8_t *__restrict__ w, int64_t rows, int64_t nb01, int64_t K, const uint8_t *__restrict__ act,
                  int64_t row_size, float *__restrict__ dst, int64_t dst_stride) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (row >= rows) return;
    const uint8_t *x = w + row * nb01;
    const uint8_t *y = act + (int64_t)blockIdx.y * row_size;
    float s;
    if (TYPE == GGB_TYPE_Q4_K) s = dot_q4_K(x, y, (int)(K / kQK), lane);
    else if (TYPE == GGB_TYPE_Q6_K) s = dot_q6_K(x, y, (int)(K / kQK), lane);
    else s = dot_f16(x, y, K, lane);
    if (lane == 0) dst[(int64_t)blockIdx.y * dst_stride + row] = s;
}

// [UPSTREAM] quantize_row_q8_K_reference for one 256-element block spread over a warp: lane L holds elements 8L..8L+7.
// Returns the lane's eight codes and the block's d (0 for an all-zero block); shared by the stand-alone quantiser and by
// the mat-vec kernels that quantise their fp32 activation row while they stage it.
__device__ __forceinline__ float q8k_quantize_lane(const float (&v)[8], int lane, int (&q)[8]) {
    // first element attaining max |x| (strict > in the scalar loop)
    float amax = 0.0f, mx = 0.0f;
    int idx = 0;
#pragma unroll
    for (int l = 0; l < 8; l++) {
        const float ax = fabsf(v[l]);
        if (ax > amax) { amax = ax; mx = v[l]; idx = 8 * lane + l; }
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        const float oa = __shfl_xor_sync(0xffffffffu, amax, off), om = __shfl_xor_sync(0xffffffffu, mx, off);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, off);
        if (oa > amax || (oa == amax && oi < idx)) { amax = oa; mx = om; idx = oi; }
    }
    if (!(amax > 0.0f)) { // "if (!amax)": all zero (a NaN block cannot reach amax > 0 either; ggml leaves it at 0)
#pragma unroll
        for (int l = 0; l < 8; l++) q[l] = 0;
        return 0.0f;
    }
    const float iscale = __fdiv_rn(-128.0f, mx);
#pragma unroll
    for (int l = 0; l < 8; l++) {
        const float val = __fadd_rn(__fmul_rn(iscale, v[l]), 12582912.0f); // nearest_int: round half to even
        q[l] = min(127, (__float_as_int(val) & 0x007fffff) - 0x00400000);
    }
    return __fdiv_rn(1.0f, iscale);
}

// one warp per 256-element block
__global__ void __launch_bounds__(kWarps * 32)
quantize_q8_K_kernel(const float *__restrict__ x, int64_t n_blocks, uint8_t *__restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t b = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (b >= n_blocks) return;
    const float4 f0 = *reinterpret_cast<const float4 *>(x + b * kQK + 8 * lane);
    const float4 f1 = *reinterpret_cast<const float4 *>(x + b * kQK + 8 * lane + 4);
    const float v[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
    int q[8];
    const float d = q8k_quantize_lane(v, lane, q);
    uint8_t *o = out + b * kQ8K;
    int s = 0;
#pragma unroll
    for (int l = 0; l < 8; l++) s += q[l];
    const uint32_t p0 = (q[0] & 0xff) | ((q[1] & 0xff) << 8) | ((q[2] & 0xff) << 16) | ((uint32_t)(q[3] & 0xff) << 24);
    const uint32_t p1 = (q[4] & 0xff) | ((q[5] & 0xff) << 8) | ((q[6] & 0xff) << 16) | ((uint32_t)(q[7] & 0xff) << 24);
    *reinterpret_cast<uint32_t *>(o + 4 + 8 * lane) = p0;
    *reinterpret_cast<uint32_t *>(o + 8 + 8 * lane) = p1;
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    if (!(lane & 1)) *reinterpret_cast<int16_t *>(o + 260 + lane) = (int16_t)s; // bsums[lane / 2]
    if (lane == 0) *reinterpret_cast<float *>(o) = d;
}


// ---------------------------------------------------------------- packed form (resident weights)
// The AoS kernel above spends 14 shuffles and ~60 instructions on a super-block.  Weights that stay on the device are
// re-laid out ONCE as fragments of integer tensor-core tiles: 16 rows x one sub-block are the A operand, and the B
// operand's column l holds the activations of lane-sum index l (zero elsewhere), so one mma.sync gives the integer part
// sum(code * a) of 16 rows x 8 lane sums; four multiply-adds a lane apply the sub-block's scales.  The integers are
// exact in any order.  The fp32 part keeps the scalar order: a warp leaves d * aux32[l] of its super-block in shared
// memory and 128 threads (row, l) add them to sums[l] super-block by super-block, then sumf += sums[0..7].
//
// A tile is 16 rows; a warp takes one super-block of it (an item), the warps of a CTA take consecutive super-blocks,
// and the next item's 2.3 (Q4_K) or 3.3 KB (Q6_K) are on their way while one is computed.  Layout of an item with R rows
// (R = 16; Q4_K's last tile has what is left, Q6_K pads it), lane (g, c) of the warp owning rows g and g + 8:
//   Q4_K: header[R][16 B] as in ggml | X[2][R][4 c][16 B], word i of plane p: sub-block 4p + i, byte b: low nibble =
//         element 4c + b, high nibble = element 16 + 4c + b                                     (144 B a row, as before)
//   Q6_K: L[2][R][4 c][16 B], word i of plane p: low nibbles = elements 4c + b of sub-block 8p + 2i, high nibbles =
//         those of 8p + 2i + 1 | H[R][4 c][16 B], word i: bits 2m of byte b = upper two bits (the top one inverted) of
//         element 4c + b of sub-block 4i + m | scales[R][16] | d[R]                              (210 B a row)
// A Q6_K byte (lo << 2 | hi << 6) with its top bit inverted is 4 * (q - 32) as int8; the 4 leaves by an exact shift.
//
// Bound by HBM and by the unpacking in turn (a tensor-core instruction's codes cost a warp about 15 others: instructions issue in 70 % of the
// cycles, 5.1 TB/s).  256000 x 2048: Q6_K 122 -> 75 us, Q4_K 91 -> 72 us in graph replays (a row a
// warp, a dot of four codes per instruction and lane sum).  Launched ahead like a step's kernels, which makes up for the codes' longer way where a
// matrix has few tiles: 256 x 2048 Q6_K 2.8 -> 2.55, Q4_K 2.35 -> 2.55 us (3.0 and 2.75 in plain launches).
constexpr int kActSB = 304;  // staged activation super-block, Q4_K: 256 B of codes | pair sums int[8] | d float | pad
constexpr int kActSB6 = 272; // Q6_K: 256 B of codes | d float | pad
constexpr int kTileRows = 16;

__host__ __device__ inline int64_t q6k_packed_bytes(int64_t rows, int nb) { return (rows + kTileRows - 1) / kTileRows * kTileRows * nb * kQ6K; }

// thread = (row, super-block, c)
__global__ void __launch_bounds__(256) q4k_repack_kernel(const uint8_t *__restrict__ raw, int64_t rows, int64_t nb01, int nb,
                                                        uint8_t *__restrict__ out) {
    const int64_t idx = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (idx >= rows * nb * 4) return;
    const int c = (int)(idx & 3);
    const int64_t rb = idx >> 2, row = rb / nb;
    const int sb = (int)(rb - row * nb), r = (int)(row % kTileRows);
    const int64_t row0 = row - r;
    const int R = (int)min((int64_t)kTileRows, rows - row0);
    const uint8_t *x = raw + row * nb01 + (int64_t)sb * kQ4K;
    uint8_t *o = out + (row0 * nb + (int64_t)sb * R) * kQ4K;
    *reinterpret_cast<uint32_t *>(o + 16 * r + 4 * c) = ld_u32(x + 4 * c); // d, dmin, scales
    for (int p = 0; p < 2; p++) {
        uint32_t w[4];
        for (int i = 0; i < 4; i++) { // sub-block j = 4p + i: nibble (j & 1) of the bytes of chunk j / 2
            const int j = 4 * p + i, sh = (j & 1) * 4;
            const uint8_t *q = x + 16 + 32 * (j >> 1) + 4 * c;
            w[i] = ((ld_u32(q) >> sh) & 0x0f0f0f0fu) | (((ld_u32(q + 16) >> sh) & 0x0f0f0f0fu) << 4);
        }
        *reinterpret_cast<uint4 *>(o + 16 * R + (p * R + r) * 64 + 16 * c) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

__global__ void __launch_bounds__(256) q6k_repack_kernel(const uint8_t *__restrict__ raw, int64_t rows, int64_t nb01, int nb,
                                                        uint8_t *__restrict__ out) {
    const int64_t idx = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (idx >= rows * nb * 4) return;
    const int c = (int)(idx & 3);
    const int64_t rb = idx >> 2, row = rb / nb;
    const int sb = (int)(rb - row * nb), r = (int)(row % kTileRows);
    const uint8_t *x = raw + row * nb01 + (int64_t)sb * kQ6K;
    uint8_t *o = out + ((row - r) * nb + (int64_t)sb * kTileRows) * kQ6K;
    // element e of the scalar code's aux8 (ggml QK_K = 256 layout): chunk e / 128, quarter = (e % 128) / 32, i = e % 32
    auto code = [&](int e) {
        const int ch = e >> 7, quarter = (e >> 5) & 3, i = e & 31;
        const uint8_t ql = x[64 * ch + 32 * (quarter & 1) + i], qh = x[128 + 32 * ch + i];
        return (uint32_t)((quarter & 2) ? (ql >> 4) : (ql & 0xF)) | (uint32_t)((qh >> (2 * quarter)) & 3) << 4;
    };
    uint32_t lo[8] = {}, hi[4] = {};
#pragma unroll
    for (int j = 0; j < 16; j++)
#pragma unroll
        for (int b = 0; b < 4; b++) {
            const uint32_t q = code(16 * j + 4 * c + b) ^ 0x20u;
            lo[j >> 1] |= (q & 0xFu) << (8 * b + 4 * (j & 1));
            hi[j >> 2] |= (q >> 4) << (8 * b + 2 * (j & 3));
        }
    for (int p = 0; p < 2; p++)
        *reinterpret_cast<uint4 *>(o + (p * kTileRows + r) * 64 + 16 * c) = make_uint4(lo[4 * p], lo[4 * p + 1], lo[4 * p + 2], lo[4 * p + 3]);
    *reinterpret_cast<uint4 *>(o + 128 * kTileRows + r * 64 + 16 * c) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    for (int b = 0; b < 4; b++) o[192 * kTileRows + 16 * r + 4 * c + b] = x[192 + 4 * c + b];
    if (c == 0) *reinterpret_cast<uint16_t *>(o + 208 * kTileRows + 2 * r) = *reinterpret_cast<const uint16_t *>(x + 208);
}

// byte i of w as a signed number
template <int I>
__device__ __forceinline__ int byte_s8(uint32_t w) {
    int v;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(v) : "r"(w), "n"(0x8880 + 0x1111 * I));
    return v;
}

__device__ __forceinline__ uint32_t comp(const uint4 &v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// one item of a lane: rows g (index 0) and g + 8 (index 1)
template <bool Q6>
struct kq_item {
    uint4 x[2][2];        // [row][plane]
    uint4 h[Q6 ? 2 : 1];  // Q6_K: upper bits
    uint4 hd[2];          // Q4_K: header, Q6_K: scales
    uint16_t d[2];        // Q6_K

    __device__ __forceinline__ void load(const uint8_t *w, int64_t rows, int nb, int64_t tile, int sb, int lane) {
        const int g = lane >> 2;
        const int64_t row0 = tile * kTileRows;
        const int R = Q6 ? kTileRows : (int)min((int64_t)kTileRows, rows - row0);
        const uint8_t *o = w + (row0 * nb + (int64_t)sb * R) * (Q6 ? kQ6K : kQ4K);
        const uint8_t *codes = Q6 ? o : o + 16 * R;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int r = Q6 ? g + 8 * u : min(g + 8 * u, R - 1); // a row past the end is read as the last one and not stored
#pragma unroll
            for (int p = 0; p < 2; p++) x[u][p] = ldg_stream_u4(codes + (p * R + r) * 64 + 16 * (lane & 3));
            if (Q6) {
                h[Q6 ? u : 0] = ldg_stream_u4(o + 128 * kTileRows + r * 64 + 16 * (lane & 3));
                hd[u] = __ldg(reinterpret_cast<const uint4 *>(o + 192 * kTileRows + 16 * r));
                d[u] = __ldg(reinterpret_cast<const uint16_t *>(o + 208 * kTileRows + 2 * r));
            } else {
                hd[u] = __ldg(reinterpret_cast<const uint4 *>(o + 16 * r));
            }
        }
    }
};

// aux32 of rows g and g + 8, lane sums 2c and 2c + 1, of a super-block whose activations start at ya: half a super-block at a time, the second half's
// registers moved down
__device__ __forceinline__ void kq_dot(const kq_item<true> &it, const uint8_t *ya, int c, uint32_t mask, int (&aux)[4]) {
    uint4 x[2] = {it.x[0][0], it.x[1][0]};
    uint2 h[2], sc[2];
#pragma unroll
    for (int u = 0; u < 2; u++) h[u] = make_uint2(it.h[u].x, it.h[u].y), sc[u] = make_uint2(it.hd[u].x, it.hd[u].y);
#pragma unroll
    for (int p = 0; p < 2; p++) {
#pragma unroll
        for (int jq = 0; jq < 2; jq++) {
            const uint4 act = *reinterpret_cast<const uint4 *>(ya + 128 * p + 64 * jq + 16 * c);
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const int j = 4 * jq + m; // of the half
                uint32_t a[2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const uint32_t lo = comp(x[u], j >> 1), hi = jq ? h[u].y : h[u].x;
                    a[u] = ((j & 1 ? lo >> 2 : lo << 2) & 0x3c3c3c3cu) | ((hi << (6 - 2 * m)) & 0xc0c0c0c0u);
                }
                int v[4];
                asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a[0]), "r"(a[1]), "r"(comp(act, m) & mask), "r"(0));
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const uint32_t w = jq ? sc[u].y : sc[u].x;
                    const int s = m == 0 ? byte_s8<0>(w) : m == 1 ? byte_s8<1>(w) : m == 2 ? byte_s8<2>(w) : byte_s8<3>(w);
                    aux[2 * u] += s * v[2 * u];
                    aux[2 * u + 1] += s * v[2 * u + 1];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 2; u++) x[u] = it.x[u][1], h[u] = make_uint2(it.h[u].z, it.h[u].w), sc[u] = make_uint2(it.hd[u].z, it.hd[u].w);
    }
}

__device__ __forceinline__ void kq_dot(const kq_item<false> &it, const uint8_t *ya, int c, uint32_t mask, int (&aux)[4]) {
    uint4 x[2] = {it.x[0][0], it.x[1][0]};
    uint32_t sc[2] = {it.hd[0].y & 0x3f3f3f3fu, it.hd[1].y & 0x3f3f3f3fu}; // 6-bit scales of sub-blocks 0..3 (src/kernals.cl:75-80)
#pragma unroll
    for (int p = 0; p < 2; p++) {
#pragma unroll
        for (int jp = 0; jp < 2; jp++) {
            const uint4 act = *reinterpret_cast<const uint4 *>(ya + 128 * p + 64 * jp + 16 * c);
#pragma unroll
            for (int m = 0; m < 2; m++) {
                const int j = 2 * jp + m; // of the half
                const uint32_t x0 = comp(x[0], j), x1 = comp(x[1], j);
                int v[4];
                asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                    : "r"(x0 & 0x0f0f0f0fu), "r"(x1 & 0x0f0f0f0fu), "r"((x0 >> 4) & 0x0f0f0f0fu), "r"((x1 >> 4) & 0x0f0f0f0fu),
                      "r"((m ? act.z : act.x) & mask), "r"((m ? act.w : act.y) & mask), "r"(0));
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int s = (int)((sc[u] >> (8 * j)) & 0xff);
                    aux[2 * u] += s * v[2 * u];
                    aux[2 * u + 1] += s * v[2 * u + 1];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 2; u++) { // sub-blocks 4..7
            x[u] = it.x[u][1];
            sc[u] = (it.hd[u].w & 0x0f0f0f0fu) | (((it.hd[u].y >> 6) & 0x03030303u) << 4);
        }
    }
}

// where word wi (elements 4 wi .. 4 wi + 3) of a super-block's activations is staged: a lane's words of four (Q6_K) or
// two (Q4_K) sub-blocks are adjacent
template <bool Q6>
__device__ __forceinline__ int act_word(int wi) {
    return Q6 ? (wi >> 4) * 64 + (wi & 3) * 16 + ((wi >> 2) & 3) * 4 : (wi >> 4) * 64 + (wi & 3) * 16 + ((wi >> 3) & 1) * 8 + ((wi >> 2) & 1) * 4;
}

// grid (x: groups of P tiles, strided; y: activation row); `chunk` super-blocks of a tile are computed at once, by a warp each:
// P > 1 only where chunk = nb.  Dynamic shared memory: nb staged super-blocks.
// F32ACT: `act` is the fp32 activation row (pitch row_size bytes); the CTA quantises it to Q8_K itself while staging
template <bool Q6, bool F32ACT>
__global__ void __launch_bounds__(kWarps * 32, 2)
kq_packed_kernel(const uint8_t *w, int64_t rows, int nb, const uint8_t *act, int64_t row_size, float *dst, int64_t dst_stride, int P, int chunk) {
    constexpr int SB = Q6 ? kActSB6 : kActSB, kD = Q6 ? 256 : 288;
    extern __shared__ __align__(16) uint8_t s_act[];
    __shared__ __align__(16) float s_t[2][kWarps][kTileRows * 8];
    __shared__ float s_m[Q6 ? 1 : 2][Q6 ? 1 : kWarps][kTileRows];
    step_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = blockDim.x >> 5;
    const int g = lane >> 2, c = lane & 3;
    const int64_t n_tiles = (rows + kTileRows - 1) / kTileRows, n_groups = (n_tiles + P - 1) / P;
    const int ip = warp / chunk, ik = warp - ip * chunk; // this warp's item of a round: tile ip of the group, super-block ik of the chunk
    kq_item<Q6> cur, nxt;
    int64_t grp = blockIdx.x;
    int sb0 = 0;
    auto valid = [&](int64_t gr, int s0) { return gr < n_groups && gr * P + ip < n_tiles && ip < P && s0 + ik < nb; };
    if (valid(grp, 0)) cur.load(w, rows, nb, grp * P + ip, ik, lane); // weights first: they take longest
    // ---- stage the activation row
    const uint8_t *y = act + (int64_t)blockIdx.y * row_size;
    if (F32ACT) {
        const float *xf = reinterpret_cast<const float *>(y);
        for (int sb = warp; sb < nb; sb += n_warps) { // a warp quantises one super-block at a time: lane = elements 8L..8L+7
            const float4 f0 = *reinterpret_cast<const float4 *>(xf + sb * kQK + 8 * lane);
            const float4 f1 = *reinterpret_cast<const float4 *>(xf + sb * kQK + 8 * lane + 4);
            const float v[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
            int q[8];
            const float d = q8k_quantize_lane(v, lane, q);
            uint8_t *base = s_act + sb * SB;
#pragma unroll
            for (int u = 0; u < 2; u++)
                *reinterpret_cast<uint32_t *>(base + act_word<Q6>(2 * lane + u)) =
                    (q[4 * u] & 0xff) | ((q[4 * u + 1] & 0xff) << 8) | ((q[4 * u + 2] & 0xff) << 16) | ((uint32_t)(q[4 * u + 3] & 0xff) << 24);
            if (!Q6) {
                int ssum = 0;
#pragma unroll
                for (int l = 0; l < 8; l++) ssum += q[l];
                ssum += __shfl_xor_sync(0xffffffffu, ssum, 1);
                ssum += __shfl_xor_sync(0xffffffffu, ssum, 2);
                if (c == 0) *reinterpret_cast<int *>(base + 256 + 4 * g) = ssum; // bsums[2j] + bsums[2j + 1]
            }
            if (lane == 0) *reinterpret_cast<float *>(base + kD) = d;
        }
    } else {
        for (int i = tid; i < nb * 64; i += blockDim.x)
            *reinterpret_cast<uint32_t *>(s_act + (i >> 6) * SB + act_word<Q6>(i & 63)) = ld_u32(y + (int64_t)(i >> 6) * kQ8K + 4 + 4 * (i & 63));
        for (int i = tid; i < nb * 9; i += blockDim.x) {
            const int sb = i / 9, k = i - sb * 9;
            const uint8_t *yb = y + (int64_t)sb * kQ8K;
            if (k == 8) *reinterpret_cast<uint32_t *>(s_act + sb * SB + kD) = ld_u32(yb);
            else if (!Q6) {
                const int16_t *bs = reinterpret_cast<const int16_t *>(yb + 260);
                *reinterpret_cast<int *>(s_act + sb * SB + 256 + 4 * k) = (int)bs[2 * k] + (int)bs[2 * k + 1];
            }
        }
    }
    __syncthreads();
    const uint32_t mask = (g >> 2) == (c & 1) ? 0xffu << (8 * (g & 3)) : 0u; // of the elements 4c .. 4c + 3, those = g mod 8
    float sums = 0.f, sumf = 0.f; // P == 1: thread (row, l)'s chains, carried from chunk to chunk
    int buf = 0;
    while (grp < n_groups) {
        int64_t grp_n = grp;
        int sb_n = sb0 + chunk;
        if (sb_n >= nb) { sb_n = 0; grp_n += gridDim.x; }
        if (valid(grp_n, sb_n)) nxt.load(w, rows, nb, grp_n * P + ip, sb_n + ik, lane);
        if (valid(grp, sb0)) {
            const uint8_t *ya = s_act + (sb0 + ik) * SB;
            int aux[4] = {0, 0, 0, 0};
            kq_dot(cur, ya, c, mask, aux);
            const float yd = *reinterpret_cast<const float *>(ya + kD);
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const float d = __fmul_rn(half_bits_to_float(Q6 ? cur.d[u] : (uint16_t)(cur.hd[u].x & 0xffff)), yd);
                const float t0 = __fmul_rn(d, (float)(Q6 ? aux[2 * u] >> 2 : aux[2 * u]));
                const float t1 = __fmul_rn(d, (float)(Q6 ? aux[2 * u + 1] >> 2 : aux[2 * u + 1]));
                *reinterpret_cast<float2 *>(&s_t[buf][warp][(g + 8 * u) * 8 + 2 * c]) = make_float2(t0, t1);
                if (!Q6) {
                    const uint32_t u2 = cur.hd[u].z & 0x3f3f3f3fu, u3 = ((cur.hd[u].w >> 4) & 0x0f0f0f0fu) | (((cur.hd[u].z >> 6) & 0x03030303u) << 4);
                    const uint32_t mn2 = ((c < 2 ? u2 : u3) >> (16 * (c & 1))) & 0xffffu; // mins of sub-blocks 2c, 2c + 1
                    const int *sp = reinterpret_cast<const int *>(ya + 256);
                    int sumi = (int)(mn2 & 0xff) * sp[2 * c] + (int)(mn2 >> 8) * sp[2 * c + 1];
                    sumi += __shfl_xor_sync(0xffffffffu, sumi, 1);
                    sumi += __shfl_xor_sync(0xffffffffu, sumi, 2);
                    const float dmin = __fmul_rn(half_bits_to_float((uint16_t)(cur.hd[u].x >> 16)), yd);
                    if (c == 0) s_m[Q6 ? 0 : buf][Q6 ? 0 : warp][g + 8 * u] = __fmul_rn(dmin, (float)sumi);
                }
            }
        }
        __syncthreads();
        // the scalar order: the super-blocks one after the other.  Two tables: the next round writes the other one.
        for (int ch = tid; ch < P * kTileRows * 8; ch += blockDim.x) {
            const int p = ch >> 7, r = (ch >> 3) & 15, l = ch & 7, n = min(chunk, nb - sb0);
            float tv[kWarps], mv[kWarps];
#pragma unroll
            for (int k = 0; k < kWarps; k++) { // past the end: x + 0 and x - 0 are x (no chain ever holds -0)
                const int i = min(p * chunk + k, kWarps - 1);
                tv[k] = k < n ? s_t[buf][i][r * 8 + l] : 0.f;
                mv[k] = !Q6 && k < n ? s_m[Q6 ? 0 : buf][Q6 ? 0 : i][r] : 0.f;
            }
#pragma unroll
            for (int k = 0; k < kWarps; k++) {
                sums = __fadd_rn(sums, tv[k]);
                if (!Q6) sumf = __fsub_rn(sumf, mv[k]);
            }
            if (sb0 + chunk >= nb) {
#pragma unroll
                for (int i = 0; i < 8; i++) sumf = __fadd_rn(sumf, __shfl_sync(0xffffffffu, sums, (lane & 24) + i));
                const int64_t row = (grp * P + p) * kTileRows + r;
                if (l == 0 && row < rows) dst[(int64_t)blockIdx.y * dst_stride + row] = sumf;
                sums = sumf = 0.f;
            }
        }
        buf ^= 1;
        grp = grp_n;
        sb0 = sb_n;
        cur = nxt;
    }
}

// ---------------------------------------------------------------- get_rows on K-quant blocks (embedding lookup)
// [UPSTREAM] dequantize_row_q4_K / dequantize_row_q6_K for the rows ids[t], times `scale` (ggml_scale): one thread per
// element, the scalar code's roundings: Q4_K y = (d * sc) * q - (dmin * m); Q6_K y = (d * scale) * (q - 32).
__global__ void __launch_bounds__(256)
get_rows_blocks_kernel(int type, const uint8_t *__restrict__ raw, int64_t n_rows, int64_t nb01, int64_t K,
                       const int32_t *__restrict__ ids, float scale, float *__restrict__ y) {
    const int64_t t = blockIdx.y;
    int64_t row = ids[t];
    row = row < 0 ? 0 : (row >= n_rows ? n_rows - 1 : row);
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= K) return;
    const int64_t sb = e >> 8;
    const int i = (int)(e & 255);
    float val;
    if (type == GGB_TYPE_Q4_K) {
        const uint8_t *x = raw + row * nb01 + sb * kQ4K;
        const int j = i >> 5; // sub-block
        uint32_t u0 = ld_u32(x + 4), u1 = ld_u32(x + 8), u2 = ld_u32(x + 12);
        const uint32_t u3 = ((u2 >> 4) & 0x0f0f0f0fu) | (((u1 >> 6) & 0x03030303u) << 4);
        const uint32_t uaux = u1 & 0x3f3f3f3fu;
        u1 = (u2 & 0x0f0f0f0fu) | (((u0 >> 6) & 0x03030303u) << 4);
        u2 = uaux;
        u0 &= 0x3f3f3f3fu;
        const int sc = (int)(((j < 4 ? u0 : u1) >> (8 * (j & 3))) & 0xff), mn = (int)(((j < 4 ? u2 : u3) >> (8 * (j & 3))) & 0xff);
        const uint32_t dd = ld_u32(x);
        const float d1 = __fmul_rn(half_bits_to_float((uint16_t)(dd & 0xffff)), (float)sc);
        const float m1 = __fmul_rn(half_bits_to_float((uint16_t)(dd >> 16)), (float)mn);
        const uint8_t q = x[16 + 32 * (j >> 1) + (i & 31)];
        const int nib = (j & 1) ? (q >> 4) : (q & 0xF);
        val = __fsub_rn(__fmul_rn(d1, (float)nib), m1);
    } else {
        const uint8_t *x = raw + row * nb01 + sb * kQ6K;
        const int c = i >> 7, quarter = (i >> 5) & 3, l = i & 31;
        const uint8_t ql = x[64 * c + 32 * (quarter & 1) + l], qh = x[128 + 32 * c + l];
        const int lo = (quarter & 2) ? (ql >> 4) : (ql & 0xF);
        const int a = (int)(int8_t)(lo | (((qh >> (2 * quarter)) & 3) << 4)) - 32;
        const float d = half_bits_to_float((uint16_t)ld_u16(x + 208));
        val = __fmul_rn(__fmul_rn(d, (float)(int8_t)x[192 + (i >> 4)]), (float)a);
    }
    y[t * K + e] = __fmul_rn(val, scale);
}

} // namespace

extern "C" {

size_t ggb_type_row_bytes(int type, int64_t cols) {
    switch (type) {
    case GGB_TYPE_F32: return (size_t)cols * 4;
    case GGB_TYPE_F16: return (size_t)cols * 2;
    case GGB_TYPE_Q4_0: return (size_t)(cols / 32) * 18;
    case GGB_TYPE_Q8_0: return (size_t)(cols / 32) * 34;
    case GGB_TYPE_Q4_K: return (size_t)(cols / kQK) * kQ4K;
    case GGB_TYPE_Q6_K: return (size_t)(cols / kQK) * kQ6K;
    case GGB_TYPE_Q8_K: return (size_t)(cols / kQK) * kQ8K;
    default: return 0;
    }
}

int ggb_op_quantize_q8_K(const float *x, int64_t cols, int64_t rows, void *out) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(x && out, "null pointer");
    GGB_CHECK_ARG(cols > 0 && cols % kQK == 0 && rows > 0, "quantize_q8_K: cols %lld not a multiple of 256", (long long)cols);
    const int64_t n_blocks = rows * (cols / kQK);
    quantize_q8_K_kernel<<<(unsigned)((n_blocks + kWarps - 1) / kWarps), kWarps * 32, 0, ggb_cuda_stream()>>>(
        x, n_blocks, (uint8_t *)out);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_op_q4k_repack(const void *raw, int64_t rows, int64_t nb01, int64_t K, void *packed) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(raw && packed && rows > 0 && K > 0 && K % kQK == 0 && nb01 >= K / kQK * kQ4K && nb01 % 4 == 0,
                  "q4k_repack: bad arguments");
    const int nb = (int)(K / kQK);
    const int64_t n = rows * nb * 4;
    q4k_repack_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ggb_cuda_stream()>>>((const uint8_t *)raw, rows, nb01, nb,
                                                                                 (uint8_t *)packed);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

static int launch_packed(int type, bool f32act, const void *packed, int64_t rows, int64_t K, const void *act, int64_t row_size,
                         int64_t T, float *dst, int64_t dst_stride) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(packed && act && dst && rows > 0 && T > 0 && K > 0 && K % kQK == 0, "mul_mat_packed: bad arguments");
    const int nb = (int)(K / kQK);
    const int64_t need = f32act ? K * 4 : (int64_t)nb * kQ8K;
    GGB_CHECK_ARG(row_size >= need && row_size % (f32act ? 16 : 4) == 0, "mul_mat_packed: activation row pitch %lld", (long long)row_size);
    const bool q4 = type == GGB_TYPE_Q4_K;
    const size_t smem = (size_t)nb * (q4 ? kActSB : kActSB6);
    GGB_CHECK_ARG(smem <= 200 * 1024, "mul_mat_packed: K %lld too long for the staged activation row", (long long)K);
    auto kern = q4 ? (f32act ? kq_packed_kernel<false, true> : kq_packed_kernel<false, false>)
                   : (f32act ? kq_packed_kernel<true, true> : kq_packed_kernel<true, false>);
    if (smem > 32 * 1024) GGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // The super-blocks of a tile in as few rounds of at most 8 warps as they need, evenly.  Several tiles a CTA where a row is short and tiles are
    // left for every SM all the same; 16 warps an SM (128 registers a thread).
    const int64_t tiles = (rows + kTileRows - 1) / kTileRows;
    const int rounds = (nb + kWarps - 1) / kWarps, chunk = (nb + rounds - 1) / rounds;
    const int P = rounds > 1 ? 1 : (int)std::max<int64_t>(1, std::min<int64_t>(kWarps / nb, tiles / ggb_sm_count())), warps = chunk * P;
    const unsigned gx = (unsigned)std::min<int64_t>((tiles + P - 1) / P, (int64_t)ggb_sm_count() * (2 * kWarps / warps));
    for (int64_t t0 = 0; t0 < T; t0 += 65535) {
        const dim3 grid(gx, (unsigned)(T - t0 < 65535 ? T - t0 : 65535));
#define KQ(Q6, F32ACT)                                                                                                                                \
    GGB_CUDA(ggb_launch_step(kq_packed_kernel<Q6, F32ACT>, grid, dim3((unsigned)(warps * 32)), smem, (const uint8_t *)packed, rows, nb, (const uint8_t *)act + t0 * row_size, \
                             row_size, dst + t0 * dst_stride, dst_stride, P, chunk));
        if (q4) {
            if (f32act) { KQ(false, true) } else { KQ(false, false) }
        } else {
            if (f32act) { KQ(true, true) } else { KQ(true, false) }
        }
#undef KQ
        GGB_LAUNCH_CHECK();
    }
    return GGB_OK;
}

int ggb_op_mul_mat_q4k_packed(const void *packed, int64_t rows, int64_t K, const void *act, int64_t row_size, int64_t T,
                              float *dst, int64_t dst_stride) {
    return launch_packed(GGB_TYPE_Q4_K, false, packed, rows, K, act, row_size, T, dst, dst_stride);
}

int ggb_op_mul_mat_q6k_packed(const void *packed, int64_t rows, int64_t K, const void *act, int64_t row_size, int64_t T,
                              float *dst, int64_t dst_stride) {
    return launch_packed(GGB_TYPE_Q6_K, false, packed, rows, K, act, row_size, T, dst, dst_stride);
}

int ggb_op_mul_mat_kq_packed_f32(int type, const void *packed, int64_t rows, int64_t K, const float *x, int64_t T, float *dst,
                                 int64_t dst_stride) {
    GGB_CHECK_ARG(type == GGB_TYPE_Q4_K || type == GGB_TYPE_Q6_K, "mul_mat_kq_packed_f32: type %d", type);
    return launch_packed(type, true, packed, rows, K, x, K * 4, T, dst, dst_stride);
}

size_t ggb_q6k_packed_bytes(int64_t rows, int64_t K) { return (size_t)q6k_packed_bytes(rows, (int)(K / kQK)); }

int ggb_op_q6k_repack(const void *raw, int64_t rows, int64_t nb01, int64_t K, void *packed) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(raw && packed && rows > 0 && K > 0 && K % kQK == 0 && nb01 >= K / kQK * kQ6K && nb01 % 2 == 0,
                  "q6k_repack: bad arguments");
    const int nb = (int)(K / kQK);
    const int64_t n = rows * nb * 4;
    q6k_repack_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ggb_cuda_stream()>>>((const uint8_t *)raw, rows, nb01, nb,
                                                                                 (uint8_t *)packed);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_op_get_rows_blocks(int type, const void *raw, int64_t n_rows, int64_t nb01, int64_t K, const int32_t *ids, int64_t T,
                           float scale, float *y) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(raw && ids && y && T > 0 && T <= 65535 && n_rows > 0, "get_rows_blocks: bad arguments");
    GGB_CHECK_ARG((type == GGB_TYPE_Q4_K || type == GGB_TYPE_Q6_K) && K > 0 && K % kQK == 0, "get_rows_blocks: type %d / K %lld", type, (long long)K);
    GGB_CHECK_ARG(nb01 >= (int64_t)ggb_type_row_bytes(type, K) && nb01 % (type == GGB_TYPE_Q4_K ? 4 : 2) == 0, "get_rows_blocks: row pitch %lld", (long long)nb01);
    const dim3 grid((unsigned)((K + 255) / 256), (unsigned)T);
    get_rows_blocks_kernel<<<grid, 256, 0, ggb_cuda_stream()>>>(type, (const uint8_t *)raw, n_rows, nb01, K, ids, scale, y);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_op_mul_mat_blocks(int type, const void *w, int64_t rows, int64_t nb01, int64_t K, const void *act,
                          int64_t row_size, int64_t T, float *dst, int64_t dst_stride) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(w && act && dst, "null pointer");
    GGB_CHECK_ARG(rows > 0 && T > 0 && K > 0, "mul_mat_blocks: bad extents");
    const bool kq = type == GGB_TYPE_Q4_K || type == GGB_TYPE_Q6_K;
    if (!kq && type != GGB_TYPE_F16) {
        ggb_set_error("mul_mat_blocks: no kernel for type %d", type);
        return GGB_ERR_UNSUPPORTED;
    }
    GGB_CHECK_ARG(!kq || K % kQK == 0, "mul_mat_blocks: K %lld not a multiple of 256", (long long)K);
    GGB_CHECK_ARG(nb01 >= (int64_t)ggb_type_row_bytes(type, K) && nb01 % (type == GGB_TYPE_Q4_K ? 4 : 2) == 0,
                  "mul_mat_blocks: src0 row pitch %lld", (long long)nb01);
    const int64_t act_row = (int64_t)ggb_type_row_bytes(kq ? GGB_TYPE_Q8_K : GGB_TYPE_F16, K);
    GGB_CHECK_ARG(row_size >= act_row && row_size % (kq ? 4 : 2) == 0, "mul_mat_blocks: activation row pitch %lld",
                  (long long)row_size);
    const uint8_t *wb = (const uint8_t *)w, *ab = (const uint8_t *)act;
    cudaStream_t st = ggb_cuda_stream();
    for (int64_t t0 = 0; t0 < T; t0 += 65535) { // grid.y carries the activation row
        const dim3 grid((unsigned)((rows + kWarps - 1) / kWarps), (unsigned)(T - t0 < 65535 ? T - t0 : 65535));
        const uint8_t *a0 = ab + t0 * row_size;
        float *d0 = dst + t0 * dst_stride;
        if (type == GGB_TYPE_Q4_K)
            raw_matvec_kernel<GGB_TYPE_Q4_K><<<grid, kWarps * 32, 0, st>>>(wb, rows, nb01, K, a0, row_size, d0, dst_stride);
        else if (type == GGB_TYPE_Q6_K)
            raw_matvec_kernel<GGB_TYPE_Q6_K><<<grid, kWarps * 32, 0, st>>>(wb, rows, nb01, K, a0, row_size, d0, dst_stride);
        else
            raw_matvec_kernel<GGB_TYPE_F16><<<grid, kWarps * 32, 0, st>>>(wb, rows, nb01, K, a0, row_size, d0, dst_stride);
        GGB_LAUNCH_CHECK();
    }
    return GGB_OK;
}

} // extern "C"
