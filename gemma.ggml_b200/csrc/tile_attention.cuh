// tile_attention.cuh — attention of a portion of tokens over a paged bf16 cache on the tensor cores (tcgen05), for soft-max heads,
// differential heads (two maps) and sigmoid heads.  What becomes of a head's weighted sums is the including file's.
//
// A CTA owns 128 rows of queries: tokens x the query heads of one key head (for two maps: 64 of those, then the same 64 with the
// second map), so a key tile is read once for the whole group and its causal edge is short.  Queries and weights are fp32 numbers and
// stay so: each is the sum of three bf16 numbers (split3), so a product with a bf16 key or value is three products of the tensor cores,
// exact before they are added up in fp32 tensor memory (which truncates the running sum once per 16 of them: a score is off by up to 3 D / 16
// steps of 2^-23, a weighted sum by half a step of 2^-24 per 16 keys and part; below the bf16 of the result).
//
//   scores   S [128][64 keys] = (q_l + q_m + q_h) K^T: queries in shared memory, K tile K-major as the cache rows lie
//   weights  two threads a row (32 keys each, no shuffles): tcgen05.ld, soft cap, mask, exp or sigmoid, split, back to tensor memory over the scores
//   output   O [128][Dv] += (p_l + p_m + p_h) V: weights from tensor memory, the V tile as the cache rows lie (MN-major B operand)
//
// Two groups of eight warps take the key tiles alternately, each with its own scores, maximum, sum and output, so the tensor cores work
// for one group while the other one computes weights; the two are added up at the end.  A warp stages the K tiles, one the V tiles
// (cp.async, page table per row), one warp issues every MMA.  Soft-max scores are counted in powers of two.  A maximum is kept until a score exceeds it by 8 log2 e (the weights
// then reach e^8, and sum and output are relative to the kept one all the same), so the output is hardly ever rescaled.
//
// An infinite number is not the sum of its three parts (inf, NaN, NaN), and a part of a finite query or weight that is zero makes NaN of an
// infinite key or value; so does a weight of zero of a value that the row does not see.  A row whose sums are not all finite is therefore
// computed once more over its visible keys by fp32 multiply-adds (plain_row): an infinite key, value or query gives what the plain
// arithmetic gives for it.
//
// What bounds it: the instructions around the weights (two numbers an instruction where the unit has a packed form: fma.rn.f32x2), then the
// MMAs.  1024 tokens x 16 heads of 128 (4 key heads) at position 1024, window 1024 + 4 kept positions, soft cap, gate: 41 us, 210 TFLOP/s of
// the products asked for (57 us with four warps a group and one thread a row, number by number; 785 us by the fp32 CUDA cores, tiles of 32
// queries x 32 keys); 777 tokens of sigmoid heads at position 1024, no window: 53 us (64 us; 686 us).
#pragma once

#include <algorithm>

#include "dense.cuh"
#include "tc.cuh"

namespace tile_attn {

constexpr int kRows = 128, kKeys = 64; // rows of a CTA, keys of a tile
constexpr int kWarps = 16;              // that turn scores into weights
constexpr int kThreads = 32 * (kWarps + 4), kMmaWarp = kWarps + 2;
constexpr int kMaxBlocks = 3; // 64-wide blocks of a key or value: D, Dv <= 192
constexpr int kBarWords = 64; // barriers, tensor-memory slot, `dead`, in 4-byte words

enum { SOFTMAX = 0, SIGMOID = 1 };

struct shape {
    const float *q; // [T][H][MAPS][D]
    const __nv_bfloat16 *cache;
    int64_t cache_ld;
    const int32_t *table;
    int B;
    const int32_t *pos0;
    int64_t T;
    int H, G, D, Dv;
    int64_t window;
    int chunked;
    int64_t keep;
    float cap;
    const float *r1, *r2, *pb; // sigmoid heads: distance penalty and offset
    int *wait_error;
};

constexpr int kStats = 12; // rows of 128 numbers: maximum and sum at the end; per group and half a row's maxima, two tables (softmax), later sums
inline int pad64(int n) { return (n + 63) / 64 * 64; }
// sigmoid heads: penalties of one tile, a row of them per head of the group, rows of a warp in different banks
__host__ __device__ inline int pen_pitch(int TQ, int hpg) { return (TQ + kKeys + 31) / 32 * 32 + (hpg <= 32 ? 32 / hpg : 1); }
inline size_t smem_bytes(int mode, int maps, int D, int Dv, int hpg) {
    const size_t tiles = (size_t)3 * kRows * pad64(D) * 2 + 2 * (size_t)kKeys * (maps * pad64(D) + pad64(Dv)) * 2;
    const size_t finish = (size_t)kRows * (Dv + 1) * 4; // the output rows, over the tiles
    const size_t pen = mode == SIGMOID ? (size_t)2 * hpg * pen_pitch(kRows / maps / hpg, hpg) * 4 : 0;
    return 1024 + (tiles > finish ? tiles : finish) + kBarWords * 4 + (size_t)kStats * kRows * 4 + pen;
}
// Sizes the kernel takes (bf16 cache).  D, Dv and the offsets of a head's keys and values in a cache row are whole 16-byte pieces and
// whole MMA steps; tensor memory holds 2 x (scores of the maps, then weights) + 2 x Dv columns.
// From 32 tokens on, as the CUDA-core tile form that stays for fp32 caches and other sizes: fewer tokens spread their keys over CTAs.
inline bool fits(int mode, int maps, int D, int Dv, int H, int G, const float *q, const void *cache, int64_t T) {
    return T >= 32 && D % 16 == 0 && D <= 64 * kMaxBlocks && Dv % 16 == 0 && Dv <= 128 && H / G <= kRows / maps && (uintptr_t)cache % 16 == 0 && (uintptr_t)q % 16 == 0 &&
           smem_bytes(mode, maps, D, Dv, H / G) <= 227 * 1024;
}

__device__ __forceinline__ int64_t first_visible(int64_t i, int64_t size, int chunked) {
    if (size <= 0) return 0;
    return chunked ? i - i % size : max((int64_t)0, i - size + 1);
}
// cap * tanh(s / cap) of 16 scores without a branch per score.  |y| <= 0.6: an odd polynomial, coefficients fitted to tanh by least
// squares at Chebyshev nodes (largest relative error 1.3 x 2^-24 with these roundings); beyond: 1 - 2 e / (1 + e), e = exp(-2 |y|), computed
// only when a score of the warp is that large.
__device__ __forceinline__ void soft_cap16(float *z, float cap, float inv_cap) {
    const f32x2 ic = pack2(inv_cap, inv_cap), cc = pack2(cap, cap);
    auto both = [](float v) { return pack2(v, v); };
    f32x2 y[8], t[8];
    float big = 0.f;
#pragma unroll
    for (int c = 0; c < 8; c++) {
        y[c] = mul2(pack2(z[2 * c], z[2 * c + 1]), ic);
        const float2 v = unpack2(y[c]);
        big = fmaxf(big, fmaxf(fabsf(v.x), fabsf(v.y)));
    }
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const f32x2 u = mul2(y[c], y[c]);
        f32x2 p = fma2(u, both(-0.005893945228308439f), both(0.020794617012143135f));
        p = fma2(u, p, both(-0.053783293813467026f));
        p = fma2(u, p, both(0.13331915438175201f));
        p = fma2(u, p, both(-0.33333298563957214f));
        t[c] = fma2(mul2(y[c], u), p, y[c]);
    }
    if (__any_sync(0xffffffffu, !(big <= 0.6f))) {
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const float2 yv = unpack2(y[c]), tv = unpack2(t[c]);
            float w[2] = {tv.x, tv.y};
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float v = e ? yv.y : yv.x, ay = fabsf(v), x = expf(-2.0f * ay);
                const float b = fmaf(-2.0f * x, __frcp_rn(1.0f + x), 1.0f);
                w[e] = ay <= 0.6f ? w[e] : copysignf(b, v); // (a NaN stays one: x is)
            }
            t[c] = pack2(w[0], w[1]);
        }
    }
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const float2 v = unpack2(mul2(cc, t[c]));
        z[2 * c] = v.x, z[2 * c + 1] = v.y;
    }
}
// 1 / (1 + exp(-z)): the reciprocal by one Newton step from the approximate one (no division's slow path); exp(-z) stays finite, a NaN
// stays one
__device__ __forceinline__ float sigmoid_fast(float z) {
    float e, r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(e) : "f"(-z), "f"(88.0f));
    const float d = 1.0f + expf(e);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fmaf(r, fmaf(-d, r, 1.0f), r);
}
// the same for two numbers.  exp(x) = 2^t (1 + ln 2 r), t = x log2 e rounded, r what the rounding left (rms error 6e-8; expf 4e-8,
// t alone 1.2e-6 at 87).  -z is kept within
// +-88 (beyond, the result is 0 or 1 to 32 bits).
__device__ __forceinline__ f32x2 sigmoid_fast2(f32x2 z) {
    auto both = [](float v) { return pack2(v, v); };
    const float2 v = unpack2(z);
    float x, y, rx, ry;
    asm("min.NaN.f32 %0, %1, %2;\nmax.NaN.f32 %0, %0, %3;" : "=f"(x) : "f"(-v.x), "f"(88.0f), "f"(-88.0f));
    asm("min.NaN.f32 %0, %1, %2;\nmax.NaN.f32 %0, %0, %3;" : "=f"(y) : "f"(-v.y), "f"(88.0f), "f"(-88.0f));
    const f32x2 a = pack2(x, y), t = mul2(a, both(kLog2e)), rest = fma2(a, both(kLog2e), mul2(t, both(-1.f)));
    const f32x2 r = fma2(a, both(kLog2eRest), rest); // log2 e is not an fp32 number: what is missing goes with the rest
    const float2 tv = unpack2(t);
    f32x2 e = pack2(ex2_approx(tv.x), ex2_approx(tv.y));
    e = fma2(mul2(e, r), both(kLn2), e);
    const f32x2 d = add2(e, both(1.f));
    const float2 dv = unpack2(d);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rx) : "f"(dv.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ry) : "f"(dv.y));
    const f32x2 q = pack2(rx, ry), err = fma2(mul2(d, both(-1.f)), q, both(1.f));
    return fma2(q, err, q);
}
__device__ __forceinline__ float penalty(float r1, float r2, int64_t dist) { return dist > 0 ? r1 * log1pf(r2 * (float)dist) : 0.f; }

// the key tiles of a CTA: those of the kept positions [0, n_keep) first, then [jlo, i_last]
struct tiles {
    int64_t jlo, n_keep, i_last;
    int n_kt, n;
    __device__ __forceinline__ tiles(int64_t jlo_, int64_t keep, int64_t i_last_) : jlo(jlo_), n_keep(min(keep, jlo_)), i_last(i_last_) {
        n_kt = (int)((n_keep + kKeys - 1) / kKeys);
        n = n_kt + (int)((i_last - jlo) / kKeys) + 1;
    }
    __device__ __forceinline__ int64_t first(int t) const { return t < n_kt ? (int64_t)kKeys * t : jlo + (int64_t)kKeys * (t - n_kt); }
    __device__ __forceinline__ int64_t last(int t) const { return t < n_kt ? n_keep - 1 : i_last; } // last position a tile may hold
};

// barriers of a CTA, byte offsets: two stages each of K, V, scores and weights
enum { K_FULL = 0, K_FREE = 16, V_FULL = 32, V_FREE = 48, S_FULL = 64, P_FULL = 80, DONE = 96, Q_FULL = 104, SLOT = 128 };

struct mma_args {
    uint32_t bars, sq, q_split, sk, k_stage, k_part, sv, v_stage, tmem, reg_cols, o_col;
    int ksteps, Dv, NT;
    volatile int *dead;
};
// the warp that issues every MMA.  KS: D / 16, or 0 for a number known at run time only
template <int MAPS, bool SPLIT, int KS> __device__ __forceinline__ void mma_role(const mma_args &m) {
    const uint32_t id_s = umma_idesc(128, kKeys), id_o = umma_idesc(128, m.Dv, true);
    const uint32_t q_lo = umma_desc_lo(m.sq, 16), k_lo = umma_desc_lo(m.sk, 16), v_lo = umma_desc_lo(m.sv, kKeys * 128);
    auto scores = [&](int n) {
        const uint32_t s = n & 1;
        mbar_wait_bounded(m.bars + K_FULL + 8 * s, (n >> 1) & 1, m.dead);
        tc_fence_after();
#pragma unroll
        for (int mp = 0; mp < MAPS; mp++) {
            const uint32_t d = m.tmem + s * m.reg_cols + mp * 64, kl = k_lo + ((s * m.k_stage + mp * m.k_part) >> 4);
            if (KS > 0) {
#pragma unroll
                for (int part = 2; part >= 0; part--) { // the small parts first
                    const uint32_t ql = q_lo + part * ((KS + 3) / 4 * (kRows * 8));
#pragma unroll
                    for (int k = 0; k < KS; k++) // 16 numbers are 2 descriptor units, 64 a block of rows
                        umma_ss(d, ql + (k >> 2) * (kRows * 8) + 2 * (k & 3), kl + (k >> 2) * (kKeys * 8) + 2 * (k & 3), id_s, part < 2 || k > 0);
                }
            } else {
                uint32_t acc = 0;
                for (int part = 2; part >= 0; part--)
                    for (int k = 0; k < m.ksteps; k++) {
                        umma_ss(d, q_lo + part * (m.q_split >> 4) + (k >> 2) * (kRows * 8) + 2 * (k & 3), kl + (k >> 2) * (kKeys * 8) + 2 * (k & 3), id_s, acc);
                        acc = 1;
                    }
            }
        }
        umma_arrive(m.bars + S_FULL + 8 * s);
        umma_arrive(m.bars + K_FREE + 8 * s);
    };
    if (SPLIT && m.NT == 0) return;
    mbar_wait_bounded(m.bars + Q_FULL, 0, m.dead);
    scores(0);
    if (m.NT > 1) scores(1);
    for (int n = 0; n < m.NT; n++) {
        const uint32_t s = n & 1;
        mbar_wait_bounded(m.bars + P_FULL + 8 * s, (n >> 1) & 1, m.dead);
        mbar_wait_bounded(m.bars + V_FULL + 8 * s, (n >> 1) & 1, m.dead);
        tc_fence_after();
        const uint32_t o = m.tmem + m.o_col + s * m.Dv, p = m.tmem + s * m.reg_cols, vl = v_lo + ((s * m.v_stage) >> 4);
#pragma unroll
        for (int part = 2; part >= 0; part--)
#pragma unroll
            for (int k = 0; k < kKeys / 16; k++) // 16 keys: two groups of 8 rows of 128 bytes
                umma_ts(o, p + k * 24 + part * 8, vl + k * 128, id_o, part < 2 || k > 0 ? 1u : n >= 2);
        umma_arrive(m.bars + V_FREE + 8 * s);
        if (n + 2 < m.NT) scores(n + 2); // behind this tile's weights: the MMAs of a thread run in order
    }
    umma_arrive(m.bars + DONE);
}

struct row_job {
    const float *q;
    const __nv_bfloat16 *k, *v; // a head's keys (of the map) and values in cache row 0
    int64_t ld;
    const int32_t *table;
    int B;
    int64_t lo, keep, i; // positions [0, min(keep, lo)) and [lo, i]
    int D, Dv;
    float cap, r1, r2, pb;
};
// one row by one warp, a key a lane: weighted sums to out[Dv], maximum and denominator to *m_out and *l_out
template <int MODE> __device__ __forceinline__ void plain_row(const row_job &j, float *out, float *m_out, float *l_out) {
    const int lane = threadIdx.x & 31;
    const int64_t n_keep = MODE == SOFTMAX ? min(j.keep, j.lo) : 0, total = n_keep + (j.i - j.lo + 1);
    float acc[4] = {0.f, 0.f, 0.f, 0.f}, m = -INFINITY, l = 0.f; // Dv <= 128
    for (int64_t n0 = 0; n0 < total; n0 += 32) {
        const int keys = (int)min((int64_t)32, total - n0);
        const int64_t n = n0 + min(lane, keys - 1), at = n < n_keep ? n : j.lo + (n - n_keep);
        const int64_t row = ((int64_t)j.table[at / j.B] * j.B + at % j.B) * j.ld;
        float s = 0.f, p = 0.f;
        for (int d = 0; d < j.D; d++) s = fmaf(to_f32(j.k[row + d]), j.q[d], s);
        if (MODE == SOFTMAX) {
            if (j.cap > 0.f) s = j.cap * tanhf(s / j.cap);
            const float mx = fmaxf(m, warp_max_f32(lane < keys ? s : -INFINITY)), corr = mx == -INFINITY ? 1.f : expf(m - mx);
            if (lane < keys && s != -INFINITY) p = expf(s - mx);
            l = fmaf(l, corr, warp_sum_f32(p));
            for (int r = 0; r < 4; r++) acc[r] *= corr;
            m = mx;
        } else if (lane < keys) {
            p = sigmoid_fast(s - penalty(j.r1, j.r2, j.i - at) + j.pb);
        }
        for (int u = 0; u < keys; u++) {
            const float pu = __shfl_sync(0xffffffffu, p, u);
            const __nv_bfloat16 *v = j.v + __shfl_sync(0xffffffffu, row, u);
            for (int r = 0; r < 4; r++)
                if (lane + 32 * r < j.Dv) acc[r] = fmaf(pu, to_f32(v[lane + 32 * r]), acc[r]);
        }
    }
    for (int r = 0; r < 4; r++)
        if (lane + 32 * r < j.Dv) out[lane + 32 * r] = acc[r];
    if (lane == 0) *m_out = m, *l_out = l;
    __syncwarp();
}

// the rows first + step b of a CTA, b the set bits, once more; out of line, so that the code that every call runs through stays short
template <int MODE, int MAPS>
__device__ __noinline__ void plain_rows(const shape &a, uint32_t again, int first, int step, int64_t t0, int64_t i0, int g, int hpg, int n_pairs, float *of, float *st) {
    constexpr int PR = kRows / MAPS;
    while (again) {
        const int rr = first + step * (__ffs((int)again) - 1), rm = MAPS == 1 ? 0 : rr / PR, rp = rr - rm * PR, rq = rp / hpg, h = g * hpg + (rp - rq * hpg);
        again &= again - 1;
        if (rp >= n_pairs) continue;
        row_job j{a.q + (((t0 + rq) * a.H + h) * MAPS + rm) * a.D, a.cache + ((int64_t)g * MAPS + rm) * a.D, a.cache + (int64_t)a.G * MAPS * a.D + (int64_t)g * a.Dv,
                  a.cache_ld, a.table, a.B, first_visible(i0 + rq, a.window, a.chunked), MODE == SOFTMAX ? a.keep : 0, i0 + rq, a.D, a.Dv, a.cap, 0.f, 0.f, 0.f};
        if (MODE == SIGMOID && a.r1) j.r1 = a.r1[h], j.r2 = a.r2[h];
        if (MODE == SIGMOID && a.pb) j.pb = a.pb[h];
        plain_row<MODE>(j, of + rr * (a.Dv + 1), st + rr, st + kRows + rr);
    }
}

// Few CTAs take a cluster each, whose `parts` CTAs have the key tiles in turn.  One row of it by one warp: the parts' sums from their shared memory, added in order
// relative to the largest maximum, over this CTA's.  false: one of them is not finite
template <int MODE> __device__ __forceinline__ bool gather_row(int parts, int rr, int Dv, float *of, float *st) {
    const int lane = threadIdx.x & 31;
    const float odd = lane < 4 * parts ? ld_cluster_f32(cluster_addr(smem_u32(st + (2 + (lane & 3)) * kRows + rr), lane >> 2)) : 0.f; // a part's four quarters
    if (__any_sync(0xffffffffu, odd != 0.f)) return false;
    const uint32_t row = smem_u32(of + rr * (Dv + 1));
    float f = lane < parts ? 1.f : 0.f;
    if (MODE == SOFTMAX) {
        const uint32_t at = cluster_addr(smem_u32(st + rr), min(lane, parts - 1));
        const float m = ld_cluster_f32(at), l = ld_cluster_f32(at + 4 * kRows), M = warp_max_f32(lane < parts ? m : -INFINITY);
        f = lane < parts && m != -INFINITY ? expf(m - M) : 0.f;
        float L = 0.f;
        for (int z = 0; z < parts; z++) L = fmaf(__shfl_sync(0xffffffffu, l, z), __shfl_sync(0xffffffffu, f, z), L);
        if (lane == 0) st[rr] = M, st[kRows + rr] = L;
    }
    float x[4] = {0.f, 0.f, 0.f, 0.f}; // Dv <= 128
    for (int z = 0; z < parts; z++) {
        const uint32_t from = cluster_addr(row, z) + 4 * lane;
        const float fz = __shfl_sync(0xffffffffu, f, z);
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (lane + 32 * u < Dv) x[u] = fmaf(ld_cluster_f32(from + 128 * u), fz, x[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
        if (lane + 32 * u < Dv) of[rr * (Dv + 1) + lane + 32 * u] = x[u];
    return true;
}

// FIN: what becomes of a row, a warp's work when the sums stand in shared memory: load() requests what a row needs from memory, row()
// gets it with the sums of the row (of both maps) and their maximum and denominators
// SPLIT: a cluster of CTAs shares the key tiles
template <int MODE, int MAPS, bool SPLIT, typename FIN>
__global__ void __launch_bounds__(kThreads, 1) attn_kernel(const __grid_constant__ shape a, const FIN fin) {
    extern __shared__ uint8_t ta_raw[];
    const uint32_t raw0 = smem_u32(ta_raw), base = (raw0 + 1023u) & ~1023u;
    uint8_t *gbase = ta_raw + (base - raw0);
    const int D64 = (a.D + 63) / 64, V64 = (a.Dv + 63) / 64;
    const uint32_t q_split = (uint32_t)D64 * kRows * 128;                         // bytes of one of the three parts of q
    const uint32_t k_part = (uint32_t)D64 * kKeys * 128, k_stage = MAPS * k_part; // a map's keys, a stage
    const uint32_t v_stage = (uint32_t)V64 * kKeys * 128;
    const uint32_t sk = base + 3 * q_split, sv = sk + 2 * k_stage;
    const uint32_t tiles_end = 3 * q_split + 2 * (k_stage + v_stage), of_end = (uint32_t)kRows * (a.Dv + 1) * 4;
    const uint32_t ctl = max(tiles_end, of_end); // multiples of 512 bytes
    const uint32_t bars = base + ctl;
    uint32_t *ctlw = reinterpret_cast<uint32_t *>(gbase + ctl);
    volatile int *dead = reinterpret_cast<volatile int *>(ctlw + 40);
    float *st = reinterpret_cast<float *>(ctlw + kBarWords); // [group][m, l][128]
    float *pen = st + kStats * kRows;                        // sigmoid: [group][heads][pitch]

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    constexpr int PR = kRows / MAPS; // (token, head) pairs of a CTA
    const int g = blockIdx.y, hpg = a.H / a.G, TQ = PR / hpg;
    // the CTAs with the most keys first
    const int64_t t0 = (int64_t)(gridDim.x - 1 - blockIdx.x) * TQ;
    const int nq = (int)min((int64_t)TQ, a.T - t0), n_pairs = nq * hpg;
    if (tid == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(bars + K_FULL + 8 * s, 1);
            mbar_init(bars + K_FREE + 8 * s, 1);
            mbar_init(bars + V_FULL + 8 * s, 1);
            mbar_init(bars + V_FREE + 8 * s, 1);
            mbar_init(bars + S_FULL + 8 * s, 1);
            mbar_init(bars + P_FULL + 8 * s, 8);
        }
        mbar_init(bars + DONE, 1);
        mbar_init(bars + Q_FULL, kWarps);
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) tmem_alloc512(bars + SLOT);
    early_wait();
    const int64_t i0 = (int64_t)*a.pos0 + t0, i_last = i0 + nq - 1;
    const tiles tl(first_visible(i0, a.window, a.chunked), MODE == SOFTMAX ? a.keep : 0, i_last);
    // tiles z, z + parts, ...; three a part at least, and a CTA too many has none
    const int z = SPLIT ? blockIdx.z : 0, parts = SPLIT ? max(1, min((int)gridDim.z, tl.n / 3)) : 1, NT = !SPLIT ? tl.n : z < parts ? (tl.n - 1 - z) / parts + 1 : 0;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    step_next();
    const uint32_t tmem = __shfl_sync(0xffffffffu, ctlw[SLOT / 4], 0);
    const uint32_t reg_cols = MAPS == 1 ? 96 : 128; // scores [MAPS][64], then weights over them
    const uint32_t o_col = 2 * reg_cols;

    if (warp == kWarps || warp == kWarps + 1) {
        // ---- a warp stages K, one V: eight lanes a 128-byte piece of a row
        const bool is_k = warp == kWarps;
        const int sub = lane >> 3, pc = lane & 7;
        const int pcs = (is_k ? a.D : a.Dv) / 8; // 16-byte pieces of a row (and map)
        const uint32_t stage_bytes = is_k ? k_stage : v_stage, s0 = is_k ? sk : sv;
        const int full = is_k ? K_FULL : V_FULL, fre = is_k ? K_FREE : V_FREE;
        const __nv_bfloat16 *part0 = a.cache + (is_k ? (int64_t)g * MAPS * a.D : (int64_t)a.G * MAPS * a.D + (int64_t)g * a.Dv);
        // row 4 k + sub of the tile goes to 512 k + 128 sub, its piece pc to place pc ^ (row & 7): two patterns, k even and odd
        const uint32_t at0 = s0 + sub * 128 + ((pc ^ sub) << 4), at1 = s0 + sub * 128 + ((pc ^ (sub + 4)) << 4);
        for (int n = 0; n < NT; n++) {
            const int s = n & 1;
            // lane = row for the page table; a row past the last one repeats it (weight 0)
            uint32_t my_row[2];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const uint32_t j = (uint32_t)min(tl.first(z + n * parts) + 32 * u + lane, tl.last(z + n * parts)), pg = j / (uint32_t)a.B;
                my_row[u] = (uint32_t)a.table[pg] * (uint32_t)a.B + (j - pg * a.B);
            }
            if (n >= 2) mbar_wait_warp(bars + fre + 8 * s, ((n >> 1) - 1) & 1, dead);
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const __nv_bfloat16 *row = part0 + __shfl_sync(0xffffffffu, my_row[k >> 3], (4 * k + sub) & 31) * (uint64_t)a.cache_ld + 8 * pc;
                const uint32_t dst = ((k & 1) ? at1 : at0) + s * stage_bytes + k * 512;
#pragma unroll
                for (int mp = 0; mp < MAPS; mp++)
#pragma unroll
                    for (int c = 0; c < kMaxBlocks; c++)
                        if (8 * c + pc < pcs && (mp == 0 || is_k)) cp_async16(dst + mp * k_part + (uint32_t)c * (kKeys * 128), row + mp * a.D + 64 * c);
            }
            // handed over before the next stage is waited for: that one is only freed behind this tile
            cp_async_commit();
            cp_async_wait<0>();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + full + 8 * s);
        }
    } else if (warp == kMmaWarp) {
        // the whole warp, converged; a number of K steps known to the compiler makes an MMA a few instructions
        const mma_args ma{bars, base, q_split, sk, k_stage, k_part, sv, v_stage, tmem, reg_cols, o_col, a.D / 16, a.Dv, NT, dead};
        if (a.D == 128) mma_role<MAPS, SPLIT, 8>(ma);
        else if (a.D == 64) mma_role<MAPS, SPLIT, 4>(ma);
        else mma_role<MAPS, SPLIT, 0>(ma);
    } else if (warp < kWarps && (!SPLIT || NT > 0)) {
        // the rows of q as three bf16 numbers each, rows and coordinates past the end as zeros: four numbers a thread, eight loads in flight
        {
            const int gpr = 16 * D64, n_items = kRows * gpr;
            for (int it0 = tid; it0 < n_items; it0 += 8 * 32 * kWarps) {
                float4 x[8];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int it = it0 + 32 * kWarps * u, r = it / gpr, d = 4 * (it - r * gpr);
                    const int mp = MAPS == 1 ? 0 : r / PR, pr = MAPS == 1 ? r : r - mp * PR, qi = pr / hpg;
                    x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (it < n_items && pr < n_pairs && d < a.D)
                        x[u] = *reinterpret_cast<const float4 *>(a.q + (((t0 + qi) * a.H + (int64_t)g * hpg + (pr - qi * hpg)) * MAPS + mp) * a.D + d);
                }
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int it = it0 + 32 * kWarps * u, r = it / gpr, d = 4 * (it - r * gpr);
                    if (it >= n_items) break;
                    uint32_t h[2], m[2], l[2];
                    f32x2 q01 = pack2(x[u].x, x[u].y), q23 = pack2(x[u].z, x[u].w);
                    if (MODE == SOFTMAX) q01 = mul2(q01, pack2(kLog2e, kLog2e)), q23 = mul2(q23, pack2(kLog2e, kLog2e)); // scores in powers of two
                    split3(q01, h[0], m[0], l[0]);
                    split3(q23, h[1], m[1], l[1]);
                    const uint32_t at = base + (uint32_t)(d >> 6) * (kRows * 128) + r * 128 + ((((d >> 3) & 7) ^ (r & 7)) << 4) + (d & 4) * 2;
                    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at), "r"(h[0]), "r"(h[1]) : "memory");
                    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at + q_split), "r"(m[0]), "r"(m[1]) : "memory");
                    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at + 2 * q_split), "r"(l[0]), "r"(l[1]) : "memory");
                }
            }
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bars + Q_FULL);
        // ---- weights: group grp takes the tiles n = grp, grp + 2, ...; a thread owns 32 keys of one row, two threads the row
        const int grp = warp >> 3, half = (warp >> 2) & 1, lq = warp & 3, r = 32 * lq + lane;
        const int mp = MAPS == 1 ? 0 : r / PR, pr = MAPS == 1 ? r : r - mp * PR, qi = pr / hpg, hh = pr - qi * hpg;
        const int64_t i = i0 + qi, lo = first_visible(i, a.window, a.chunked);
        const bool live = pr < n_pairs;
        const uint32_t lanes = (uint32_t)(32 * lq) << 16;
        const uint32_t ts = tmem + lanes + grp * reg_cols, to = tmem + lanes + o_col + grp * a.Dv;
        const float cap = a.cap * kLog2e, inv_cap = a.cap > 0.f ? kLn2 / a.cap : 0.f;
        float m = -INFINITY, l = 0.f, hpb = 0.f;
        const int pitch = pen_pitch(TQ, hpg);
        float *mypen = pen + grp * hpg * pitch;
        if (MODE == SIGMOID && a.pb && live) hpb = a.pb[g * hpg + hh];
        for (int n = grp; n < NT; n += 2) {
            const int tile = z + n * parts;
            const int64_t j0 = tl.first(tile), jl = min(tl.last(tile), j0 + kKeys - 1);
            const bool whole = jl - j0 == kKeys - 1 && jl <= i0 && (tile < tl.n_kt || j0 >= first_visible(i_last, a.window, a.chunked));
            if (MODE == SIGMOID && a.r1) { // the penalties a tile can meet: distances (i0 - j0) + qi - jj, qi < TQ, jj < 64
                if (n > grp) bar_sync(1 + grp, 256);
                for (int e = (tid & 255); e < hpg * (TQ + kKeys - 1); e += 256) {
                    const int eh = e / (TQ + kKeys - 1), ed = e - eh * (TQ + kKeys - 1);
                    mypen[eh * pitch + ed] = penalty(a.r1[g * hpg + eh], a.r2[g * hpg + eh], i0 - j0 + ed - (kKeys - 1));
                }
            }
            mbar_wait_warp(bars + S_FULL + 8 * grp, (n >> 1) & 1, dead);
            tc_fence_after();
            // the first and one past the last visible key of the row, from j0; a kept prefix inside a window tile as a third bound
            int c_lo = 0, c_hi = kKeys, c_keep = 0;
            if (!whole) {
                const int64_t hi = min(jl, i) - j0 + 1, lo_c = lo - j0, kp = a.keep - j0;
                c_hi = live ? (int)max((int64_t)0, min((int64_t)kKeys, hi)) : 0;
                c_lo = (int)max((int64_t)0, min((int64_t)kKeys, lo_c));
                c_keep = MODE == SOFTMAX ? (int)max((int64_t)0, min((int64_t)kKeys, kp)) : 0;
            }
            // both halves' scores are in registers before either one's weights go over them (the barrier)
            float x[2][16], mm = 0.f;
            f32x2 sum[2] = {0, 0};
            auto masked = [&](float *y, int c0, float none) {
#pragma unroll
                for (int c = 0; c < 16; c++) y[c] = (c0 + c < c_hi && (c0 + c >= c_lo || c0 + c < c_keep)) ? y[c] : none;
            };
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int c0 = 32 * half + 16 * k;
                tmem_load16(ts + mp * 64 + c0, reinterpret_cast<uint32_t *>(x[k]));
                if (MODE != SOFTMAX) continue;
                if (a.cap > 0.f) soft_cap16(x[k], cap, inv_cap);
                if (!whole) masked(x[k], c0, -INFINITY);
#pragma unroll
                for (int c = 0; c < 16; c++) mx4[c & 3] = fmaxf(mx4[c & 3], x[k][c]);
            }
            if (MODE == SOFTMAX) {
                float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                float *swap = st + (4 + 4 * ((n >> 1) & 1) + 2 * grp) * kRows + r; // two tables: the next tile writes the other one
                swap[half * kRows] = mx;
                bar_sync(1 + grp, 256);
                mx = fmaxf(mx, swap[(half ^ 1) * kRows]);
                float corr = 1.f;
                const bool grow = mx > m + 8.f * kLog2e || (m == -INFINITY && mx > -INFINITY);
                if (grow) {
                    corr = exp2f(m - mx); // m = -inf: 0
                    m = mx;
                    l *= corr;
                }
                if (n >= 2 && __any_sync(0xffffffffu, grow)) { // the tile before has been added: its MMAs precede this tile's scores
#pragma unroll 1
                    for (int c = 16 * half; c < a.Dv; c += 32) {
                        uint32_t o[16];
                        tmem_load16(to + c, o);
#pragma unroll
                        for (int u = 0; u < 16; u++) o[u] = __float_as_uint(__uint_as_float(o[u]) * corr);
                        tmem_store16(to + c, o);
                    }
                }
                mm = m == -INFINITY ? 0.f : m; // nothing visible yet: every weight is exp(-inf) = 0
            } else {
                bar_sync(1 + grp, 256);
            }
            const float *prow = MODE == SIGMOID ? mypen + hh * pitch + qi + kKeys - 1 : nullptr;
            // the weights of 16 keys go to 24 columns [p_h | p_m | p_l] from 24 k on
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int c0 = 32 * half + 16 * k;
                float *y = x[k];
                f32x2 w[8];
                if (MODE == SOFTMAX) {
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        const float2 t = unpack2(add2(pack2(y[2 * c], y[2 * c + 1]), pack2(-mm, -mm)));
                        w[c] = pack2(ex2_approx(t.x), ex2_approx(t.y));
                        sum[c & 1] = add2(sum[c & 1], w[c]);
                    }
                } else {
                    if (a.r1) {
#pragma unroll
                        for (int c = 0; c < 16; c++) y[c] -= prow[-(c0 + c)];
                    }
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        const float2 v = unpack2(sigmoid_fast2(add2(pack2(y[2 * c], y[2 * c + 1]), pack2(hpb, hpb))));
                        y[2 * c] = v.x, y[2 * c + 1] = v.y;
                    }
                    if (!whole) masked(y, c0, 0.f);
#pragma unroll
                    for (int c = 0; c < 8; c++) w[c] = pack2(y[2 * c], y[2 * c + 1]);
                }
                uint32_t ph[8], pm[8], pl[8];
#pragma unroll
                for (int c = 0; c < 8; c++) split3(w[c], ph[c], pm[c], pl[c]);
                const uint32_t tp = ts + (c0 >> 4) * 24;
                tmem_store8(tp, ph);
                tmem_store8(tp + 8, pm);
                tmem_store8(tp + 16, pl);
            }
            const float2 s2 = unpack2(add2(sum[0], sum[1]));
            l += s2.x + s2.y;
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + P_FULL + 8 * grp);
        }
        // ---- both groups' sums meet: O = O_0 f_0 + O_1 f_1 relative to the larger maximum, as rows in shared memory
        const int quarter = 2 * grp + half;
        mbar_wait_warp(bars + DONE, 0, dead); // all MMAs are done: the tiles are no longer read
        tc_fence_after();
        bar_sync(3, 32 * kWarps);
        if (MODE == SOFTMAX) {
            st[(4 + quarter) * kRows + r] = l;
            if (half == 0) st[(2 + grp) * kRows + r] = m;
            bar_sync(3, 32 * kWarps);
        }
        float f0 = 1.f, f1 = NT > 1 ? 1.f : 0.f, M = 0.f, L = 1.f;
        if (MODE == SOFTMAX) {
            const float m0 = st[2 * kRows + r], l0 = st[4 * kRows + r] + st[5 * kRows + r], m1 = st[3 * kRows + r], l1 = st[6 * kRows + r] + st[7 * kRows + r];
            M = fmaxf(m0, m1) * kLn2;
            f0 = over_e(m0, M);
            f1 = over_e(m1, M);
            L = l0 * f0 + l1 * f1;
            bar_sync(3, 32 * kWarps);
            if (quarter == 0) {
                st[r] = M;
                st[kRows + r] = L;
            }
        }
        float *of = reinterpret_cast<float *>(gbase);
        const int op = a.Dv + 1, n16 = a.Dv / 16;
        float odd = MODE == SOFTMAX ? 0.f * L : 0.f; // 0, or NaN when a sum of the row is not finite
        for (int cb = quarter; cb < n16; cb += 4) {
            uint32_t o0[16], o1[16];
            tmem_load16(tmem + lanes + o_col + 16 * cb, o0);
            if (NT > 1) tmem_load16(tmem + lanes + o_col + a.Dv + 16 * cb, o1);
#pragma unroll
            for (int u = 0; u < 16; u++) {
                float v = __uint_as_float(o0[u]) * f0;
                if (NT > 1) v = fmaf(__uint_as_float(o1[u]), f1, v);
                of[r * op + 16 * cb + u] = v;
                odd = fmaf(0.f, v, odd);
            }
        }
        st[(2 + quarter) * kRows + r] = odd;
        bar_sync(3, 32 * kWarps);
        if (SPLIT && parts > 1) { // this CTA's pairs: z, z + parts, ...
            __syncwarp();
            cluster_sync(); // the sums of all parts stand
            for (int p = z + parts * warp; p < n_pairs; p += parts * kWarps)
                for (int rr = p; rr < kRows; rr += PR)
                    if (!gather_row<MODE>(parts, rr, a.Dv, of, st)) plain_rows<MODE, MAPS>(a, 1u, rr, 0, t0, i0, g, hpg, n_pairs, of, st);
            __syncwarp();
            cluster_sync(); // and are read
        } else { // a warp's 8 rows: warp, warp + 16, ...; those whose sums are not finite once more, without the split
            const float *er = st + warp + kWarps * (lane & 7);
            const uint32_t again = __ballot_sync(0xffffffffu, (er[2 * kRows] + er[3 * kRows]) + (er[4 * kRows] + er[5 * kRows]) != 0.f) & 0xffu;
            if (again) plain_rows<MODE, MAPS>(a, again, warp, kWarps, t0, i0, g, hpg, n_pairs, of, st);
        }
        // a warp a row, four rows' reads from memory in flight
        for (int p0 = z + parts * warp; p0 < n_pairs; p0 += 4 * parts * kWarps) {
            typename FIN::reads rd[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int p = min(p0 + parts * kWarps * u, n_pairs - 1), pq = p / hpg;
                fin.load(rd[u], i0 + pq, t0 + pq, g * hpg + (p - pq * hpg), lane);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int p = p0 + parts * kWarps * u, pq = p / hpg;
                if (p >= n_pairs) break;
                fin.row(rd[u], of + p * op, of + (p + PR) * op, st[p], st[kRows + p], MAPS == 2 ? st[kRows + p + PR] : 0.f, t0 + pq, g * hpg + (p - pq * hpg), lane);
            }
        }
        tc_fence_before();
    }
    if (SPLIT && !(warp < kWarps && parts > 1 && NT > 0)) { // the other threads of a cluster come by both of its barriers, too
        __syncwarp();
        cluster_sync();
        cluster_sync();
    }
    __syncthreads();
    if (warp == kMmaWarp) {
        settle(dead);
        tc_fence_after();
        tmem_free512(tmem);
        if (lane == 0 && *dead) *a.wait_error = 1;
    }
}

// Few CTAs (few key heads, portions that are not long) leave SMs without work: up to eight CTAs then share a CTA's key tiles.  How many positions come before
// the portion is known on the device only, and a cluster costs 2 us (its two meetings; and more numbers than the loop over tiles has registers for), so that the portion
// itself (or its window) has to hold what saves that at position 0: three tiles a part, and ten of them where there is a maximum to find.  Soft-max heads, two parts, graph
// replays: 385 tokens x 4 heads (1 key head) of 64 17.5 us (15.3 alone), 512 18.3 (17.4), 512 x 2 (2) of 128 21.5 (20.9), 640 19.4 (19.0) and 22.8 (23.8), a window of 400 18.8 (17.2); sigmoid
// heads, 385 x 4 (1) of 64 17.0 (17.0), 640 19.4 (23.1).  Four parts, heads of 128: 1000 tokens x 4 heads (1) at position 900 26.4 us (48.5 alone).
// No more parts than clusters of them run at once: the last ones would wait for the first (777 tokens x 8 heads (8) of 64, 56 clusters of four, 36; alone 25; 2048 x 1, 16 clusters of
// eight 28.7, of four 20.3), which pays only where the first ones, without a window, have few tiles and the last ones many (4500 x 1, 36 clusters of four 34, of two 48).  With more CTAs
// than SMs two parts cost: 777 tokens of 16 sigmoid heads (4) at 1024, 100 CTAs: 63.8 (53.6).
template <int MODE, int MAPS, typename FIN> int launch(const shape &a, const FIN &fin) {
    const int TQ = kRows / MAPS / (a.H / a.G);
    const int64_t ctas = (a.T + TQ - 1) / TQ * a.G, own = (a.window > 0 ? std::min(a.T, a.window) : a.T) / kKeys; // tiles of the portion
    const size_t alone = smem_bytes(MODE, MAPS, a.D, a.Dv, a.H / a.G), shared = std::max(alone, kOneCtaSmem); // clusters with tensor memory
    auto split = attn_kernel<MODE, MAPS, true, FIN>;
    unsigned parts = 1;
    for (int rc, n; parts < 8 && own >= (MODE == SOFTMAX ? 10 : 6) && parts * 2 <= own / 3 && ctas * parts * 2 <= ggb_sm_count(); parts *= 2) {
        if ((rc = ggb_allow_smem(split, shared))) return rc;
        if ((rc = ggb_clusters_at_once_of(reinterpret_cast<const void *>(split), (int)parts * 2, kThreads, shared, &n))) return rc;
        if (ctas > n && (a.window > 0 || own < 20 * parts)) break;
    }
    const size_t smem = parts > 1 ? shared : alone;
    auto kfn = parts > 1 ? split : attn_kernel<MODE, MAPS, false, FIN>;
    const int rc = ggb_allow_smem(kfn, smem);
    if (rc) return rc;
    const ggb_cluster cluster{1, 1, parts};
    GGB_CUDA(ggb_launch_early(kfn, cluster, dim3((unsigned)((a.T + TQ - 1) / TQ), (unsigned)a.G, parts), dim3(kThreads), smem, a, fin));
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

} // namespace tile_attn
