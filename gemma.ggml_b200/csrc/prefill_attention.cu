// prefill_attention.cu — causal attention of a prompt over the fp16 KV cache (position-major [n_ctx][Hkv * d]) on the tensor cores
// (tcgen05), the batched form of the reference's nodes kq -> soft_max_ext -> kqv (ref: src/gemma_model.cpp:454-489).
//
// The reference rounds q and the weights to fp16 and the cache is fp16, so both contractions are fp16 products with fp32 sums as they stand:
//   S [128 rows][64 keys] = fp16(q) K^T, m = the row's maximum over ALL its keys, e = fp16(exp(s - m)), O [128][d] += e V, out = O / sum(e)
// (e is rounded where the older kernels round e / sum(e): one rounding less).  The maximum is known before the first weight because the
// scores are computed twice, a first time for the maximum alone: the tensor cores idle anyway, and neither the output nor the sum is ever
// rescaled.
//
// A CTA owns 128 rows: 128 / G tokens x the G query heads of one key head, so that a key tile is read once for all of them.  Two groups of
// four warps take the key tiles in turn, a thread a row; one warp requests K and V tiles (TMA, two stages each), one issues every MMA; weights
// go back to tensor memory over the scores and are the A operand of the second product.
// Where those are few CTAs (32 for 512 tokens x 8 heads of one key head), the key tiles of 128 rows are dealt to the CTAs of a cluster: the maxima meet
// between the two passes, and each CTA adds up its share of the rows from the others' shared memory, in order.
// Bound by the chain scores -> weights -> output of the CTAs with the most keys.  512 tokens x 8 heads x 256 over one key head: 81 us a layer by
// plain dot products, 25 by one CTA, 18 by four.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "prefill_attention.cuh"
#include "tc.cuh"

namespace {

constexpr int kRows = 128, kKeys = 64, kThreads = 320, kTmaWarp = 8, kMmaWarp = 9;
constexpr uint32_t kOCol = 2 * kKeys; // tensor memory: two score buffers, then the output
enum { K_FULL = 0, K_FREE = 16, V_FULL = 32, V_FREE = 48, S_FULL = 64, S_FREE = 80, P_FULL = 96, PV_DONE = 112, DONE = 128, SLOT = 136, kBarBytes = 160 };

struct attn_args {
    const float *q;
    const __half *kc, *vc;
    int T, pos0, H, Hkv, D;
    const uint16_t *exp_table;
    float *out;
    __nv_bfloat16 *out_bf16;
    int *failed;
};
struct attn_maps {
    CUtensorMap k, v;
};

__host__ __device__ inline size_t tile_bytes(int D) { return (size_t)(kRows + 4 * kKeys) * D * 2; }
inline size_t smem_bytes(int D) { return 1024 + tile_bytes(D) + kBarBytes + kRows * (2 * 4 + 2 * 8 + 4 + 4); }

__host__ __device__ constexpr uint32_t idesc_f16(int M, int N, bool b_mn) { // fp32 accumulators, A and B fp16
    return (1u << 4) | (b_mn ? 1u << 16 : 0u) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// A row whose sums are not all finite, once more in plain arithmetic by 256 threads (an infinite value behind the row's last key makes
// NaN of a zero weight in a tile).  s: at least n_kv floats, red: 16 doubles.
__device__ __noinline__ void plain_row(const attn_args &a, int t, int h, float *s, double *red) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_kv = a.pos0 + t + 1;
    const int64_t stride = (int64_t)a.Hkv * a.D, off = (int64_t)(h / (a.H / a.Hkv)) * a.D;
    const float *q = a.q + ((int64_t)t * a.H + h) * a.D;
    float m = -INFINITY;
    for (int j = tid; j < n_kv; j += 256) {
        float acc = 0.f;
        for (int d = 0; d < a.D; d++) acc = fmaf(__half2float(a.kc[j * stride + off + d]), __half2float(__float2half_rn(q[d])), acc);
        s[j] = acc;
        m = fmaxf(m, acc);
    }
    m = warp_max_f32(m);
    if (lane == 0) red[warp] = m;
    bar_sync(1, 256);
    for (int w = 0; w < 8; w++) m = fmaxf(m, (float)red[w]);
    double sum = 0.0;
    for (int j = tid; j < n_kv; j += 256) {
        const float e = half_bits_to_float(a.exp_table[float_to_half_bits(s[j] - m)]);
        s[j] = e;
        sum += (double)e;
    }
    sum = warp_sum_f64(sum);
    if (lane == 0) red[8 + warp] = sum;
    bar_sync(1, 256);
    sum = 0.0;
    for (int w = 0; w < 8; w++) sum += red[8 + w];
    const float inv = (float)(1.0 / sum);
    if (tid < a.D) {
        float o = 0.f;
        for (int j = 0; j < n_kv; j++) o = fmaf(__half2float(a.vc[j * stride + off + tid]), __half2float(__float2half_rn(s[j] * inv)), o);
        const int64_t at = ((int64_t)t * a.H + h) * a.D + tid;
        if (a.out) a.out[at] = o;
        if (a.out_bf16) a.out_bf16[at] = __float2bfloat16_rn(o);
    }
    bar_sync(1, 256);
}

// C: CTAs of a cluster, that share the key tiles
template <int C>
__global__ void __launch_bounds__(kThreads, 1) attn_prefill_tile_kernel(const __grid_constant__ attn_maps maps, const __grid_constant__ attn_args a) {
    extern __shared__ uint8_t raw[];
    const uint32_t raw0 = smem_u32(raw), base = (raw0 + 1023u) & ~1023u;
    uint8_t *gbase = raw + (base - raw0);
    const int D = a.D, blocks = D / 64;
    const uint32_t stage = (uint32_t)kKeys * D * 2; // bytes of a K or V tile
    const uint32_t sk = base + (uint32_t)kRows * D * 2, sv = sk + 2 * stage, bars = sv + 2 * stage;
    uint8_t *ctl = gbase + (bars - base);
    volatile int *dead = reinterpret_cast<volatile int *>(ctl + SLOT + 4);
    double *s_sum = reinterpret_cast<double *>(ctl + kBarBytes); // [group][row]
    float *s_max = reinterpret_cast<float *>(s_sum + 2 * kRows); // [group][row]
    float *s_inv = s_max + 2 * kRows;                            // [row]
    int *s_bad = reinterpret_cast<int *>(s_inv + kRows);         // [row]

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int g = blockIdx.y, hpg = a.H / a.Hkv, TQ = kRows / hpg;
    const int t0 = (int)(gridDim.x - 1 - blockIdx.x) * TQ; // the CTAs with the most keys first
    const int nq = min(TQ, a.T - t0), n_rows = nq * hpg;
    const int rank = C > 1 ? (int)blockIdx.z : 0, all = (a.pos0 + t0 + nq - 1) / kKeys + 1;
    const int NT = (all - rank + C - 1) / C; // key tiles rank, rank + C, ... (all >= 1, C <= 8: at least 0)

    if (tid == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(bars + K_FULL + 8 * s, 1);
            mbar_init(bars + K_FREE + 8 * s, 1);
            mbar_init(bars + V_FULL + 8 * s, 1);
            mbar_init(bars + V_FREE + 8 * s, 1);
            mbar_init(bars + S_FULL + 8 * s, 1);
            mbar_init(bars + S_FREE + 8 * s, 4);
            mbar_init(bars + P_FULL + 8 * s, 4);
            mbar_init(bars + PV_DONE + 8 * s, 1);
        }
        mbar_init(bars + DONE, 1);
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) tmem_alloc512(bars + SLOT);
    early_wait();
    if (warp < 8) { // queries, rounded to fp16: 8 numbers a step, neighbouring lanes along a row, eight steps in flight
        const int pieces = D / 8, n = kRows * pieces;
        for (int i0 = tid; i0 < n; i0 += 8 * 256) {
            float4 x[8][2];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int i = i0 + 256 * u, r = i / pieces, pc = i - r * pieces, tq = r / hpg;
                x[u][0] = x[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (i < n && r < n_rows) {
                    const float4 *src = reinterpret_cast<const float4 *>(a.q + ((int64_t)(t0 + tq) * a.H + g * hpg + (r - tq * hpg)) * D + 8 * pc);
                    x[u][0] = src[0], x[u][1] = src[1];
                }
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int i = i0 + 256 * u, r = i / pieces, pc = i - r * pieces;
                if (i >= n) break;
                const float4 y = x[u][0], z = x[u][1];
                const __half2 h[4] = {__floats2half2_rn(y.x, y.y), __floats2half2_rn(y.z, y.w), __floats2half2_rn(z.x, z.y), __floats2half2_rn(z.z, z.w)};
                *reinterpret_cast<uint4 *>(gbase + (pc >> 3) * (kRows * 128) + r * 128 + (((pc & 7) ^ (r & 7)) << 4)) = *reinterpret_cast<const uint4 *>(h);
            }
        }
        fence_async_smem();
        if (tid < kRows) s_bad[tid] = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    step_next();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<const uint32_t *>(ctl + SLOT), 0);

    // three meetings of a cluster: maxima, sums, sums read.  These warps have part in none, but count.
    if (C > 1 && warp >= kTmaWarp) cluster_arrive();
    auto count_on = [&]() {
        if (C > 1) cluster_wait(), cluster_sync();
    };
    auto meet = [&]() {
        __syncwarp();
        if (C > 1) cluster_sync();
        else bar_sync(1, 256);
    };
    auto at_rank = [&](uint32_t addr, int c) { return C > 1 ? cluster_addr(addr, c) : addr; };
    if (warp == kTmaWarp) {
        if (lane == 0) {
            for (int n = 0; n < 2 * NT; n++) {
                const int s = n & 1, j = n < NT ? n : n - NT;
                if (!mbar_wait_bounded(bars + K_FREE + 8 * s, ((n >> 1) & 1) ^ 1, dead)) break;
                mbar_expect_tx(bars + K_FULL + 8 * s, stage);
                for (int b = 0; b < blocks; b++) tma_load_2d(sk + s * stage + b * (kKeys * 128), &maps.k, g * D + 64 * b, kKeys * (rank + C * j), bars + K_FULL + 8 * s);
                if (n >= NT) {
                    const int v = j & 1;
                    if (!mbar_wait_bounded(bars + V_FREE + 8 * v, ((j >> 1) & 1) ^ 1, dead)) break;
                    mbar_expect_tx(bars + V_FULL + 8 * v, stage);
                    for (int b = 0; b < blocks; b++) tma_load_2d(sv + v * stage + b * (kKeys * 128), &maps.v, g * D + 64 * b, kKeys * (rank + C * j), bars + V_FULL + 8 * v);
                }
            }
        }
        __syncwarp();
        count_on();
    } else if (warp == kMmaWarp) {
        const uint32_t id_s = idesc_f16(kRows, kKeys, false), id_o = idesc_f16(kRows, D, true);
        const uint32_t q_lo = umma_desc_lo(base, 16), k_lo = umma_desc_lo(sk, 16), v_lo = umma_desc_lo(sv, kKeys * 128);
        auto scores = [&](int n) {
            const uint32_t s = n & 1, kl = k_lo + ((s * stage) >> 4);
            mbar_wait_bounded(bars + K_FULL + 8 * s, (n >> 1) & 1, dead);
            if (n >= 2) { // the buffer's last user: the maximum of tile n - 2, or the second product of tile n - 2 - NT
                if (n - 2 < NT) mbar_wait_bounded(bars + S_FREE + 8 * s, ((n - 2) >> 1) & 1, dead);
                else mbar_wait_bounded(bars + PV_DONE + 8 * s, ((n - 2 - NT) >> 1) & 1, dead);
            }
            tc_fence_after();
            for (int b = 0; b < blocks; b++)
#pragma unroll
                for (int k = 0; k < 4; k++) // 16 numbers are 2 descriptor units
                    umma_ss(tmem + s * kKeys, q_lo + b * (kRows * 8) + 2 * k, kl + b * (kKeys * 8) + 2 * k, id_s, b > 0 || k > 0);
            umma_arrive(bars + S_FULL + 8 * s);
            umma_arrive(bars + K_FREE + 8 * s);
        };
        for (int n = 0; n < NT; n++) scores(n);
        if (NT) scores(NT);
        for (int m = 0; m < NT; m++) {
            if (m + 1 < NT) scores(NT + m + 1);
            const uint32_t s = (NT + m) & 1, v = m & 1;
            mbar_wait_bounded(bars + P_FULL + 8 * s, (m >> 1) & 1, dead);
            mbar_wait_bounded(bars + V_FULL + 8 * v, (m >> 1) & 1, dead);
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < kKeys / 16; k++) // 16 keys: two groups of 8 rows of 128 bytes
                umma_ts(tmem + kOCol, tmem + s * kKeys + k * 8, v_lo + ((v * stage) >> 4) + k * 128, id_o, m > 0 || k > 0);
            umma_arrive(bars + V_FREE + 8 * v);
            umma_arrive(bars + PV_DONE + 8 * s);
        }
        umma_arrive(bars + DONE);
        count_on();
    } else {
        const int grp = warp >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t lanes = (uint32_t)(warp & 3) << 21; // 32 lanes of tensor memory a warp
        const uint32_t s_addr = tmem + lanes + grp * kKeys;
        const int i_row = a.pos0 + t0 + min(row, n_rows - 1) / hpg;
        float m = -INFINITY;
        for (int n = grp; n < NT; n += 2) {
            mbar_wait_warp(bars + S_FULL + 8 * grp, (n >> 1) & 1, dead);
            tc_fence_after();
            const int last = i_row - kKeys * (rank + C * n); // the row's last key of this tile
#pragma unroll
            for (int c0 = 0; c0 < kKeys; c0 += 32) {
                uint32_t v[32];
                tmem_load32(s_addr + c0, v);
#pragma unroll
                for (int c = 0; c < 32; c++) m = fmaxf(m, c0 + c <= last ? __uint_as_float(v[c]) : -INFINITY);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + S_FREE + 8 * grp);
        }
        s_max[grp * kRows + row] = m;
        meet();
        float parts[2 * C];
#pragma unroll
        for (int c = 0; c < C; c++) {
            const uint32_t there = at_rank(smem_u32(s_max + row), c);
            parts[2 * c] = ld_cluster_f32(there), parts[2 * c + 1] = ld_cluster_f32(there + 4 * kRows);
        }
#pragma unroll
        for (int c = 0; c < 2 * C; c++) m = fmaxf(m, parts[c]);
        const float l2e = 1.4426950408889634f, m2 = m * l2e;
        double sum = 0.0;
        for (int n = NT + ((NT ^ grp) & 1); n < 2 * NT; n += 2) {
            mbar_wait_warp(bars + S_FULL + 8 * grp, (n >> 1) & 1, dead);
            tc_fence_after();
            const int last = i_row - kKeys * (rank + C * (n - NT));
#pragma unroll
            for (int c0 = 0; c0 < kKeys; c0 += 32) {
                uint32_t v[32], w[16];
                tmem_load32(s_addr + c0, v);
                float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    float e[2];
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e[u]) : "f"(fmaf(__uint_as_float(v[c + u]), l2e, -m2)));
                        e[u] = c0 + c + u <= last ? e[u] : 0.f;
                    }
                    const __half2 h = __floats2half2_rn(e[0], e[1]);
                    w[c >> 1] = *reinterpret_cast<const uint32_t *>(&h);
                    const float2 f = __half22float2(h);
                    part[c & 2] += f.x;
                    part[(c & 2) + 1] += f.y;
                }
                sum += (double)((part[0] + part[1]) + (part[2] + part[3]));
                tmem_store16(s_addr + (c0 >> 1), w); // half 0's weights lie over scores 0..15, read before; half 1's over 16..31
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + P_FULL + 8 * grp);
        }
        s_sum[grp * kRows + row] = sum;
        mbar_wait_warp(bars + DONE, 0, dead);
        tc_fence_after();
        bar_sync(1, 256);
        if constexpr (C == 1) {
            sum = s_sum[row] + s_sum[kRows + row];
            const float inv = (float)(1.0 / sum);
            const int tq = row / hpg, half = D / 2;
            const int64_t at = ((int64_t)(t0 + tq) * a.H + g * hpg + (row - tq * hpg)) * D + grp * half;
            // rows of bf16 in shared memory (the tiles are no longer read), from there whole lines: the o-projection's A operand, rounded exactly as
            // ggb_op_cvt_f32_bf16 would
            bool finite = isfinite((float)sum);
            const uint32_t pitch = 2 * D + 16;
            for (int c0 = 0; c0 < half; c0 += 32) {
                uint32_t v[32];
                tmem_load32(tmem + lanes + kOCol + grp * half + c0, v);
                float o[32];
#pragma unroll
                for (int c = 0; c < 32; c++) {
                    o[c] = __uint_as_float(v[c]) * inv;
                    finite = finite && isfinite(o[c]);
                }
                if (row < n_rows && a.out) {
#pragma unroll
                    for (int c = 0; c < 32; c++) a.out[at + c0 + c] = o[c];
                }
#pragma unroll
                for (int c = 0; c < 32; c += 8)
                    *reinterpret_cast<uint4 *>(gbase + row * pitch + 2 * (grp * half + c0 + c)) =
                        make_uint4(pack_bf16x2(o[c], o[c + 1]), pack_bf16x2(o[c + 2], o[c + 3]), pack_bf16x2(o[c + 4], o[c + 5]), pack_bf16x2(o[c + 6], o[c + 7]));
            }
            if (!finite) s_bad[row] = 1;
            bar_sync(1, 256);
            if (a.out_bf16)
                for (int i = tid, pieces = D / 8; i < n_rows * pieces; i += 256) {
                    const int r = i / pieces, pc = i - r * pieces, q = r / hpg;
                    *reinterpret_cast<uint4 *>(a.out_bf16 + ((int64_t)(t0 + q) * a.H + g * hpg + (r - q * hpg)) * D + 8 * pc) = *reinterpret_cast<const uint4 *>(gbase + r * pitch + 16 * pc);
                }
        } else {
            // this CTA's sums, fp32, where the tiles were (they are no longer read): 16-byte piece p of row r at place p ^ (r & 7)
            const int half = D / 2, pieces = D / 4;
            for (int c0 = 0; c0 < half; c0 += 32) {
                uint32_t v[32];
                if (NT) tmem_load32(tmem + lanes + kOCol + grp * half + c0, v);
#pragma unroll
                for (int c = 0; c < 32; c += 4)
                    *reinterpret_cast<uint4 *>(gbase + (row * pieces + (((grp * half + c0 + c) >> 2) ^ (row & 7))) * 16) = NT ? make_uint4(v[c], v[c + 1], v[c + 2], v[c + 3]) : make_uint4(0, 0, 0, 0);
            }
            meet();
            // a share of the rows, from all CTAs of the cluster
            constexpr int R = kRows / C, U = 8 / C; // rows, pieces of them a thread has in flight (D is a multiple of 64: R * pieces of 256 U)
            const int r0 = rank * R;
            if (tid < R) {
                double part[2 * C], sum = 0.0;
#pragma unroll
                for (int c = 0; c < C; c++) {
                    const uint32_t there = at_rank(smem_u32(s_sum + r0 + tid), c);
                    part[2 * c] = ld_cluster_f64(there), part[2 * c + 1] = ld_cluster_f64(there + 8 * kRows);
                }
#pragma unroll
                for (int c = 0; c < C; c++) sum += part[2 * c] + part[2 * c + 1];
                s_inv[r0 + tid] = (float)(1.0 / sum);
                if (!isfinite((float)sum)) s_bad[r0 + tid] = 1;
            }
            bar_sync(1, 256);
            for (int i0 = tid; i0 < R * pieces; i0 += 256 * U) {
                float4 x[U][C];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int i = i0 + 256 * u, r = r0 + i / pieces, p = i % pieces;
#pragma unroll
                    for (int c = 0; c < C; c++) x[u][c] = ld_cluster_f32x4(at_rank(base + (r * pieces + (p ^ (r & 7))) * 16, c));
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int i = i0 + 256 * u, r = r0 + i / pieces, p = i % pieces, tq = r / hpg;
                    float4 o = x[u][0];
#pragma unroll
                    for (int c = 1; c < C; c++) o.x += x[u][c].x, o.y += x[u][c].y, o.z += x[u][c].z, o.w += x[u][c].w;
                    const float inv = s_inv[r];
                    o.x *= inv, o.y *= inv, o.z *= inv, o.w *= inv;
                    if (r >= n_rows) continue;
                    if (!(isfinite(o.x) && isfinite(o.y) && isfinite(o.z) && isfinite(o.w))) s_bad[r] = 1;
                    const int64_t at = ((int64_t)(t0 + tq) * a.H + g * hpg + (r - tq * hpg)) * D + 4 * p;
                    if (a.out) a.out[at] = o.x, a.out[at + 1] = o.y, a.out[at + 2] = o.z, a.out[at + 3] = o.w;
                    if (a.out_bf16) *reinterpret_cast<uint2 *>(a.out_bf16 + at) = make_uint2(pack_bf16x2(o.x, o.y), pack_bf16x2(o.z, o.w)); // as ggb_op_cvt_f32_bf16 would
                }
            }
        }
    }
    __syncwarp();
    if (C > 1) cluster_sync(); // the others have read this CTA's sums
    else if (warp < 8) bar_sync(1, 256);
    if (warp < 8 && !*dead)
        for (int r = rank * (kRows / C); r < min((rank + 1) * (kRows / C), n_rows); r++)
            if (s_bad[r]) plain_row(a, t0 + r / hpg, g * hpg + r % hpg, reinterpret_cast<float *>(gbase), s_sum);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kMmaWarp) {
        settle(dead);
        tmem_free512(tmem);
    }
    if (tid == 0 && *dead) *a.failed = 1;
}

} // namespace

bool ggb_attn_prefill_fits(const float *q, const void *kcache, const void *vcache, int64_t T, int pos0, int H, int Hkv, int d, const float *out, const void *out_bf16) {
    const uintptr_t align = (uintptr_t)q | (uintptr_t)kcache | (uintptr_t)vcache | (uintptr_t)out_bf16;
    // few keys: a CTA of the older kernels has a token and four heads (or a warp a token and head), and there are many of them; one of these takes
    // 8 to 16 us however few keys its 128 rows see (8 heads of 256 over one: 64 tokens 12.5 against 16.6 us, 128 tokens 19.0 against 18.6, 16 tokens behind
    // 500 positions 57 against 29; 8 over 8: 33 tokens 11.4 against 12.5, 64 tokens 18.7 against 13.5)
    const int few = H / Hkv % 4 == 0 ? 128 : 48;
    return T >= 16 && pos0 >= 0 && pos0 + T >= few && d % 64 == 0 && d <= 256 && H / Hkv <= kRows && align % 16 == 0 && (size_t)(pos0 + T) * 4 <= tile_bytes(d);
}

int ggb_attn_prefill_tiles(const float *q, const void *kcache, const void *vcache, int64_t T, int pos0, int H, int Hkv, int d, float *out, void *out_bf16) {
    attn_maps maps;
    const int64_t n_kv = pos0 + T, ld = (int64_t)Hkv * d; // positions past the last one arrive as zeros
    int rc = ggb_tensor_map_bf16(&maps.k, kcache, n_kv, ld, ld, kKeys); // (16-bit numbers as they lie)
    if (!rc) rc = ggb_tensor_map_bf16(&maps.v, vcache, n_kv, ld, ld, kKeys);
    if (rc) return rc;
    const attn_args a{q, (const __half *)kcache, (const __half *)vcache, (int)T, pos0, H, Hkv, d, ggb_exp_table_dev(), out, (__nv_bfloat16 *)out_bf16, ggb_wait_error_flag()};
    const int TQ = kRows / (H / Hkv), tiles = (int)((T + TQ - 1) / TQ) * Hkv, n_tiles = (int)((n_kv + kKeys - 1) / kKeys);
    // CTAs that share the key tiles of 128 rows, and the adding up: up to 4 while there are SMs for them (8 heads of 256 over one: 512 tokens 25 us by
    // one, 22, 18; 128 tokens 17, 16, 16); 8 for many keys and so few rows that clusters of 8 find room at once (64 tokens behind 1000 positions: 43, 29,
    // 22, 19; 512 tokens, 256 CTAs: 48).  Heads of up to 128 over two tiles of keys: 7.5 us by one, 8.4, 8.7
    int C = 1;
    while (C < 4 && 2 * C * tiles <= ggb_sm_count() && n_tiles >= (d > 128 ? 2 : 3)) C *= 2;
    if (C == 4 && 8 * tiles <= 112 && n_tiles >= 8) C = 8;
    const size_t smem = C > 1 ? std::max(smem_bytes(d), kOneCtaSmem) : smem_bytes(d);
    auto kern = C == 8 ? attn_prefill_tile_kernel<8> : C == 4 ? attn_prefill_tile_kernel<4> : C == 2 ? attn_prefill_tile_kernel<2> : attn_prefill_tile_kernel<1>;
    if ((rc = ggb_allow_smem(kern, smem))) return rc;
    GGB_CUDA(ggb_launch_early(kern, ggb_cluster{1, 1, (unsigned)C}, dim3((unsigned)((T + TQ - 1) / TQ), (unsigned)Hkv, (unsigned)C), dim3(kThreads), smem, maps, a));
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}
