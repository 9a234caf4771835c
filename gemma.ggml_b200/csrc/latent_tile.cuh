// latent_tile.cuh — latent attention of a portion of tokens on the tensor cores (tcgen05), bf16 cache and matrices.
//
// Every head reads the same cache rows [c | kr], so the rows of a CTA are tokens x heads, 128 of them, scored against tiles of 256
// positions.  Queries and weights are fp32 numbers and stay so: each is the sum of three bf16 numbers (split3, tc.cuh), a product with a
// bf16 row three products of the tensor cores.
//
// latent_tile_kernel.  The queries of 128 rows are 128 x (R + Dr) x 3 bf16 numbers, 442 KB at R = 512: more than a CTA's shared memory,
// so per tile of positions they are read again in blocks of 64 coordinates (fp32, converted on the way into shared memory), each beside
// the same block of 256 cache rows: scores S [128][256] in tensor memory.  Then 64 positions at a time become weights in shared memory
// and multiply the same rows' latents, O [128][up to 256] in the other half of tensor memory: a latent wider than 256 is cut in two over
// CTAs that repeat the scores (a CTA that held all of O would have no room for scores).  Both kinds of steps use the same two buffers for
// the left and four for the right operand, two steps ahead, one warp issuing the MMAs.
//
// What bounds it: the MMAs (58 % of the tensor cores' cycles, a half of the scores repeated at R > 256), then the rounds in which the weights
// of a tile wait for its last scores.  1024 tokens x 16 heads at position 1024, R = 512, Dr = 64: 234 us, 239 TFLOP/s of the products asked
// for (3420 us on the fp32 CUDA cores, two tokens a CTA); from 9 tokens on: fewer are steps, which spread their positions over warps.
//
// Infinite numbers are not the sums of their parts: a row (of a CTA) or an output whose sums are not finite is computed once more by fp32
// multiply-adds over what it sees (plain_part, plain_out), as tile_attention.cuh does.
//
// latent_out_kernel.  out = W_uv (sum of the parts): 128 tokens of one head, the merged fp32 rows converted in blocks of 64 (244 -> 28 us
// for the 1024 tokens above, bound by reading the parts).
#pragma once

#include "dense.cuh"
#include "tc.cuh"

namespace latent_tile {

constexpr int kRows = 128, kKeys = 256, kSub = 64;
constexpr int kWarps = 8, kThreads = 32 * (kWarps + 1);
constexpr uint32_t kPart = kRows * 128;         // one bf16 part of a left operand: 128 rows of 64 numbers
constexpr uint32_t kLeft = 3 * kPart, kRight = kKeys * 128;
constexpr uint32_t kTiles = 2 * kLeft + 4 * kRight;
constexpr size_t kSmem = 1024 + kTiles + 256 + 3 * kRows * 4;
enum { FULL = 0, FREE = 16, S_FULL = 32, SLOT = 64, DEAD = 72 };

struct args {
    const float *qa; // [T][H][QK]
    const __nv_bfloat16 *cache;
    int64_t ldk;
    const int32_t *table;
    int B;
    const int32_t *pos0;
    int T, H, R, QK, Vp; // Vp: latent coordinates of a CTA's output
    int64_t window;
    float *part;
    int *wait_error;
};

// 128 rows x QK, R a multiple of 32 so that half a latent is whole MMA steps and 16-byte pieces.  From 9 tokens on; two CTAs' rows or fewer
// whose positions are not split (there are few of them then: a caller splits a hundred and more) are quicker on the CUDA cores: 16 tokens x
// 8 heads of 256 at position 0 14 us (25), 24 tokens x 4 heads of 128 at 50 20 us (22), 9 x 16 of 512 at 0 and 50 22 and 36 us (34, 34).
inline bool fits(int R, int Dr, int H, int64_t T, int n_split, const void *qa, const void *cache) {
    return T >= 9 && T < (1 << 24) && (n_split > 1 || T * H > 2 * kRows) && H <= kRows && R % 32 == 0 && R <= 512 && Dr % 16 == 0 && (uintptr_t)qa % 16 == 0 && (uintptr_t)cache % 16 == 0;
}

// 2048 groups of four numbers of a left operand's block: thread tid takes groups tid + 256 u, row = group / 16
template <bool LOG2E = false> // times log2 e
__device__ __forceinline__ void store_left(uint32_t dst, int tid, const float4 (&x)[8]) {
#pragma unroll
    for (int u = 0; u < 8; u++) {
        const int g = tid + 256 * u, r = g >> 4, d = 4 * (g & 15);
        uint32_t h[2], m[2], l[2];
        f32x2 v = pack2(x[u].x, x[u].y), w = pack2(x[u].z, x[u].w);
        if (LOG2E) v = mul2(v, pack2(kLog2e, kLog2e)), w = mul2(w, pack2(kLog2e, kLog2e));
        split3(v, h[0], m[0], l[0]);
        split3(w, h[1], m[1], l[1]);
        const uint32_t at = dst + r * 128 + (((d >> 3) ^ (r & 7)) << 4) + (d & 4) * 2;
        asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at), "r"(h[0]), "r"(h[1]) : "memory");
        asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at + kPart), "r"(m[0]), "r"(m[1]) : "memory");
        asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at + 2 * kPart), "r"(l[0]), "r"(l[1]) : "memory");
    }
}
// D += (l + m + h) B over up to four steps of 16; b_step: descriptor units from one step to the next
__device__ __forceinline__ void mma_block(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t b_step, uint32_t idesc, int steps, uint32_t acc) {
#pragma unroll
    for (int part = 2; part >= 0; part--) // the small parts first
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (k < steps) {
                umma_ss(d, a_lo + part * (kPart >> 4) + 2 * k, b_lo + k * b_step, idesc, acc);
                acc = 1;
            }
}

struct row_job {
    const float *q;
    const __nv_bfloat16 *cache;
    int64_t ld;
    const int32_t *table;
    int B;
    int64_t lo, i, jlo; // the row sees [lo, i]; tiles count from jlo
    int split, n_split, QK, v0, Vp;
};
// one row's part by one warp, a position a lane: weighted sums to out[Vp], maximum and denominator to m and l
__device__ __noinline__ void plain_part(const row_job &j, float *out, float &m, float &l) {
    const int lane = threadIdx.x & 31;
    float acc[8]; // Vp <= 256
    for (int r = 0; r < 8; r++) acc[r] = 0.f;
    m = -INFINITY, l = 0.f;
    for (int64_t j0 = j.jlo + (int64_t)kKeys * j.split; j0 <= j.i; j0 += (int64_t)kKeys * j.n_split)
        for (int n0 = 0; n0 < kKeys; n0 += 32) {
            const int64_t at = min(max(j0 + n0 + lane, j.lo), j.i);
            const bool vis = at == j0 + n0 + lane;
            const uint32_t seen = __ballot_sync(0xffffffffu, vis);
            if (!seen) continue;
            const int64_t row = ((int64_t)j.table[at / j.B] * j.B + at % j.B) * j.ld;
            float s = 0.f, p = 0.f;
            for (int d = 0; d < j.QK; d++) s = fmaf(to_f32(j.cache[row + d]), j.q[d], s);
            const float mx = fmaxf(m, warp_max_f32(vis ? s : -INFINITY)), corr = mx == -INFINITY ? 1.f : expf(m - mx);
            if (vis && s != -INFINITY) p = expf(s - mx);
            l = fmaf(l, corr, warp_sum_f32(p));
            for (int r = 0; r < 8; r++) acc[r] *= corr;
            m = mx;
            for (int u = 0; u < 32; u++) {
                if (!(seen >> u & 1)) continue;
                const float pu = __shfl_sync(0xffffffffu, p, u);
                const __nv_bfloat16 *v = j.cache + __shfl_sync(0xffffffffu, row, u) + j.v0;
                for (int r = 0; r < 8; r++)
                    if (lane + 32 * r < j.Vp) acc[r] = fmaf(pu, to_f32(v[lane + 32 * r]), acc[r]);
            }
        }
    for (int r = 0; r < 8; r++)
        if (lane + 32 * r < j.Vp) out[lane + 32 * r] = acc[r];
    __syncwarp();
}

__global__ void __launch_bounds__(kThreads, 1) latent_tile_kernel(const args a) {
    extern __shared__ uint8_t lt_raw[];
    const uint32_t raw0 = smem_u32(lt_raw), base = (raw0 + 1023u) & ~1023u;
    uint8_t *gbase = lt_raw + (base - raw0);
    const uint32_t left = base, right = base + 2 * kLeft, bars = base + kTiles;
    volatile int *dead = reinterpret_cast<volatile int *>(gbase + kTiles + DEAD);
    float *mxs = reinterpret_cast<float *>(gbase + kTiles + 256); // [group][128] maxima, at the end sums
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int TQ = kRows / a.H, n_split = gridDim.y, split = blockIdx.y, v0 = blockIdx.z * a.Vp;
    const int t0 = (int)(gridDim.x - 1 - blockIdx.x) * TQ; // the CTAs with the most positions first
    const int nq = min(TQ, a.T - t0), rows = nq * a.H;
    const int64_t i0 = (int64_t)*a.pos0 + t0, i_last = i0 + nq - 1;
    const int64_t jlo = a.window > 0 ? max((int64_t)0, i0 - a.window + 1) : 0;
    const int nc = (a.QK + 63) / 64; // blocks of 64 coordinates
    const int nt = (int)((i_last - jlo) / kKeys) + 1;
    const int n_mine = split < nt ? (nt - 1 - split) / n_split + 1 : 0; // tiles split, split + n_split, ...
    if (tid == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(bars + FULL + 8 * s, kWarps);
            mbar_init(bars + FREE + 8 * s, 1);
        }
        mbar_init(bars + S_FULL, 1);
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kWarps) tmem_alloc512(bars + SLOT);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<uint32_t *>(gbase + kTiles + SLOT), 0), t_o = tmem + 256;
    auto tile_first = [&](int k) { return jlo + (int64_t)kKeys * (split + k * n_split); };
    auto tile_subs = [&](int k) { return (int)(min(i_last - tile_first(k), (int64_t)kKeys - 1) / kSub) + 1; };

    if (warp == kWarps) {
        const uint32_t id_o = umma_idesc(128, a.Vp, true);
        const uint32_t l_lo = umma_desc_lo(left, 16), k_lo = umma_desc_lo(right, 16), v_lo = umma_desc_lo(right, kSub * 128);
        uint32_t b = 0; // step: left operand buffer b & 1, right one b & 3
        for (int k = 0; k < n_mine; k++) {
            const int subs = tile_subs(k);
            const uint32_t id_s = umma_idesc(128, kSub * subs);
            for (int c = 0; c < nc; c++, b++) {
                mbar_wait_bounded(bars + FULL + 8 * (b & 1), (b >> 1) & 1, dead);
                tc_fence_after();
                mma_block(tmem, l_lo + (b & 1) * (kLeft >> 4), k_lo + (b & 3) * (kRight >> 4), 2, id_s, min(4, (a.QK - 64 * c) / 16), c > 0);
                umma_arrive(bars + FREE + 8 * (b & 1));
            }
            umma_arrive(bars + S_FULL);
            for (int s = 0; s < subs; s++, b++) {
                mbar_wait_bounded(bars + FULL + 8 * (b & 1), (b >> 1) & 1, dead);
                tc_fence_after();
                mma_block(t_o, l_lo + (b & 1) * (kLeft >> 4), v_lo + (b & 3) * (kRight >> 4), 128, id_o, 4, k > 0 || s > 0);
                umma_arrive(bars + FREE + 8 * (b & 1));
            }
        }
    } else {
        const int r = 32 * (warp & 3) + lane, grp = warp >> 2;
        const int64_t i = i0 + r / a.H, lo = a.window > 0 ? i - a.window + 1 : 0;
        const bool live = r < rows;
        const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
        const float *q0 = a.qa + (int64_t)t0 * a.H * a.QK;
        float m = -INFINITY, m_true = -INFINITY, l = 0.f;
        uint32_t cur[8], nxt[8]; // cache rows of this thread's positions (tid / 8 + 32 u of the tile): this tile's, the next one's
        const int pc = tid & 7, pr = tid >> 3;
        auto look_up = [&](int k, uint32_t (&row)[8]) {
            if (k >= n_mine) return;
            const int64_t j0 = tile_first(k);
#pragma unroll
            for (int u = 0; u < 8; u++) { // a row past the last one repeats it (weight 0)
                const uint32_t j = (uint32_t)min(j0 + pr + 32 * u, i_last), pg = j / (uint32_t)a.B;
                row[u] = (uint32_t)a.table[pg] * (uint32_t)a.B + (j - pg * a.B);
            }
        };
        // the right operand of step x of a tile (blocks of coordinates, then blocks of positions) into buffer buf
        auto load_right = [&](int x, int subs, const uint32_t (&row)[8], uint32_t buf) {
            const uint32_t dst = right + buf * kRight + pr * 128 + ((pc ^ (pr & 7)) << 4);
            if (x < nc) {
                if (64 * x + 8 * pc < a.QK) {
#pragma unroll
                    for (int u = 0; u < 8; u++)
                        if (u < 2 * subs) cp_async16(dst + u * 32 * 128, a.cache + row[u] * (uint64_t)a.ldk + 64 * x + 8 * pc);
                }
            } else if (x < nc + subs) {
#pragma unroll
                for (int u = 0; u < 8; u++) { // two halves of 32 positions x four blocks of 64 coordinates
                    const int s = x - nc, ru = u & 1, blk = u >> 1;
                    uint32_t rw = row[ru];
#pragma unroll
                    for (int w = 1; w < 4; w++) rw = s == w ? row[2 * w + ru] : rw;
                    if (64 * blk + 8 * pc < a.Vp) cp_async16(dst + ru * 32 * 128 + blk * (kSub * 128), a.cache + rw * (uint64_t)a.ldk + v0 + 64 * blk + 8 * pc);
                }
            }
        };
        float4 x[8];
        auto load_q = [&](int c) {
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int g = tid + 256 * u, qr = g >> 4, d = 64 * c + 4 * (g & 15);
                x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (qr < rows && d < a.QK) x[u] = __ldg(reinterpret_cast<const float4 *>(q0 + (int64_t)qr * a.QK + d));
            }
        };
        uint32_t b = 0;
        auto hand_over = [&]() { // the left operand is written and the right one of this step has landed
            cp_async_wait<2>();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + FULL + 8 * (b & 1));
            b++;
        };
        auto wait_free = [&]() { // the step that used this left buffer (and the right one two steps ahead) is done
            if (b >= 2) mbar_wait_warp(bars + FREE + 8 * (b & 1), ((b >> 1) - 1) & 1, dead);
        };
        look_up(0, cur);
        if (n_mine > 0) {
            load_q(0);
            load_right(0, tile_subs(0), cur, 0);
            cp_async_commit();
            load_right(1, tile_subs(0), cur, 1);
            cp_async_commit();
        }
        for (int k = 0; k < n_mine; k++) {
            const int subs = tile_subs(k), steps = nc + subs, subs_n = k + 1 < n_mine ? tile_subs(k + 1) : 0;
            look_up(k + 1, nxt);
            // two steps ahead, into the next tile where this one ends
            auto load_ahead = [&](int step) {
                const int x2 = step + 2;
                if (x2 < steps) load_right(x2, subs, cur, (b + 2) & 3);
                else if (subs_n > 0) load_right(x2 - steps, subs_n, nxt, (b + 2) & 3);
                cp_async_commit();
            };
            for (int c = 0; c < nc; c++) {
                wait_free();
                load_ahead(c);
                store_left<true>(left + (b & 1) * kLeft, tid, x); // scores in powers of two
                load_q(c + 1 < nc ? c + 1 : 0);
                hand_over();
            }
            const int64_t j0 = tile_first(k);
            const int n_keys = (int)min(i_last - j0 + 1, (int64_t)kKeys);
            const bool whole = n_keys == kKeys && j0 + kKeys - 1 <= i0 && (a.window <= 0 || j0 >= i_last - a.window + 1);
            const int c_hi = live ? (int)max((int64_t)0, min((int64_t)n_keys, i - j0 + 1)) : 0, c_lo = (int)max((int64_t)0, min((int64_t)kKeys, lo - j0));
            mbar_wait_warp(bars + S_FULL, k & 1, dead);
            tc_fence_after();
            { // maximum of the tile: a group takes every other 64 positions
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
                for (int cc = 0; cc < 8; cc++) {
                    const int c0 = 128 * (cc >> 2) + 64 * grp + 16 * (cc & 3);
                    if (c0 >= kSub * subs) break;
                    float s[16];
                    tmem_load16(tmem + lanes + c0, reinterpret_cast<uint32_t *>(s));
                    if (!whole) {
#pragma unroll
                        for (int c = 0; c < 16; c++) s[c] = (c0 + c < c_hi && c0 + c >= c_lo) ? s[c] : -INFINITY;
                    }
#pragma unroll
                    for (int c = 0; c < 16; c++) mx4[c & 3] = fmaxf(mx4[c & 3], s[c]);
                }
                mxs[grp * kRows + r] = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                bar_sync(1, 32 * kWarps);
                const float mx = fmaxf(mxs[r], mxs[kRows + r]);
                bar_sync(1, 32 * kWarps);
                m_true = fmaxf(m_true, mx);
                float corr = 1.f;
                const bool grow = mx > m + 8.f * kLog2e || (m == -INFINITY && mx > -INFINITY); // a maximum is kept until a score exceeds it by 8 log2 e
                if (grow) {
                    corr = exp2f(m - mx);
                    m = mx;
                    l *= corr;
                }
                if (k > 0 && __any_sync(0xffffffffu, grow)) { // the scores came behind the products of the tile before
#pragma unroll 1
                    for (int c = 16 * grp; c < a.Vp; c += 32) {
                        uint32_t o[16];
                        tmem_load16(t_o + lanes + c, o);
#pragma unroll
                        for (int u = 0; u < 16; u++) o[u] = __float_as_uint(__uint_as_float(o[u]) * corr);
                        tmem_store16(t_o + lanes + c, o);
                    }
                    tmem_wait_st();
                }
            }
            const float mm = m == -INFINITY ? 0.f : m;
            for (int s = 0; s < subs; s++) {
                // weights of 64 positions, 32 a group: four 16-byte pieces of each part of the thread's row
                uint32_t ph[16], pm[16], pl[16];
                f32x2 sum[2] = {0, 0};
#pragma unroll
                for (int hf = 0; hf < 2; hf++) {
                    const int c0 = kSub * s + 32 * grp + 16 * hf;
                    float p[16];
                    tmem_load16(tmem + lanes + c0, reinterpret_cast<uint32_t *>(p));
                    if (!whole) {
#pragma unroll
                        for (int c = 0; c < 16; c++) p[c] = (c0 + c < c_hi && c0 + c >= c_lo) ? p[c] : -INFINITY;
                    }
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        const float2 t = unpack2(add2(pack2(p[2 * c], p[2 * c + 1]), pack2(-mm, -mm)));
                        const f32x2 w = pack2(ex2_approx(t.x), ex2_approx(t.y));
                        sum[c & 1] = add2(sum[c & 1], w);
                        split3(w, ph[8 * hf + c], pm[8 * hf + c], pl[8 * hf + c]);
                    }
                }
                const float2 s2 = unpack2(add2(sum[0], sum[1]));
                l += s2.x + s2.y;
                tc_fence_before(); // the last of these scores are read before the next tile's are written
                wait_free();
                load_ahead(nc + s);
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const uint32_t at = left + (b & 1) * kLeft + r * 128 + (((4 * grp + v) ^ (r & 7)) << 4);
                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(ph[4 * v]), "r"(ph[4 * v + 1]), "r"(ph[4 * v + 2]), "r"(ph[4 * v + 3]) : "memory");
                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + kPart), "r"(pm[4 * v]), "r"(pm[4 * v + 1]), "r"(pm[4 * v + 2]), "r"(pm[4 * v + 3]) : "memory");
                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + 2 * kPart), "r"(pl[4 * v]), "r"(pl[4 * v + 1]), "r"(pl[4 * v + 2]), "r"(pl[4 * v + 3]) : "memory");
                }
                hand_over();
            }
#pragma unroll
            for (int u = 0; u < 8; u++) cur[u] = nxt[u];
        }
        cp_async_wait<0>();
        // ---- the part: relative to the true maximum, rows through shared memory
        if (b > 0) {
            mbar_wait_warp(bars + FREE + 8 * ((b - 1) & 1), ((b - 1) >> 1) & 1, dead);
            tc_fence_after();
        }
        mxs[grp * kRows + r] = l;
        bar_sync(1, 32 * kWarps);
        m_true *= kLn2; // what other parts are compared with
        const float f = over_e(m, m_true), l_row = (mxs[r] + mxs[kRows + r]) * f;
        float odd = 0.f * l_row; // 0, or NaN when a sum of the row is not finite
        if (grp == 0) mxs[2 * kRows + r] = l_row - l_row == 0.f ? m_true : NAN; // what this row's sums are relative to, where that is known
        bar_sync(1, 32 * kWarps);
        float *of = reinterpret_cast<float *>(gbase);
        const int op = a.Vp + 1;
        for (int c = 16 * grp; c < a.Vp; c += 32) {
            uint32_t o[16];
            if (n_mine > 0) tmem_load16(t_o + lanes + c, o);
#pragma unroll
            for (int u = 0; u < 16; u++) {
                const float v = f == 0.f ? 0.f : __uint_as_float(o[u]) * f;
                of[r * op + c + u] = v;
                odd = fmaf(0.f, v, odd);
            }
        }
        mxs[grp * kRows + r] = odd;
        if (grp == 0 && live && blockIdx.z == 0) {
            float *o = a.part + (((int64_t)(t0 + r / a.H) * n_split + split) * a.H + r % a.H) * (a.R + 2);
            o[0] = m_true;
            o[1] = l_row;
        }
        bar_sync(1, 32 * kWarps);
        { // a warp's 16 rows: warp, warp + 8, ...; those whose sums are not finite once more, without the split
            const int er = warp + kWarps * (lane & 15);
            uint32_t again = __ballot_sync(0xffffffffu, mxs[er] + mxs[kRows + er] != 0.f) & 0xffffu;
            while (again) {
                const int p = warp + kWarps * (__ffs((int)again) - 1);
                again &= again - 1;
                if (p >= rows) continue;
                const int64_t pi = i0 + p / a.H;
                const row_job j{q0 + (int64_t)p * a.QK, a.cache, a.ldk, a.table, a.B, a.window > 0 ? max((int64_t)0, pi - a.window + 1) : 0, pi, jlo, split, n_split, a.QK, v0, a.Vp};
                float pm, pl;
                plain_part(j, of + p * op, pm, pl);
                const float known = mxs[2 * kRows + p];
                if (known == known) { // the other half of the latent stays relative to this maximum: so does this one
                    const float g = pm == -INFINITY ? 1.f : expf(pm - known);
                    for (int c = lane; c < a.Vp; c += 32) of[p * op + c] *= g;
                } else if (lane == 0 && blockIdx.z == 0) {
                    float *o = a.part + (((int64_t)(t0 + p / a.H) * n_split + split) * a.H + p % a.H) * (a.R + 2);
                    o[0] = pm;
                    o[1] = pl;
                }
                __syncwarp();
            }
        }
        for (int p = warp; p < rows; p += kWarps) {
            float *o = a.part + (((int64_t)(t0 + p / a.H) * n_split + split) * a.H + p % a.H) * (a.R + 2) + 2 + v0;
            for (int c = lane; c < a.Vp; c += 32) o[c] = of[p * op + c];
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == kWarps) {
        settle(dead);
        tc_fence_after();
        tmem_free512(tmem);
        if (lane == 0 && *dead) *a.wait_error = 1;
    }
}

// ---- out[t][h] = W_uv_h (the parts' sum): 128 tokens of a head, blocks of 64 latent coordinates
struct out_args {
    const float *part;
    int n_split;
    const float *sink;
    const __nv_bfloat16 *w_uv; // [H][Dv][R]
    int T, H, R, Dv;
    const float *gate;
    int64_t ldg;
    __nv_bfloat16 *out;
    int *wait_error;
};
constexpr uint32_t kOutW = 256 * 128; // a block of W_uv: up to 256 rows of 64 numbers
constexpr int kOutSplits = 16;        // parts a row's weights are kept for
constexpr size_t kOutSmem = 1024 + 2 * (kLeft + kOutW) + 256 + (size_t)kRows * kOutSplits * 4;
inline bool out_fits(int R, int Dv, int64_t T, int n_split, const void *part, const void *w_uv, const void *out) {
    return T >= 32 && T < (1 << 24) && R % 16 == 0 && Dv % 16 == 0 && Dv <= 256 && n_split <= kOutSplits && (uintptr_t)part % 8 == 0 && (uintptr_t)w_uv % 16 == 0 &&
           (uintptr_t)out % 4 == 0;
}

// one output by one thread: w_uv's row against the merged parts (p0, weights wsm, ps numbers from one part to the next)
__device__ __noinline__ float plain_out(const float *p0, const float *wsm, int ns, int64_t ps, const __nv_bfloat16 *w, int R) {
    float y = 0.f;
    for (int d = 0; d < R; d++) {
        float x = 0.f;
        for (int s = 0; s < ns; s++) x = fmaf(p0[s * ps + 2 + d], wsm[s], x);
        y = fmaf(to_f32(w[d]), x, y);
    }
    return y;
}

__global__ void __launch_bounds__(kThreads, 1) latent_out_kernel(const out_args a) {
    extern __shared__ uint8_t lt_raw[];
    const uint32_t raw0 = smem_u32(lt_raw), base = (raw0 + 1023u) & ~1023u;
    uint8_t *gbase = lt_raw + (base - raw0);
    constexpr uint32_t kStage = kLeft + kOutW, kCtl = 2 * kStage;
    const uint32_t bars = base + kCtl;
    volatile int *dead = reinterpret_cast<volatile int *>(gbase + kCtl + DEAD);
    float *wsm = reinterpret_cast<float *>(gbase + kCtl + 256); // [128][n_split] weight of a part
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int h = blockIdx.y, t0 = blockIdx.x * kRows, nq = min(kRows, a.T - t0), ns = a.n_split;
    const int64_t ps = (int64_t)a.H * (a.R + 2); // from one part of a token to the next
    const float *p0 = a.part + ((int64_t)t0 * ns * a.H + h) * (a.R + 2);
    const int nc = (a.R + 63) / 64;
    if (tid == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(bars + FULL + 8 * s, kWarps);
            mbar_init(bars + FREE + 8 * s, 1);
        }
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kWarps) tmem_alloc512(bars + SLOT);
    if (tid < kRows && tid < nq) { // maximum and denominator over the parts and the sink
        const float *p = p0 + (int64_t)tid * ns * ps;
        const float sk = a.sink ? a.sink[h] : -INFINITY;
        float M = sk, L = 0.f;
        for (int s = 0; s < ns; s++) M = fmaxf(M, p[s * ps]);
        for (int s = 0; s < ns; s++) L = fmaf(p[s * ps + 1], expf(p[s * ps] - M), L);
        if (a.sink) L += expf(sk - M);
        const float inv = 1.0f / L;
        for (int s = 0; s < ns; s++) wsm[tid * ns + s] = expf(p[s * ps] - M) * inv;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<uint32_t *>(gbase + kCtl + SLOT), 0);
    if (warp == kWarps) {
        const uint32_t idesc = umma_idesc(128, a.Dv), l_lo = umma_desc_lo(base, 16), w_lo = umma_desc_lo(base + kLeft, 16);
        for (int c = 0; c < nc; c++) {
            const uint32_t s = c & 1;
            mbar_wait_bounded(bars + FULL + 8 * s, (c >> 1) & 1, dead);
            tc_fence_after();
            mma_block(tmem, l_lo + s * (kStage >> 4), w_lo + s * (kStage >> 4), 2, idesc, min(4, (a.R - 64 * c) / 16), c > 0);
            umma_arrive(bars + FREE + 8 * s);
        }
    } else {
        const int pc = tid & 7, pr = tid >> 3;
        for (int c = 0; c < nc; c++) {
            const uint32_t s = c & 1;
            float4 x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int sp = 0; sp < ns; sp++) {
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int g = tid + 256 * u, r = g >> 4, d = 64 * c + 4 * (g & 15);
                    if (r < nq && d < a.R) { // rows of R + 2 numbers: 8-byte aligned
                        const float2 *src = reinterpret_cast<const float2 *>(p0 + ((int64_t)r * ns + sp) * ps + 2 + d);
                        const float2 y = __ldg(src), z = __ldg(src + 1);
                        const float w = wsm[r * ns + sp];
                        x[u].x = fmaf(y.x, w, x[u].x), x[u].y = fmaf(y.y, w, x[u].y), x[u].z = fmaf(z.x, w, x[u].z), x[u].w = fmaf(z.y, w, x[u].w);
                    }
                }
            }
            if (c >= 2) mbar_wait_warp(bars + FREE + 8 * s, ((c >> 1) - 1) & 1, dead);
            if (64 * c + 8 * pc < a.R)
                for (int v = pr; v < a.Dv; v += 32)
                    cp_async16(base + s * kStage + kLeft + v * 128 + ((pc ^ (v & 7)) << 4), a.w_uv + ((int64_t)h * a.Dv + v) * a.R + 64 * c + 8 * pc);
            cp_async_commit();
            store_left(base + s * kStage, tid, x);
            cp_async_wait<0>();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + FULL + 8 * s);
        }
        mbar_wait_warp(bars + FREE + 8 * ((nc - 1) & 1), ((nc - 1) >> 1) & 1, dead);
        tc_fence_after();
        const int r = 32 * (warp & 3) + lane, t = t0 + r;
        const float gsc = a.gate && r < nq ? 1.0f / (1.0f + expf(-a.gate[(int64_t)t * a.ldg + h])) : 1.0f;
        for (int c = 16 * (warp >> 2); c < a.Dv; c += 32) {
            uint32_t o[16];
            tmem_load16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + c, o);
            if (r < nq) {
#pragma unroll
                for (int u = 0; u < 16; u++)
                    if (!(fabsf(__uint_as_float(o[u])) < INFINITY))
                        o[u] = __float_as_uint(plain_out(p0 + (int64_t)r * ns * ps, wsm + r * ns, ns, ps, a.w_uv + ((int64_t)h * a.Dv + c + u) * a.R, a.R));
                uint32_t *dst = reinterpret_cast<uint32_t *>(a.out + ((int64_t)t * a.H + h) * a.Dv + c);
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    float y = __uint_as_float(o[2 * u]), z = __uint_as_float(o[2 * u + 1]);
                    if (a.gate) y *= gsc, z *= gsc;
                    dst[u] = pack_bf16x2(y, z);
                }
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == kWarps) {
        settle(dead);
        tc_fence_after();
        tmem_free512(tmem);
        if (lane == 0 && *dead) *a.wait_error = 1;
    }
}

} // namespace latent_tile
