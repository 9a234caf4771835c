// moe.cu — mixture of experts: the router (fp32 logits, the `top` largest, soft-max over the chosen ones only), the
// grouping of (token, slot) pairs by expert, the two grouped products (gemm.cu, gemm_any.cu, or dense.cu: linear_tile_kernel, GROUPED) and the
// weighted sum.  A token's result does not depend on which other tokens share the step: every slot is computed by
// itself in k order and the `top` slot outputs are added in slot order.
#include <cuda_bf16.h>

#include <algorithm>
#include <math.h>

#include "common.cuh"
#include "dense.cuh"
#include "gemm_any.cuh"
#include "tc.cuh"

namespace {

// one warp: w . h in fp32, the same order of sums wherever it is called from
template <typename E>
__device__ __forceinline__ float router_dot(const E *__restrict__ hr, const float *__restrict__ wr, int64_t W, int lane) {
    float s = 0.f;
    if (W % 4 == 0) {
        struct alignas(4 * sizeof(E)) quad { // four numbers in one load: rows of a multiple of four are aligned to it
            E v[4];
        };
#pragma unroll 8
        for (int64_t k = (int64_t)lane * 4; k < W; k += 128) {
            const float4 wv = *reinterpret_cast<const float4 *>(wr + k);
            const quad hv = *reinterpret_cast<const quad *>(hr + k);
            s = fmaf(wv.x, to_f32(hv.v[0]), s);
            s = fmaf(wv.y, to_f32(hv.v[1]), s);
            s = fmaf(wv.z, to_f32(hv.v[2]), s);
            s = fmaf(wv.w, to_f32(hv.v[3]), s);
        }
    } else {
        for (int64_t k = lane; k < W; k += 32) s = fmaf(wr[k], to_f32(hr[k]), s);
    }
    return warp_sum_f32(s);
}

// router logits: a warp per (token, expert), z[t][e] = w[e] . h[t] + b[e] in fp32
template <typename E>
__global__ void __launch_bounds__(256) moe_logits_kernel(const E *h, int64_t W, int64_t T, const float *w,
                                                         const float *b, int n_exp, float *z) {
    step_wait();
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= T * n_exp) return;
    const int64_t t = i / n_exp;
    const int e = (int)(i - t * n_exp);
    const float s = router_dot(h + t * W, w + (int64_t)e * W, W, lane);
    if (lane == 0) z[i] = s + (b ? b[e] : 0.f);
}

// one warp: `top` rounds of arg-max over a token's logits z (ties: the lower index; z is used up), soft-max over the chosen; sel: [top] scratch
__device__ __forceinline__ void select_top_warp(float *z, float *sel, int n_exp, int top, int64_t t, int lane, int32_t *idx, float *wt) {
    for (int k = 0; k < top; k++) {
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        for (int e = lane; e < n_exp; e += 32) {
            const float v = z[e];
            if (v > bv || (v == bv && e < bi)) { bv = v; bi = e; }
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, off);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
            if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0) {
            if (bi >= n_exp) bi = 0; // logits that are no numbers: any expert, but one that exists
            idx[t * top + k] = bi;
            sel[k] = bv;
            z[bi] = -INFINITY;
        }
        __syncwarp();
    }
    if (lane == 0) {
        float m = sel[0], sum = 0.f; // sel[0] is the largest
        for (int k = 0; k < top; k++) {
            sel[k] = expf(sel[k] - m);
            sum += sel[k];
        }
        for (int k = 0; k < top; k++) wt[t * top + k] = sel[k] / sum;
    }
}

// one warp per token
__global__ void __launch_bounds__(32) moe_select_kernel(const float *zg, int n_exp, int top, int32_t *idx,
                                                        float *wt) {
    step_wait();
    extern __shared__ float z[]; // [n_exp] logits, then [top] chosen values
    const int64_t t = blockIdx.x;
    const int lane = threadIdx.x;
    for (int e = lane; e < n_exp; e += 32) z[e] = zg[t * n_exp + e];
    __syncwarp();
    select_top_warp(z, z + n_exp, n_exp, top, t, lane, idx, wt);
}

// A portion of tokens: a warp computes 4 tokens x 4 experts, so that a row of the router is read once for four tokens and a token's row once
// for four experts (a warp per logit reads 268 MB through L2 for 1024 tokens x 32 experts of width 2048).  Every logit is the same
// sum in the same order as router_dot's, to the bit: a choice between experts does not depend on how many tokens share the call.
// Bound by instruction issue.
constexpr int kLogitExperts = 4;
template <typename E>
__global__ void __launch_bounds__(256) moe_logits_tile_kernel(const E *h, int64_t W, int64_t T, const float *w, const float *b, int n_exp, float *z) {
    step_wait();
    struct alignas(4 * sizeof(E)) quad {
        E v[4];
    };
    const int lane = threadIdx.x & 31, groups = (n_exp + kLogitExperts - 1) / kLogitExperts;
    const int64_t item = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5), t0 = item / groups * kLogitExperts;
    const int e0 = (int)(item % groups) * kLogitExperts;
    if (t0 >= T) return;
    const E *hr[kLogitExperts];
    const float *wr[kLogitExperts];
#pragma unroll
    for (int i = 0; i < kLogitExperts; i++) { // past the end: the last one again, not stored
        hr[i] = h + min(t0 + i, T - 1) * W;
        wr[i] = w + (int64_t)min(e0 + i, n_exp - 1) * W;
    }
    float s[kLogitExperts * kLogitExperts]; // [token][expert]
#pragma unroll
    for (int i = 0; i < kLogitExperts * kLogitExperts; i++) s[i] = 0.f;
#pragma unroll 2
    for (int64_t k = (int64_t)lane * 4; k < W; k += 128) {
        float hv[kLogitExperts][4];
        float4 wv[kLogitExperts];
#pragma unroll
        for (int i = 0; i < kLogitExperts; i++) {
            const quad q = *reinterpret_cast<const quad *>(hr[i] + k);
            wv[i] = *reinterpret_cast<const float4 *>(wr[i] + k);
#pragma unroll
            for (int c = 0; c < 4; c++) hv[i][c] = to_f32(q.v[c]);
        }
#pragma unroll
        for (int i = 0; i < kLogitExperts; i++)
#pragma unroll
            for (int j = 0; j < kLogitExperts; j++) {
                float &a = s[i * kLogitExperts + j];
                a = fmaf(wv[j].x, hv[i][0], a);
                a = fmaf(wv[j].y, hv[i][1], a);
                a = fmaf(wv[j].z, hv[i][2], a);
                a = fmaf(wv[j].w, hv[i][3], a);
            }
    }
    // sixteen sums at once, each by the additions of warp_sum_f32: a lane ends with sum lane / 2
#pragma unroll
    for (int n = 8, off = 16; n >= 1; n >>= 1, off >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < n; i++) s[i] = __fadd_rn(up ? s[n + i] : s[i], __shfl_xor_sync(0xffffffffu, up ? s[i] : s[n + i], off));
    }
    s[0] = __fadd_rn(s[0], __shfl_xor_sync(0xffffffffu, s[0], 1));
    const int i = lane >> 3, j = (lane >> 1) & 3;
    if (!(lane & 1) && t0 + i < T && e0 + j < n_exp) z[(t0 + i) * n_exp + e0 + j] = s[0] + (b ? b[e0 + j] : 0.f);
}

// The same of TT (4 or 8) tokens x 4 experts a warp, where there are no more CTAs than SMs; `wide` of a CTA's eight warps stand beside each other
// with the same tokens, whose rows come from L1 to all but one of them.  TOP: the experts are 32 at most, and a warp then chooses for each token of the CTA
// (idx and wt), which spares a launch.
// Bound by the issue of instructions (two multiply-adds in one) and by L2's latency, against which each lane brings its own numbers of the next kLogitAhead
// steps of 128 into shared memory: all that an SM has for one CTA.  1024 x 32 x 2048: 10.6 us with the choice (11.7 with two steps in registers; 11.0 with 4 x 4 tiles, single multiply-adds and
// another launch for the choice); 1024 x 16 x 1024: 5.5 (6.5).
constexpr int kLogitWarps = 8, kLogitAhead = 4;
template <typename E, int TT> constexpr size_t logit_smem() { return (size_t)kLogitAhead * 32 * kLogitWarps * (kLogitExperts * 16 + TT * 4 * sizeof(E)); }
template <typename E, int TT, bool TOP>
__global__ void __launch_bounds__(32 * kLogitWarps) moe_logits_cta_kernel(const E *h, int64_t W, int64_t T, const float *w, const float *b, int n_exp, int wide, float *z, int top,
                                                                           int32_t *idx, float *wt) {
    constexpr int NE = kLogitExperts, NS = TT * NE, AT = kLogitAhead; // sums of a warp; steps under way
    extern __shared__ uint8_t lg_raw[];
    __shared__ float zs[TOP ? NS * kLogitWarps : 1], sel[TOP ? NS * kLogitWarps : 1]; // [token][expert]
    step_wait();
    struct alignas(4 * sizeof(E)) quad {
        E v[4];
    };
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tokens = TT * (kLogitWarps / wide), tw = warp / wide * TT;
    const int64_t tc = (int64_t)blockIdx.x * tokens, t0 = tc + tw;
    const int e0 = ((int)blockIdx.y * wide + warp % wide) * NE;
    if (!TOP && (e0 >= n_exp || t0 >= T)) return;
    const E *hr = h + min(t0, T - 1) * W;
    const float *wr = w + (int64_t)min(e0, n_exp - 1) * W;
    uint32_t ho[TT], wo[NE]; // rows past the end: the last one again, not stored
#pragma unroll
    for (int i = 0; i < TT; i++) ho[i] = (uint32_t)((min(t0 + i, T - 1) - min(t0, T - 1)) * W);
#pragma unroll
    for (int j = 0; j < NE; j++) wo[j] = (uint32_t)((min(e0 + j, n_exp - 1) - min(e0, n_exp - 1)) * W);
    f32x2 s2[TT / 2 * NE]; // [two tokens][expert]
#pragma unroll
    for (int i = 0; i < TT / 2 * NE; i++) s2[i] = 0;
    // a lane's own numbers: [step][row][thread], w in pieces of 16 bytes, then h
    const uint32_t wb = smem_u32(lg_raw) + threadIdx.x * 16, hb = smem_u32(lg_raw) + AT * NE * blockDim.x * 16 + threadIdx.x * sizeof(quad);
    const uint32_t wp = blockDim.x * 16, hp = blockDim.x * sizeof(quad); // from one row to the next
    auto load = [&](int64_t k, int u) {
        if (k < W) {
#pragma unroll
            for (int i = 0; i < TT; i++)
                asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(hb + (u * TT + i) * hp), "l"(hr + k + ho[i]), "n"(sizeof(quad)) : "memory");
#pragma unroll
            for (int j = 0; j < NE; j++) cp_async16(wb + (u * NE + j) * wp, wr + k + wo[j]);
        }
        cp_async_commit();
    };
#pragma unroll
    for (int u = 0; u < AT - 1; u++) load(4 * lane + 128 * u, u);
    for (int64_t k0 = 4 * lane; k0 < W; k0 += 128 * AT)
#pragma unroll
        for (int u = 0; u < AT; u++) {
            const int64_t k = k0 + 128 * u;
            load(k + 128 * (AT - 1), (u + AT - 1) % AT);
            if (k >= W) continue;
            cp_async_wait<AT - 1>();
            quad hq[TT];
            float4 wq[NE];
#pragma unroll
            for (int i = 0; i < TT; i++) hq[i] = *reinterpret_cast<const quad *>(lg_raw + (hb - smem_u32(lg_raw)) + (u * TT + i) * hp);
#pragma unroll
            for (int j = 0; j < NE; j++) wq[j] = *reinterpret_cast<const float4 *>(lg_raw + (wb - smem_u32(lg_raw)) + (u * NE + j) * wp);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                f32x2 w2[NE];
#pragma unroll
                for (int j = 0; j < NE; j++) {
                    const float x = c == 0 ? wq[j].x : c == 1 ? wq[j].y : c == 2 ? wq[j].z : wq[j].w;
                    w2[j] = pack2(x, x);
                }
#pragma unroll
                for (int i = 0; i < TT / 2; i++) {
                    const f32x2 h2 = pack2(to_f32(hq[2 * i].v[c]), to_f32(hq[2 * i + 1].v[c]));
#pragma unroll
                    for (int j = 0; j < NE; j++) s2[i * NE + j] = fma2(w2[j], h2, s2[i * NE + j]);
                }
            }
        }
    cp_async_wait<0>();
    __syncwarp();
    // all sums at once, each by the additions of warp_sum_f32: a lane ends with sum lane (of 32) or lane / 2 (of 16)
    float s[NS]; // [token][expert]
#pragma unroll
    for (int i = 0; i < TT / 2; i++)
#pragma unroll
        for (int j = 0; j < NE; j++) {
            const float2 v = unpack2(s2[i * NE + j]);
            s[2 * i * NE + j] = v.x, s[(2 * i + 1) * NE + j] = v.y;
        }
#pragma unroll
    for (int n = NS / 2, off = 16; n >= 1; n >>= 1, off >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < n; i++) s[i] = __fadd_rn(up ? s[n + i] : s[i], __shfl_xor_sync(0xffffffffu, up ? s[i] : s[n + i], off));
    }
    if (NS == 16) s[0] = __fadd_rn(s[0], __shfl_xor_sync(0xffffffffu, s[0], 1));
    const int own = NS == 16 ? lane >> 1 : lane, i = own / NE, j = own % NE;
    if ((NS == 32 || !(lane & 1)) && e0 + j < n_exp) {
        const float v = s[0] + (b ? b[e0 + j] : 0.f);
        if (t0 + i < T) z[(t0 + i) * n_exp + e0 + j] = v;
        if (TOP) zs[(tw + i) * wide * NE + e0 + j] = v;
    }
    if (TOP) {
        __syncthreads();
        for (int t = warp; t < tokens && tc + t < T; t += kLogitWarps) select_top_warp(zs + t * wide * NE, sel + t * wide * NE, n_exp, top, tc + t, lane, idx, wt);
    }
}

// The form by the number of logits: below a warp for every scheduler of the chip, tiles would leave SMs idle.  Tiles by CTAs that share rows only while there are no
// more of them than SMs (more: 4096 x 32 x 2048 27.0 us by warps, 38.6; 1536 x 20 10.9, 20.3; 1024 x 128 25.7, 39.0), without idle warps (20, 33 or 40 experts; 1024 x 33 x 2048
// 11.1, 19.1) and with four warps beside each other at least (4096 x 4 11.4, 15.8), of long rows if the choice takes another launch (128 x 128 x 256 4.9, 5.2; x 2048 9.7, 9.5; 256 x 64 10.3, 9.6).
// Eight tokens a warp only of bf16 rows (1024 x 32 x 2048 10.9, 10.5; fp32 11.8, 12.4), with the choice (256 x 128 10.7, 12.9).  chosen: idx and wt have been computed too
template <typename E>
int logits_launch(const E *h, int64_t W, int64_t T, const float *w, const float *b, int n_exp, float *z, int top = 0, int32_t *idx = nullptr, float *wt = nullptr,
                  bool *chosen = nullptr) {
    const int64_t groups = (n_exp + kLogitExperts - 1) / kLogitExperts, tiles = (T + 3) / 4 * groups;
    if (W % 4 == 0 && tiles >= 4 * ggb_sm_count()) {
        const int wide = (int)std::min<int64_t>(groups, kLogitWarps), rows = kLogitWarps / wide; // warps beside each other; where they are four or eight
        const unsigned ey = (unsigned)((groups + wide - 1) / wide);
        const bool fits = (groups == 4 || groups % 8 == 0) && W < (1 << 28), fused = chosen && ey == 1;
        auto ctas = [&](int tokens) { return (T + tokens * rows - 1) / (tokens * rows); };
        int rc = GGB_OK;
#define TILE(TT, TOP)                                                                                                                              \
    if ((rc = ggb_allow_smem(moe_logits_cta_kernel<E, TT, TOP>, logit_smem<E, TT>()))) return rc;                                                \
    ggb_launch_step(moe_logits_cta_kernel<E, TT, TOP>, dim3((unsigned)ctas(TT), ey), dim3(32 * kLogitWarps), logit_smem<E, TT>(), h, W, T, w, b, n_exp, wide, z, top, idx, wt)
        if (fits && ctas(4) * ey <= ggb_sm_count() && (fused || W >= 512)) {
            if (chosen) *chosen = fused;
            if (fused) { TILE(4, true); } else { TILE(4, false); }
        } else if (sizeof(E) == 2 && fits && fused && groups == 8 && ctas(8) <= ggb_sm_count()) {
            *chosen = true;
            if constexpr (sizeof(E) == 2) { TILE(8, true); }
        } else ggb_launch_step(moe_logits_tile_kernel<E>, dim3((unsigned)((tiles + 7) / 8)), dim3(256), 0, h, W, T, w, b, n_exp, z);
#undef TILE
    } else ggb_launch_step(moe_logits_kernel<E>, dim3((unsigned)((T * n_exp + 7) / 8)), dim3(256), 0, h, W, T, w, b, n_exp, z);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

// one warp: the choice scores of every group but the `keep` best ones (larger score, then lower index) become -inf
__device__ __forceinline__ void drop_groups_warp(float *ch, const float *gsc, int gs, int n_groups, int keep, int lane) {
    for (int g = lane; g < n_groups; g += 32) {
        int before = 0;
        for (int o = 0; o < n_groups; o++) before += (gsc[o] > gsc[g]) || (gsc[o] == gsc[g] && o < g);
        if (before >= keep)
            for (int e = g * gs; e < (g + 1) * gs; e++) ch[e] = -INFINITY;
    }
    __syncwarp();
}

// one warp per token, sigmoid scores with a choice correction and groups: s = sigmoid(z); the choice score of expert e is
// s_e + corr_e; the experts form n_groups equal groups of neighbours, a group's score is the sum of its two largest
// choice scores, and only experts of the `keep` best groups (ties: the lower group) can be chosen; among them the `top`
// largest choice scores win (ties: the lower index).  The weight of a chosen expert is its plain s, not renormalised.
// one warp; sc holds the logits on entry (the scores afterwards), ch and gsc are scratch
__device__ __forceinline__ void select_sigmoid_warp(float *sc, float *ch, float *gsc, const float *__restrict__ corr, int n_exp, int top, int n_groups,
                                                    int keep, int64_t t, int lane, int32_t *__restrict__ idx, float *__restrict__ wt) {
    const int gs = n_exp / n_groups;
    for (int e = lane; e < n_exp; e += 32) {
        const float s = 1.0f / (1.0f + expf(-sc[e]));
        sc[e] = s;
        ch[e] = s + (corr ? corr[e] : 0.f);
    }
    __syncwarp();
    if (keep < n_groups) {
        for (int g = lane; g < n_groups; g += 32) { // the two largest of the group, in index order
            float a = -INFINITY, b = -INFINITY;
            for (int e = g * gs; e < (g + 1) * gs; e++) {
                const float v = ch[e];
                if (v > a) { b = a; a = v; }
                else if (v > b) b = v;
            }
            gsc[g] = gs > 1 ? a + b : a;
        }
        __syncwarp();
        drop_groups_warp(ch, gsc, gs, n_groups, keep, lane);
    }
    for (int k = 0; k < top; k++) {
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        for (int e = lane; e < n_exp; e += 32) {
            const float v = ch[e];
            if (!isnan(sc[e]) && sc[e] >= 0.f && (v > bv || (v == bv && e < bi))) { bv = v; bi = e; }
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, off);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
            if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0) {
            if (bi >= n_exp) bi = 0; // logits that are no numbers: any expert, but one that exists
            idx[t * top + k] = bi;
            wt[t * top + k] = sc[bi];
            sc[bi] = -1.0f; // taken: a score is never negative otherwise
        }
        __syncwarp();
    }
}

// one warp per token, soft-max scores over ALL experts with a choice correction and groups: s = softmax(z); the choice score
// of expert e is s_e + corr_e; the experts form n_groups equal groups of neighbours, a group's score is its largest choice
// score and only experts of the `keep` best groups (ties: the lower group) can be chosen; the `top` largest win (ties: the
// lower index); the weight of a chosen expert is its s divided by the chosen ones' sum (+ 1e-20), times scale.  sc holds the
// logits on entry (the scores afterwards), ch and gsc are scratch.
__device__ __forceinline__ void select_softmax_warp(float *sc, float *ch, float *gsc, const float *__restrict__ corr, int n_exp, int top, int n_groups,
                                                    int keep, float scale, int64_t t, int lane, int32_t *__restrict__ idx, float *__restrict__ wt) {
    float m = -INFINITY;
    for (int e = lane; e < n_exp; e += 32) m = fmaxf(m, sc[e]);
    m = warp_max_f32(m);
    float sum = 0.f;
    for (int e = lane; e < n_exp; e += 32) {
        const float p = expf(sc[e] - m);
        sc[e] = p;
        sum += p;
    }
    sum = warp_sum_f32(sum);
    for (int e = lane; e < n_exp; e += 32) {
        const float p = sc[e] / sum;
        sc[e] = p;
        ch[e] = p + (corr ? corr[e] : 0.f);
    }
    __syncwarp();
    if (keep < n_groups) {
        const int gs = n_exp / n_groups;
        for (int g = lane; g < n_groups; g += 32) {
            float a = -INFINITY;
            for (int e = g * gs; e < (g + 1) * gs; e++) a = fmaxf(a, ch[e]);
            gsc[g] = a;
        }
        __syncwarp();
        drop_groups_warp(ch, gsc, gs, n_groups, keep, lane);
    }
    float chosen = 0.f; // lane 0: sum of the chosen scores, in slot order
    for (int k = 0; k < top; k++) {
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        for (int e = lane; e < n_exp; e += 32) {
            const float v = ch[e];
            if (sc[e] >= 0.f && (v > bv || (v == bv && e < bi))) { bv = v; bi = e; }
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, off);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
            if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0) {
            if (bi >= n_exp) bi = 0; // logits that are no numbers: any expert, but one that exists
            idx[t * top + k] = bi;
            wt[t * top + k] = sc[bi];
            chosen += sc[bi];
            sc[bi] = -1.0f; // taken: a score is never negative otherwise
        }
        __syncwarp();
    }
    if (lane == 0) {
        chosen += 1e-20f;
        for (int k = 0; k < top; k++) wt[t * top + k] = wt[t * top + k] / chosen * scale;
    }
}

__global__ void __launch_bounds__(32) moe_select_softmax_kernel(const float *zg, int64_t ldz, const float *corr, int n_exp, int top,
                                                                int n_groups, int keep, float scale, int32_t *idx, float *wt) {
    step_wait();
    extern __shared__ float sm[]; // [n_exp] scores, [n_exp] choice scores, [n_groups] group scores
    for (int e = threadIdx.x; e < n_exp; e += 32) sm[e] = zg[(int64_t)blockIdx.x * ldz + e];
    __syncwarp();
    select_softmax_warp(sm, sm + n_exp, sm + 2 * n_exp, corr, n_exp, top, n_groups, keep, scale, blockIdx.x, threadIdx.x, idx, wt);
}

__global__ void __launch_bounds__(32) moe_select_sigmoid_kernel(const float *zg, const float *corr, int n_exp, int top,
                                                                int n_groups, int keep, int32_t *idx, float *wt) {
    step_wait();
    extern __shared__ float sm[]; // [n_exp] scores, [n_exp] choice scores, [n_groups] group scores
    for (int e = threadIdx.x; e < n_exp; e += 32) sm[e] = zg[(int64_t)blockIdx.x * n_exp + e];
    __syncwarp();
    select_sigmoid_warp(sm, sm + n_exp, sm + 2 * n_exp, corr, n_exp, top, n_groups, keep, blockIdx.x, threadIdx.x, idx, wt);
}

// few tokens (a step): logits and choice in ONE launch.  CTA (token, y) computes the logits of experts 8 y .. 8 y + 7, a warp
// each, so that the router's rows are read by many SMs; the CTA that finishes last for its token (a counter per token, put
// back to zero by that CTA) reads all logits back and chooses.  With row_src the slots are also listed as the mat-vec form
// of the grouped products reads them (slot s = row s: no order is needed there), which stands in for moe_group_kernel.
// SOFTMAX: the rule of select_softmax_warp instead.  The matrix may have n_extra more rows behind the experts' (other numbers that
// read the same input, a gate for instance): their products are left in the logits behind the experts' and choose nothing.
constexpr int kRouteStepTokens = 32, kRouteStepWarps = 8;
__device__ unsigned int g_route_done[kRouteStepTokens];

template <typename E, bool SOFTMAX>
__global__ void __launch_bounds__(32 * kRouteStepWarps) moe_route_sigmoid_step_kernel(const E *h, int64_t W, const float *w,
                                                                     const float *corr, int n_exp, int n_extra, int top, int n_groups, int keep,
                                                                     float scale, float *zg, int32_t *idx, float *wt,
                                                                     int32_t *row_src, int32_t *inv,
                                                                     int32_t *row_expert) {
    step_wait();
    extern __shared__ float sm[];
    __shared__ bool last;
    const int64_t t = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e = (int)blockIdx.y * kRouteStepWarps + warp;
    const int64_t ldz = n_exp + n_extra;
    if (e < ldz) {
        const float s = router_dot(h + t * W, w + (int64_t)e * W, W, lane);
        if (lane == 0) {
            zg[t * ldz + e] = s;
            __threadfence(); // the logit is visible before this CTA is counted
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&g_route_done[t], 1u) == gridDim.y - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int i = threadIdx.x; i < n_exp; i += blockDim.x) sm[i] = __ldcg(zg + t * ldz + i); // other CTAs wrote them: not through L1
    if (threadIdx.x == 0) g_route_done[t] = 0; // the next launch starts from zero
    __syncthreads();
    if (warp != 0) return;
    if (SOFTMAX) select_softmax_warp(sm, sm + n_exp, sm + 2 * n_exp, corr, n_exp, top, n_groups, keep, scale, t, lane, idx, wt);
    else select_sigmoid_warp(sm, sm + n_exp, sm + 2 * n_exp, corr, n_exp, top, n_groups, keep, t, lane, idx, wt);
    __syncwarp();
    if (row_src)
        for (int k = lane; k < top; k += 32) {
            const int64_t s = t * top + k;
            row_src[s] = (int32_t)t;
            inv[s] = (int32_t)s;
            row_expert[s] = idx[s];
        }
}

// one CTA: counts per expert, offsets, the list of 64-row tiles, and the sorted order of the n = T * top slots
// experts n_real .. n_exp - 1 have no matrices (identity experts): their slots are sorted like the others but get no tile
// The count of a slot is its place among its expert's, kept in registers for the first kHeld slots of a thread; offsets and tiles are prefix
// sums of a thread an expert.  Bound by latency (one CTA).  4096 slots, 32 experts: 13.4 us with one thread walking the experts, 8.8 us.
constexpr int kGroupThreads = 1024, kHeld = 8;
__global__ void __launch_bounds__(kGroupThreads) moe_group_kernel(const int32_t *idx, int n, int top, int n_exp, int n_real, int32_t *offsets,
                                                                  int32_t *row_src, int32_t *inv, int32_t *tile_expert, int32_t *tile_row0,
                                                                  int32_t *n_tiles, int32_t *row_expert) {
    step_wait();
    extern __shared__ int32_t cnt[]; // [n_exp] counts, then first rows
    __shared__ int2 s_warp[kGroupThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, NT = blockDim.x;
    int e_of[kHeld], place[kHeld];
#pragma unroll
    for (int i = 0; i < kHeld; i++) {
        const int s = tid + i * NT;
        e_of[i] = s < n ? idx[s] : -1;
    }
    for (int e = tid; e < n_exp; e += NT) cnt[e] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kHeld; i++)
        if (e_of[i] >= 0) place[i] = atomicAdd(&cnt[e_of[i]], 1);
    __syncthreads(); // the held slots have the first places
    for (int s = tid + kHeld * NT; s < n; s += NT) atomicAdd(&cnt[idx[s]], 1);
    __syncthreads();
    int2 before = make_int2(0, 0); // rows and tiles of the experts of earlier rounds
    for (int e0 = 0; e0 < n_exp; e0 += NT) {
        const int e = e0 + tid, c = e < n_exp ? cnt[e] : 0, tiles = e < n_real ? (c + 63) / 64 : 0;
        int2 sum = make_int2(c, tiles);
#pragma unroll
        for (int off = 1; off < 32; off *= 2) {
            const int x = __shfl_up_sync(0xffffffffu, sum.x, off), y = __shfl_up_sync(0xffffffffu, sum.y, off);
            if (lane >= off) sum.x += x, sum.y += y;
        }
        if (lane == 31) s_warp[warp] = sum;
        __syncthreads();
        int2 base = before;
        for (int w = 0; w < NT / 32; w++) {
            const int2 v = s_warp[w];
            if (w < warp) base.x += v.x, base.y += v.y;
            before.x += v.x, before.y += v.y;
        }
        if (e < n_exp) {
            const int off = base.x + sum.x - c, t0 = base.y + sum.y - tiles;
            offsets[e] = off;
            cnt[e] = off;
            for (int u = 0; u < tiles; u++) {
                tile_expert[t0 + u] = e;
                tile_row0[t0 + u] = off + 64 * u;
            }
        }
        __syncthreads();
    }
    if (tid == 0) {
        offsets[n_exp] = before.x;
        *n_tiles = before.y;
    }
    auto put = [&](int s, int e, int p) {
        row_src[p] = s / top;
        row_expert[p] = e;
        inv[s] = p;
    };
#pragma unroll
    for (int i = 0; i < kHeld; i++)
        if (e_of[i] >= 0) put(tid + i * NT, e_of[i], cnt[e_of[i]] + place[i]);
    if (n <= kHeld * NT) return;
    __syncthreads();
    // the held slots' places are taken
#pragma unroll
    for (int i = 0; i < kHeld; i++) atomicAdd(&cnt[e_of[i]], 1);
    __syncthreads();
    for (int s = tid + kHeld * NT; s < n; s += NT) put(s, idx[s], atomicAdd(&cnt[idx[s]], 1));
}

// few slots (decode): a warp per (sorted row, output) streams the expert's weight row with 16-byte loads
template <typename E, int ACT>
__global__ void __launch_bounds__(256) moe_vec_kernel(const E *w, int64_t N, int64_t K, const E *a, int64_t lda,
                                                      const int32_t *row_src, const int32_t *row_expert,
                                                      float *c, E *c_act, int64_t ldc, int vec, int n_real, float limit,
                                                      float alpha) {
    step_wait();
    constexpr int VE = 16 / (int)sizeof(E);
    const int lane = threadIdx.x & 31;
    const int64_t n = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int row = blockIdx.y;
    if (n >= N || row_expert[row] >= n_real) return; // an expert without matrices: nothing to compute
    // ACT 2: an expert's matrix holds N gate rows, then N up rows; output n is silu(gate_n) * up_n
    // (every other ACT: act_f32, one row per output)
    // ACT 3: the same rows; g = min(gate_n, limit), u = clamp(up_n, -limit, limit), output g * sigmoid(alpha g) * (u + 1)
    constexpr bool GATED = ACT == 2 || ACT == 3;
    const E *wr = w + ((int64_t)row_expert[row] * (GATED ? 2 * N : N) + n) * K;
    const E *wu = wr + N * K;
    const E *ar = a + (int64_t)(row_src ? row_src[row] : row) * lda;
    float acc = 0.f, up = 0.f;
    if (vec) {
#pragma unroll 4
        for (int64_t k = (int64_t)lane * VE; k < K; k += 32 * VE) {
            const uint4 wv = ldg_stream_u4(wr + k), av = *reinterpret_cast<const uint4 *>(ar + k);
            const E *we = reinterpret_cast<const E *>(&wv), *ae = reinterpret_cast<const E *>(&av);
#pragma unroll
            for (int u = 0; u < VE; u++) acc = fmaf(to_f32(we[u]), to_f32(ae[u]), acc);
            if (GATED) {
                const uint4 uv = ldg_stream_u4(wu + k);
                const E *ue = reinterpret_cast<const E *>(&uv);
#pragma unroll
                for (int u = 0; u < VE; u++) up = fmaf(to_f32(ue[u]), to_f32(ae[u]), up);
            }
        }
    } else {
        for (int64_t k = lane; k < K; k += 32) {
            acc = fmaf(to_f32(wr[k]), to_f32(ar[k]), acc);
            if (GATED) up = fmaf(to_f32(wu[k]), to_f32(ar[k]), up);
        }
    }
    acc = warp_sum_f32(acc);
    if (GATED) up = warp_sum_f32(up);
    if (lane == 0) {
        if (ACT == GGB_ACT_RELU2 || ACT == GGB_ACT_GELU_ERF) c_act[(int64_t)row * ldc + n] = from_f32<E>(act_f32(acc, ACT));
        else if (ACT == 2) c_act[(int64_t)row * ldc + n] = from_f32<E>(acc / (1.0f + expf(-acc)) * up);
        else if (ACT == 3) {
            const float g = fminf(acc, limit), u = fminf(fmaxf(up, -limit), limit);
            c_act[(int64_t)row * ldc + n] = from_f32<E>(g / (1.0f + expf(-alpha * g)) * (u + 1.0f));
        }
        else c[(int64_t)row * ldc + n] = acc;
    }
}

// few slots, an expert that every token uses beside the chosen ones: rows n_slots .. n_slots + T - 1 of the grid are the tokens'
// products with that expert's matrix, which has sizes of its own (one launch for both)
template <typename E> struct shared_product {
    const E *w, *a;
    int64_t N, K, lda, ldc;
    float *c;
    E *c_act;
    int vec;
};
template <typename E, int ACT>
__global__ void __launch_bounds__(256) moe_vec_shared_kernel(const E *w, int64_t N, int64_t K, const E *a, int64_t lda,
                                                             const int32_t *row_src, const int32_t *row_expert,
                                                             float *c, E *c_act, int64_t ldc, int vec, int n_slots,
                                                             shared_product<E> sh) {
    step_wait();
    constexpr int VE = 16 / (int)sizeof(E);
    const int lane = threadIdx.x & 31;
    const int64_t n = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int row = blockIdx.y, t = row - n_slots;
    const E *wr, *ar;
    if (t < 0) {
        if (n >= N) return;
        wr = w + ((int64_t)row_expert[row] * N + n) * K;
        ar = a + (int64_t)(row_src ? row_src[row] : row) * lda;
    } else {
        if (n >= sh.N) return;
        wr = sh.w + n * sh.K;
        ar = sh.a + t * sh.lda;
        K = sh.K, vec = sh.vec;
    }
    float acc = 0.f;
    if (vec) {
#pragma unroll 4
        for (int64_t k = (int64_t)lane * VE; k < K; k += 32 * VE) {
            const uint4 wv = ldg_stream_u4(wr + k), av = *reinterpret_cast<const uint4 *>(ar + k);
            const E *we = reinterpret_cast<const E *>(&wv), *ae = reinterpret_cast<const E *>(&av);
#pragma unroll
            for (int u = 0; u < VE; u++) acc = fmaf(to_f32(we[u]), to_f32(ae[u]), acc);
        }
    } else {
        for (int64_t k = lane; k < K; k += 32) acc = fmaf(to_f32(wr[k]), to_f32(ar[k]), acc);
    }
    acc = warp_sum_f32(acc);
    if (lane != 0) return;
    const int64_t at = t < 0 ? row * ldc + n : t * sh.ldc + n;
    if (ACT) (t < 0 ? c_act : sh.c_act)[at] = from_f32<E>(act_f32(acc, ACT));
    else (t < 0 ? c : sh.c)[at] = acc;
}

// rows of A in sorted-slot order (the tensor-core product reads its operand contiguously): y[i] = a[row_src[i]], a warp a row, 16 bytes a lane, eight of
// them under way
__global__ void __launch_bounds__(256) moe_gather_kernel(const uint4 *a, int64_t row_u4, const int32_t *row_src, int64_t n, uint4 *y) {
    step_wait();
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= n) return;
    const uint4 *src = a + (int64_t)row_src[row] * row_u4;
    uint4 *dst = y + row * row_u4;
    for (int64_t i = threadIdx.x & 31; i < row_u4; i += 256) {
        uint4 v[8];
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (i + 32 * u < row_u4) v[u] = src[i + 32 * u];
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (i + 32 * u < row_u4) dst[i + 32 * u] = v[u];
    }
}

// VEC: four numbers a thread, the slots' rows in flight together (W a multiple of four, rows on 16 bytes).  Bound by memory: 1024 x 4 rows
// of 2048 11.8 us number by number, 8.5 us.
template <bool VEC>
__global__ void moe_combine_kernel(const float *y, const int32_t *inv, const float *wt, int top,
                                   int64_t W, float *out) {
    step_wait();
    const int64_t t = blockIdx.x;
    if constexpr (VEC) {
        for (int64_t i = (int64_t)threadIdx.x * 4; i < W; i += (int64_t)blockDim.x * 4) {
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int k = 0; k < top; k++) {
                const float w = wt[t * top + k];
                const float4 v = *reinterpret_cast<const float4 *>(y + (int64_t)inv[t * top + k] * W + i);
                s.x = fmaf(w, v.x, s.x);
                s.y = fmaf(w, v.y, s.y);
                s.z = fmaf(w, v.z, s.z);
                s.w = fmaf(w, v.w, s.w);
            }
            *reinterpret_cast<float4 *>(out + t * W + i) = s;
        }
    } else {
        for (int64_t i = threadIdx.x; i < W; i += blockDim.x) {
            float s = 0.f;
            for (int k = 0; k < top; k++) s = fmaf(wt[t * top + k], y[(int64_t)inv[t * top + k] * W + i], s);
            out[t * W + i] = s;
        }
    }
}

// the same with experts that hand their input through: a slot whose expert is n_real or later adds wt * h[t]
template <typename E>
__global__ void moe_combine_identity_kernel(const float *y, const int32_t *inv, const float *wt,
                                            const int32_t *idx, int top, int n_real, int64_t W, const E *h,
                                            float *out) {
    step_wait();
    const int64_t t = blockIdx.x;
    for (int64_t i = threadIdx.x; i < W; i += blockDim.x) {
        float s = 0.f;
        for (int k = 0; k < top; k++) {
            const float v = idx[t * top + k] < n_real ? y[(int64_t)inv[t * top + k] * W + i] : to_f32(h[t * W + i]);
            s = fmaf(wt[t * top + k], v, s);
        }
        out[t * W + i] = s;
    }
}

} // namespace

extern "C" {

#define GGB_CHECK_DT(dt) GGB_CHECK_ARG((dt) == GGB_TYPE_BF16 || (dt) == GGB_TYPE_F32, "dtype %d is neither bf16 nor f32", (int)(dt))

int ggb_op_moe_route(int dt, const void *h, int64_t W, int64_t T, const float *w_router, const float *bias, int n_exp, int top,
                     float *logits, int32_t *idx, float *wt) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_DT(dt);
    GGB_CHECK_ARG(h && w_router && idx && wt && W > 0 && T > 0 && n_exp > 0 && top > 0 && top <= n_exp && n_exp <= 8192,
                  "moe_route: bad arguments");
    GGB_CHECK_ARG(logits != nullptr, "moe_route: needs T * n_exp floats for the logits");
    const size_t smem = (size_t)(n_exp + top) * 4;
    bool chosen = false;
    const int rc = dt == GGB_TYPE_BF16 ? logits_launch((const __nv_bfloat16 *)h, W, T, w_router, bias, n_exp, logits, top, idx, wt, &chosen)
                                       : logits_launch((const float *)h, W, T, w_router, bias, n_exp, logits, top, idx, wt, &chosen);
    if (rc || chosen) return rc;
    ggb_launch_step(moe_select_kernel, dim3((unsigned)T), dim3(32), smem, logits, n_exp, top, idx, wt);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_moe_step_form(int64_t n_slots) { return n_slots <= 16; }

int ggb_op_moe_route_sigmoid(int dt, const void *h, int64_t W, int64_t T, const float *w_router, const float *correction, int n_exp, int top,
                             int n_groups, int keep, float *logits, int32_t *idx, float *wt, int32_t *ws) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_DT(dt);
    GGB_CHECK_ARG(h && w_router && idx && wt && logits && W > 0 && T > 0 && n_exp > 0 && top > 0 && n_exp <= 4096, "moe_route_sigmoid: bad arguments");
    GGB_CHECK_ARG(n_groups > 0 && n_exp % n_groups == 0 && keep > 0 && keep <= n_groups && top <= keep * (n_exp / n_groups),
                  "moe_route_sigmoid: %d experts in %d groups of which %d stay cannot give %d experts", n_exp, n_groups, keep, top);
    const size_t smem = (size_t)(2 * n_exp + n_groups) * 4;
    if (T <= 32) { // a step: one launch, and the slot lists of the mat-vec form with it
        const int64_t n = T * top;
        const int mt = ggb_moe_max_tiles(n, n_exp);
        const bool lists = ws && ggb_moe_step_form(n);
        int32_t *row_src = lists ? ws + n_exp + 1 : nullptr, *inv = lists ? row_src + n : nullptr, *row_expert = lists ? inv + n + 2 * mt + 1 : nullptr;
        if (dt == GGB_TYPE_BF16)
            ggb_launch_step(moe_route_sigmoid_step_kernel<__nv_bfloat16, false>, dim3((unsigned)T, (unsigned)((n_exp + kRouteStepWarps - 1) / kRouteStepWarps)), dim3(32 * kRouteStepWarps), smem, (const __nv_bfloat16 *)h, W, w_router, correction, n_exp, 0, top, n_groups,
                                                                                         keep, 1.f, logits, idx, wt, row_src, inv, row_expert);
        else
            ggb_launch_step(moe_route_sigmoid_step_kernel<float, false>, dim3((unsigned)T, (unsigned)((n_exp + kRouteStepWarps - 1) / kRouteStepWarps)), dim3(32 * kRouteStepWarps), smem, (const float *)h, W, w_router, correction, n_exp, 0, top, n_groups, keep, 1.f,
                                                                                         logits, idx, wt, row_src, inv, row_expert);
        GGB_LAUNCH_CHECK();
        return GGB_OK;
    }
    const int rc = dt == GGB_TYPE_BF16 ? logits_launch((const __nv_bfloat16 *)h, W, T, w_router, nullptr, n_exp, logits)
                                       : logits_launch((const float *)h, W, T, w_router, nullptr, n_exp, logits);
    if (rc) return rc;
    ggb_launch_step(moe_select_sigmoid_kernel, dim3((unsigned)T), dim3(32), smem, logits, correction, n_exp, top, n_groups,
                                                                                                         keep, idx, wt);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_op_moe_route_softmax(int dt, const void *h, int64_t W, int64_t T, const float *w_router, const float *correction, int n_exp, int top,
                             float *logits, int32_t *idx, float *wt, int32_t *ws) {
    return ggb_op_moe_route_softmax_groups(dt, h, W, T, w_router, correction, n_exp, 0, top, 1, 1, 1.f, logits, idx, wt, ws);
}

int ggb_op_moe_route_softmax_groups(int dt, const void *h, int64_t W, int64_t T, const float *w_router, const float *correction, int n_exp, int n_extra,
                                    int top, int n_groups, int keep, float scale, float *logits, int32_t *idx, float *wt, int32_t *ws) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_DT(dt);
    GGB_CHECK_ARG(h && w_router && idx && wt && logits && W > 0 && T > 0 && n_exp > 0 && n_extra >= 0 && top > 0 && top <= n_exp && n_exp <= 4096,
                  "moe_route_softmax: bad arguments (%d of %d experts)", top, n_exp);
    GGB_CHECK_ARG(n_groups > 0 && n_exp % n_groups == 0 && keep > 0 && keep <= n_groups && top <= keep * (n_exp / n_groups),
                  "moe_route_softmax: %d experts in %d groups of which %d stay cannot give %d experts", n_exp, n_groups, keep, top);
    const size_t smem = (size_t)(2 * n_exp + n_groups) * 4;
    const int ldz = n_exp + n_extra;
    if (T <= kRouteStepTokens) { // a step: one launch, and the slot lists of the mat-vec form with it
        const int64_t n = T * top;
        const int mt = ggb_moe_max_tiles(n, n_exp);
        const bool lists = ws && ggb_moe_step_form(n);
        int32_t *row_src = lists ? ws + n_exp + 1 : nullptr, *inv = lists ? row_src + n : nullptr, *row_expert = lists ? inv + n + 2 * mt + 1 : nullptr;
        const dim3 grid((unsigned)T, (unsigned)((ldz + kRouteStepWarps - 1) / kRouteStepWarps));
        if (dt == GGB_TYPE_BF16)
            ggb_launch_step(moe_route_sigmoid_step_kernel<__nv_bfloat16, true>, grid, dim3(32 * kRouteStepWarps), smem,
                (const __nv_bfloat16 *)h, W, w_router, correction, n_exp, n_extra, top, n_groups, keep, scale, logits, idx, wt, row_src, inv, row_expert);
        else
            ggb_launch_step(moe_route_sigmoid_step_kernel<float, true>, grid, dim3(32 * kRouteStepWarps), smem,
                (const float *)h, W, w_router, correction, n_exp, n_extra, top, n_groups, keep, scale, logits, idx, wt, row_src, inv, row_expert);
        GGB_LAUNCH_CHECK();
        return GGB_OK;
    }
    const int rc = dt == GGB_TYPE_BF16 ? logits_launch((const __nv_bfloat16 *)h, W, T, w_router, nullptr, ldz, logits)
                                       : logits_launch((const float *)h, W, T, w_router, nullptr, ldz, logits);
    if (rc) return rc;
    ggb_launch_step(moe_select_softmax_kernel, dim3((unsigned)T), dim3(32), smem, logits, ldz, correction, n_exp, top, n_groups, keep, scale, idx, wt);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_moe_max_tiles(int64_t n_slots, int n_exp) { return (int)(n_slots / 64) + n_exp; }
size_t ggb_moe_group_ints(int64_t n_slots, int n_exp) {
    return (size_t)(n_exp + 1) + 3 * (size_t)n_slots + 2 * (size_t)ggb_moe_max_tiles(n_slots, n_exp) + 1;
}

static ggb_moe_groups groups_of(int32_t *ws, int64_t n, int n_exp, bool gather) {
    ggb_moe_groups g;
    const int mt = ggb_moe_max_tiles(n, n_exp);
    g.offsets = ws;
    g.row_src = gather ? ws + n_exp + 1 : nullptr;
    g.tile_expert = ws + n_exp + 1 + 2 * n;
    g.tile_row0 = g.tile_expert + mt;
    g.n_tiles = g.tile_row0 + mt;
    return g;
}

int ggb_op_moe_group(const int32_t *idx, int64_t T, int top, int n_exp, int32_t *ws) { return ggb_op_moe_group_identity(idx, T, top, n_exp, 0, ws); }

int ggb_op_moe_group_identity(const int32_t *idx, int64_t T, int top, int n_exp, int n_identity, int32_t *ws) {
    GGB_REQUIRE_INIT();
    const int64_t n = T * top;
    GGB_CHECK_ARG(idx && ws && T > 0 && top > 0 && n_exp > 0 && n_exp <= 8192 && n < (1ll << 30) && n_identity >= 0 && n_identity <= n_exp,
                  "moe_group: bad arguments");
    const int mt = ggb_moe_max_tiles(n, n_exp);
    int32_t *offsets = ws, *row_src = ws + n_exp + 1, *inv = row_src + n, *te = inv + n, *tr = te + mt, *nt = tr + mt, *re = nt + 1;
    int threads = 32; // a step's few slots take one warp, whose barriers cost nothing
    while (threads < kGroupThreads && (threads < n_exp || threads * kHeld < n)) threads *= 2;
    ggb_launch_step(moe_group_kernel, dim3(1), dim3(threads), (size_t)n_exp * 4, idx, (int)n, top, n_exp, n_exp - n_identity, offsets, row_src, inv, te, tr, nt, re);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_op_moe_linear(int dt, const void *w, int64_t N, int64_t K, const void *a, int64_t lda, int gather, int64_t T, int top, int n_exp,
                      const int32_t *ws, int act, void *c, int64_t ldc) {
    return ggb_op_moe_linear_identity(dt, w, N, K, a, lda, gather, T, top, n_exp, 0, ws, act, 0.f, 0.f, c, ldc);
}

int ggb_op_moe_linear_identity(int dt, const void *w, int64_t N, int64_t K, const void *a, int64_t lda, int gather, int64_t T, int top, int n_exp,
                               int n_identity, const int32_t *ws, int act, float limit, float alpha, void *c, int64_t ldc) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_DT(dt);
    GGB_CHECK_ARG(w && a && ws && c && N > 0 && K > 0 && T > 0 && lda >= K && ldc >= N && act >= 0 && act <= GGB_ACT_GELU_ERF && n_identity >= 0 &&
                      n_identity < n_exp,
                  "moe_linear: bad arguments");
    GGB_CHECK_ARG((act != 2 && act != 3) || ggb_moe_step_form(T * top), "moe_linear: the gated forms are built for steps of at most 16 slots");
    const int n_real = n_exp - n_identity;
    const ggb_moe_groups g = groups_of(const_cast<int32_t *>(ws), T * top, n_exp, gather != 0);
    if (ggb_moe_step_form(T * top)) { // decode: every slot is a mat-vec on its expert's matrix
        const int es = dt == GGB_TYPE_BF16 ? 2 : 4;
        const int vec = K % (16 / es) == 0 && lda % (16 / es) == 0 && ((uintptr_t)w | (uintptr_t)a) % 16 == 0;
        const int32_t *row_expert = g.n_tiles + 1;
        const dim3 grid((unsigned)((N + 7) / 8), (unsigned)(T * top));
#define MV(E)                                                                                                                         \
    if (act == GGB_ACT_GELU_ERF) ggb_launch_step(moe_vec_kernel<E, GGB_ACT_GELU_ERF>, grid, dim3(256), 0, (const E *)w, N, K, (const E *)a, lda, g.row_src, row_expert, nullptr, (E *)c, ldc, vec, n_real, 0.f, 0.f); \
    else if (act == 3) ggb_launch_step(moe_vec_kernel<E, 3>, grid, dim3(256), 0, (const E *)w, N, K, (const E *)a, lda, g.row_src, row_expert, nullptr, (E *)c, ldc, vec, n_real, limit, alpha); \
    else if (act == 2) ggb_launch_step(moe_vec_kernel<E, 2>, grid, dim3(256), 0, (const E *)w, N, K, (const E *)a, lda, g.row_src, row_expert, nullptr, (E *)c, ldc, vec, n_real, 0.f, 0.f); \
    else if (act) ggb_launch_step(moe_vec_kernel<E, 1>, grid, dim3(256), 0, (const E *)w, N, K, (const E *)a, lda, g.row_src, row_expert, nullptr, (E *)c, ldc, vec, n_real, 0.f, 0.f); \
    else ggb_launch_step(moe_vec_kernel<E, 0>, grid, dim3(256), 0, (const E *)w, N, K, (const E *)a, lda, g.row_src, row_expert, (float *)c, nullptr, ldc, vec, n_real, 0.f, 0.f);
        if (dt == GGB_TYPE_BF16) { MV(__nv_bfloat16) } else { MV(float) }
#undef MV
        GGB_LAUNCH_CHECK();
        return GGB_OK;
    }
    // Portions, bf16, aligned shapes, on the tensor cores: many slots in tiles of rows or of an expert's slots.  Fewer through the slot list without a
    // workspace (such a portion may be captured, and a workspace that grows would move under the graph), every 64 numbers of K summed by
    // themselves: no further off than the multiply-adds of the tile kernel, which takes what is left.  32 experts, 1408 x 2048: 480 slots 39 us
    // (47 gathered), 20 slots 24 (33).
    if (dt == GGB_TYPE_BF16 && ggb_gemm_grouped_bf16_fits(N, K, ldc) && lda == K && ((uintptr_t)a & 15) == 0) {
        const int64_t n = T * top;
        if (n >= 512) {
            const bool slots = ggb_gemm_grouped_bf16_slots(N, K, n, n_real, false, gather, act != 0);
            const void *a_sorted = a;
            const bool ahead = gather && !slots;
            if (ahead) {
                void *gbuf;
                const int rc = ggb_workspace(GGB_WS_MOE_GATHER, (size_t)n * (size_t)K * 2, &gbuf);
                if (rc) return rc;
                ggb_launch_step(moe_gather_kernel, dim3((unsigned)((n + 7) / 8)), dim3(256), 0, (const uint4 *)a, K / 8, g.row_src, n, (uint4 *)gbuf);
                GGB_LAUNCH_CHECK();
                a_sorted = gbuf;
            }
            return ggb_gemm_grouped_bf16(slots, w, N, K, a_sorted, n, n_real, g.offsets, ahead ? nullptr : g.row_src, act ? nullptr : (float *)c, act ? c : nullptr, act, ldc);
        }
        if (K >= 128 && ((uintptr_t)w & 15) == 0) // (sums of 64: 7e-8, multiply-adds 5e-8; K = 128: 7.0e-8, 7.2e-8)
            return ggb_gemm_any_grouped(w, N, K, a, lda, n, n_real, act ? nullptr : (float *)c, ldc, act ? c : nullptr, act, g);
    }
    return ggb_linear_grouped_launch(dt, w, N, K, a, lda, ggb_moe_max_tiles(T * top, n_exp), act ? nullptr : (float *)c, act ? c : nullptr,
                                     ldc, act, g);
}

int ggb_op_moe_linear_shared(int dt, const void *w, int64_t N, int64_t K, const void *a, int64_t lda, int gather, int64_t T, int top, int n_exp,
                             const int32_t *ws, int act, void *c, int64_t ldc, const void *w_s, int64_t N_s, int64_t K_s, const void *a_s, int64_t lda_s,
                             void *c_s) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_DT(dt);
    GGB_CHECK_ARG(w && a && ws && c && w_s && a_s && c_s && N > 0 && K > 0 && N_s > 0 && K_s > 0 && T > 0 && lda >= K && ldc >= N && lda_s >= K_s,
                  "moe_linear_shared: bad arguments");
    GGB_CHECK_ARG(act == GGB_ACT_NONE || act == GGB_ACT_GELU_ERF, "moe_linear_shared: activation %d", act);
    if (!ggb_moe_step_form(T * top)) { // portions: the grouped product, then the shared expert's
        const int rc = ggb_op_moe_linear(dt, w, N, K, a, lda, gather, T, top, n_exp, ws, act, c, ldc);
        if (rc) return rc;
        return act ? ggb_op_linear_act(dt, w_s, N_s, K_s, a_s, lda_s, T, act, c_s) : ggb_op_linear(dt, w_s, N_s, K_s, a_s, lda_s, T, (float *)c_s, N_s);
    }
    const ggb_moe_groups g = groups_of(const_cast<int32_t *>(ws), T * top, n_exp, gather != 0);
    const int32_t *row_expert = g.n_tiles + 1;
    const int ve = 16 / (dt == GGB_TYPE_BF16 ? 2 : 4);
    const int vec = K % ve == 0 && lda % ve == 0 && ((uintptr_t)w | (uintptr_t)a) % 16 == 0;
    const int vec_s = K_s % ve == 0 && lda_s % ve == 0 && ((uintptr_t)w_s | (uintptr_t)a_s) % 16 == 0;
    const dim3 grid((unsigned)((std::max(N, N_s) + 7) / 8), (unsigned)(T * top + T));
#define MVS(E, ACT)                                                                                                                             \
    ggb_launch_step(moe_vec_shared_kernel<E, ACT>, grid, dim3(256), 0, (const E *)w, N, K, (const E *)a, lda, g.row_src, row_expert,               \
                                                                       ACT ? nullptr : (float *)c, ACT ? (E *)c : nullptr, ldc, vec, (int)(T * top), \
                                                                       shared_product<E>{(const E *)w_s, (const E *)a_s, N_s, K_s, lda_s, N_s,      \
                                                                                         ACT ? nullptr : (float *)c_s, ACT ? (E *)c_s : nullptr, vec_s});
    if (dt == GGB_TYPE_BF16) {
        if (act) MVS(__nv_bfloat16, GGB_ACT_GELU_ERF) else MVS(__nv_bfloat16, GGB_ACT_NONE)
    } else {
        if (act) MVS(float, GGB_ACT_GELU_ERF) else MVS(float, GGB_ACT_NONE)
    }
#undef MVS
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_op_moe_combine_norm(int dt, const float *y, const int32_t *ws, const float *wt, int64_t T, int top, int n_exp, int64_t W, const float *wa,
                            float eps, float *x, const float *wy, void *out) {
    GGB_CHECK_ARG(y && ws && wt && top > 0 && n_exp > 0, "moe_combine_norm: bad arguments");
    return ggb_norm_add_norm_launch(dt, y, nullptr, ws + n_exp + 1 + T * top, wt, top, wa, eps, W, T, x, wy, out);
}

int ggb_op_moe_combine_identity(int dt, const float *y, const int32_t *ws, const float *wt, const int32_t *idx, int64_t T, int top, int n_exp,
                                int n_identity, int64_t W, const void *h, float *out) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_DT(dt);
    GGB_CHECK_ARG(y && ws && wt && idx && h && out && T > 0 && top > 0 && W > 0 && n_identity >= 0 && n_identity <= n_exp,
                  "moe_combine_identity: bad arguments");
    const int32_t *inv = ws + n_exp + 1 + T * top;
    if (dt == GGB_TYPE_BF16)
        ggb_launch_step(moe_combine_identity_kernel<__nv_bfloat16>, dim3((unsigned)T), dim3(256), 0, y, inv, wt, idx, top, n_exp - n_identity, W, (const __nv_bfloat16 *)h, out);
    else
        ggb_launch_step(moe_combine_identity_kernel<float>, dim3((unsigned)T), dim3(256), 0, y, inv, wt, idx, top, n_exp - n_identity, W, (const float *)h, out);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_op_moe_combine(const float *y, const int32_t *ws, const float *wt, int64_t T, int top, int n_exp, int64_t W, float *out) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(y && ws && wt && out && T > 0 && top > 0 && W > 0, "moe_combine: bad arguments");
    const int32_t *inv = ws + n_exp + 1 + T * top;
    const bool vec = W % 4 == 0 && ((uintptr_t)y | (uintptr_t)out) % 16 == 0;
    if (vec) ggb_launch_step(moe_combine_kernel<true>, dim3((unsigned)T), dim3(256), 0, y, inv, wt, top, W, out);
    else ggb_launch_step(moe_combine_kernel<false>, dim3((unsigned)T), dim3(256), 0, y, inv, wt, top, W, out);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

} // extern "C"
