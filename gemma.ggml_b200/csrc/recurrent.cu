// recurrent.cu — mixers whose memory is a fixed-size state instead of a row per position: the causal convolution over
// time with a carried tail, lightning attention (a decayed sum of outer products) and the gated delta rule.  All state
// is fp32 and lives in the caller's per-sequence block; a portion of T tokens continues from the state the previous
// portion left and leaves its own, so a prompt may be cut anywhere.
//
// The two recurrences share one kernel: a CTA owns one head and a slice of CV (16 or 32) value columns (columns are independent
// in both rules), NS lanes share a column and each keeps D / NS numbers of it in registers for the whole portion.
// Per token the lanes' partial sums meet through two shuffles.  Tokens are staged through shared memory in chunks by
// four more warps, one chunk ahead of the recurrence; the staging pass also does what is per token and parallel:
// activations, unit norms, decay and step size.  That is the form of steps; portions take eight tokens at a time (recurrence_chunk_kernel).
//
// Compiled with -fmad=false: multiply-adds are spelled fmaf().
#include <algorithm>

#include "common.cuh"
#include "dense.cuh"
#include "tc.cuh"

namespace {

// __frcp_rn: the correctly rounded reciprocal, one instruction sequence without the slow path of the precise division
__device__ __forceinline__ float silu_f32(float z) { return z * __frcp_rn(1.0f + expf(-z)); }
__device__ __forceinline__ float sigmoid_f32(float z) { return __frcp_rn(1.0f + expf(-z)); }
__device__ __forceinline__ float softplus_f32(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

// ------------------------------------------------------------------------------------------------ causal convolution
constexpr int kConvMaxTaps = 8, kConvTokens = 32;

// grid (channel blocks, token chunks); a thread owns one channel of one chunk and slides a window of taps inputs along
// it.  Chunk 0 is the only reader of the old tail and its only writer (after it has the old values in registers).
template <typename E>
__global__ void __launch_bounds__(128) causal_conv_kernel(const float *__restrict__ x, int64_t ldx, int64_t T, int64_t C,
                                                          const float *__restrict__ w, const float *__restrict__ bias, int taps, int add_input,
                                                          int act, float *tail, float *__restrict__ y_f32, int64_t ldy, E *__restrict__ y_dt) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const float xb = bias ? bias[c] : 0.f; // the input is x + bias; the tail keeps it so
    const int64_t t0 = (int64_t)blockIdx.y * kConvTokens, t1 = min(T, t0 + kConvTokens);
    const int nt = taps - 1;
    float wt[kConvMaxTaps], win[kConvMaxTaps], old[kConvMaxTaps];
#pragma unroll
    for (int j = 0; j < kConvMaxTaps; j++) {
        wt[j] = j < taps ? w[c * taps + j] : 0.f;
        win[j] = 0.f;
        old[j] = 0.f;
    }
    if (blockIdx.y == 0)
#pragma unroll
        for (int j = 0; j < kConvMaxTaps - 1; j++)
            if (j < nt) old[j] = tail[(int64_t)j * C + c];
    // win[j], j < taps - 1: the inputs at t0 - (taps - 1) + j
#pragma unroll
    for (int j = 0; j < kConvMaxTaps - 1; j++)
        if (j < nt) {
            const int64_t s = t0 - nt + j;
            win[j] = s >= 0 ? x[s * ldx + c] + xb : old[j]; // s < 0 only in chunk 0, where s + nt = j indexes the old tail
        }
    for (int64_t t = t0; t < t1; t++) {
        const float xv = x[t * ldx + c] + xb;
        float acc = 0.f;
#pragma unroll
        for (int j = 0; j < kConvMaxTaps - 1; j++)
            if (j < nt) acc = fmaf(wt[j], win[j], acc);
        acc = fmaf(wt[nt], xv, acc);
        if (add_input) acc += xv;
        if (act) acc = silu_f32(acc);
        if (y_f32) y_f32[t * ldy + c] = acc;
        if (y_dt) y_dt[t * C + c] = from_f32<E>(acc);
#pragma unroll
        for (int j = 0; j < kConvMaxTaps - 2; j++)
            if (j + 1 < nt) win[j] = win[j + 1];
        if (nt > 0) {
#pragma unroll
            for (int j = 0; j < kConvMaxTaps - 1; j++)
                if (j == nt - 1) win[j] = xv;
        }
    }
    if (blockIdx.y == 0) { // new tail: the last taps - 1 inputs of (old tail, x)
#pragma unroll
        for (int j = 0; j < kConvMaxTaps - 1; j++)
            if (j < nt) {
                const int64_t s = T - nt + j;
                float v = 0.f;
                if (s >= 0) v = x[s * ldx + c] + xb;
                else {
#pragma unroll
                    for (int i = 0; i < kConvMaxTaps - 1; i++)
                        if (i == (int)(s + nt)) v = old[i];
                }
                tail[(int64_t)j * C + c] = v;
            }
    }
}

// ------------------------------------------------------------------------------------------------ the recurrences
constexpr int kNS = 4;      // lanes that share a column of S
constexpr int kStageWarps = 4; // warps that stage the next chunk
constexpr int kChunk = 16;  // tokens staged at once

struct rec_args {
    const float *q, *k, *v, *b, *a;
    int64_t ld, ld_b, ld_a, T;
    int H, G, D, Dv;
    const float *decay, *A_log, *dt_bias;
    float *state, *o;
    int64_t ldo;
    int decays; // MODE 2: `a` holds the decays themselves, not the raw rows they are computed from
};

// MODE 0: lightning (q, k, v = silu of the raw rows; S <- decay S + k v^T; o = S^T q)
// MODE 1: gated delta rule (unit q and k, q * D^-1/2; S <- g S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q)
// MODE 2: the same rule with one decay per head and key channel: row d of S is multiplied by g[d]; the decays of a
//         token are staged like a q / k row
//
// CV * 4 threads run the recurrence on the chunk in one buffer while four more warps stage the next chunk into
// the other (global loads of a warp's four tokens in flight together), one barrier per chunk.
// A lane's slice of a q / k row starts DS + 4 words after its neighbour's: the four 16-byte reads of a warp fall into
// four different groups of banks (DS alone is a multiple of 8 words: all four would meet in one).
template <int DS, int CV, bool CH = false>
struct rec_smem {
    static constexpr int DP = DS * kNS;        // padded D
    static constexpr int DW = (DS + 4) * kNS;  // words of a staged row
    __device__ static __forceinline__ int at(int d) { return (d / DS) * (DS + 4) + d % DS; }
    float q[kChunk][DW], k[kChunk][DW];
    float v[kChunk][CV], g[kChunk], beta[kChunk];
    float gc[kChunk][CH ? DW : 1]; // per-channel decays
};

template <int DS, int CV, int MODE>
__device__ __forceinline__ void rec_stage(const rec_args &p, rec_smem<DS, CV, MODE == 2> &b, int64_t t0, int n, int h, int hk, int col0, int pw, int lane, float a_rate,
                                          float dtb, float q_scale) {
    constexpr int DP = DS * kNS, PL = (DP + 31) / 32, TPW = kChunk / kStageWarps; // numbers per lane and row, tokens per producer warp
    float qv[TPW][PL], kv[TPW][PL], vv[TPW], bb[TPW], aa[TPW];
    float av[MODE == 2 ? TPW : 1][MODE == 2 ? PL : 1];
#pragma unroll
    for (int u = 0; u < TPW; u++) {
        const int tt = pw + kStageWarps * u;
        const int64_t t = t0 + min(tt, n - 1); // past the chunk's end: the last token again, not stored
        const float *qr = p.q + t * p.ld + (int64_t)hk * p.D, *kr = p.k + t * p.ld + (int64_t)hk * p.D;
#pragma unroll
        for (int i = 0; i < PL; i++) {
            const int d = lane + 32 * i;
            qv[u][i] = d < p.D ? qr[d] : 0.f;
            kv[u][i] = d < p.D ? kr[d] : 0.f;
        }
        vv[u] = (lane < CV && col0 + lane < p.Dv) ? p.v[t * p.ld + (int64_t)h * p.Dv + col0 + lane] : 0.f;
        if (MODE == 1) {
            bb[u] = p.b[t * p.ld_b + h];
            aa[u] = p.a[t * p.ld_a + h];
        }
        if (MODE == 2) {
            bb[u] = p.b[t * p.ld_b + h];
            const float *ar = p.a + t * p.ld_a + (int64_t)h * p.D;
#pragma unroll
            for (int i = 0; i < PL; i++) {
                const int d = lane + 32 * i;
                av[u][i] = d < p.D ? ar[d] : 0.f;
            }
        }
    }
#pragma unroll
    for (int u = 0; u < TPW; u++) {
        const int tt = pw + kStageWarps * u;
        if (tt >= n) continue;
        float qm = 1.f, km = 1.f;
        if (MODE == 0) {
#pragma unroll
            for (int i = 0; i < PL; i++) {
                qv[u][i] = silu_f32(qv[u][i]); // silu(0) = 0: the padding stays zero
                kv[u][i] = silu_f32(kv[u][i]);
            }
            vv[u] = silu_f32(vv[u]);
        } else {
            float qs = 0.f, ks = 0.f;
#pragma unroll
            for (int i = 0; i < PL; i++) {
                qs = fmaf(qv[u][i], qv[u][i], qs);
                ks = fmaf(kv[u][i], kv[u][i], ks);
            }
            qs = warp_sum_f32(qs);
            ks = warp_sum_f32(ks);
            qm = q_scale / sqrtf(qs + 1e-6f);
            km = 1.0f / sqrtf(ks + 1e-6f);
            if (lane == 0) {
                b.beta[tt] = sigmoid_f32(bb[u]);
                if (MODE == 1) b.g[tt] = expf(-a_rate * softplus_f32(aa[u] + dtb));
            }
            if (MODE == 2) {
#pragma unroll
                for (int i = 0; i < PL; i++) {
                    const int d = lane + 32 * i;
                    if (d < DP) // rows of the padding hold zeros and stay zero
                        b.gc[tt][rec_smem<DS, CV, true>::at(d)] =
                            d >= p.D ? 1.f : p.decays ? av[u][i] : expf(-a_rate * softplus_f32(av[u][i] + p.dt_bias[(int64_t)h * p.D + d]));
                }
            }
        }
#pragma unroll
        for (int i = 0; i < PL; i++) {
            const int d = lane + 32 * i;
            if (d < DP) {
                b.q[tt][rec_smem<DS, CV, MODE == 2>::at(d)] = qv[u][i] * qm;
                b.k[tt][rec_smem<DS, CV, MODE == 2>::at(d)] = kv[u][i] * km;
            }
        }
        if (lane < CV) b.v[tt][lane] = vv[u];
    }
}

template <int DS, int CV, int MODE>
__global__ void __launch_bounds__(CV *kNS + 32 * kStageWarps) recurrence_kernel(rec_args p) {
    extern __shared__ __align__(16) unsigned char rec_raw[];
    typedef rec_smem<DS, CV, MODE == 2> smem_t;
    smem_t *buf = reinterpret_cast<smem_t *>(rec_raw);
    const int h = blockIdx.x, col0 = blockIdx.y * CV;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool producer = warp >= (CV * kNS) / 32;
    const int s = tid % kNS, cl = (tid / kNS) % CV, col = col0 + cl;
    const bool live = !producer && col < p.Dv;
    const int hk = MODE != 0 ? h / (p.H / p.G) : h; // the q / k head this head reads
    float S[DS];
    float *sp = p.state + ((int64_t)h * p.D) * p.Dv + col;
#pragma unroll
    for (int i = 0; i < DS; i++) {
        const int d = s * DS + i;
        S[i] = (live && d < p.D) ? sp[(int64_t)d * p.Dv] : 0.f;
    }
    const float decay = MODE == 0 ? p.decay[h] : 0.f;
    const float a_rate = MODE == 1 || (MODE == 2 && !p.decays) ? expf(p.A_log[h]) : 0.f, dtb = MODE == 1 ? p.dt_bias[h] : 0.f;
    const float q_scale = 1.0f / sqrtf((float)p.D);
    const int pw = warp - (CV * kNS) / 32;
    if (producer) rec_stage<DS, CV, MODE>(p, buf[0], 0, (int)min((int64_t)kChunk, p.T), h, hk, col0, pw, lane, a_rate, dtb, q_scale);
    __syncthreads();
    int cur = 0;
    for (int64_t t0 = 0; t0 < p.T; t0 += kChunk, cur ^= 1) {
        const int n = (int)min((int64_t)kChunk, p.T - t0);
        if (producer) {
            if (t0 + kChunk < p.T)
                rec_stage<DS, CV, MODE>(p, buf[cur ^ 1], t0 + kChunk, (int)min((int64_t)kChunk, p.T - t0 - kChunk), h, hk, col0, pw, lane, a_rate, dtb, q_scale);
        } else {
            const smem_t &b = buf[cur];
            for (int tt = 0; tt < n; tt++) {
                const float4 *k4 = reinterpret_cast<const float4 *>(&b.k[tt][s * (DS + 4)]);
                const float4 *q4 = reinterpret_cast<const float4 *>(&b.q[tt][s * (DS + 4)]);
                float o0 = 0.f, o1 = 0.f;
                if (MODE == 0) {
                    const float vj = b.v[tt][cl];
#pragma unroll
                    for (int i = 0; i < DS / 4; i++) {
                        const float4 kk = k4[i], qq = q4[i];
                        S[4 * i + 0] = fmaf(kk.x, vj, decay * S[4 * i + 0]);
                        S[4 * i + 1] = fmaf(kk.y, vj, decay * S[4 * i + 1]);
                        S[4 * i + 2] = fmaf(kk.z, vj, decay * S[4 * i + 2]);
                        S[4 * i + 3] = fmaf(kk.w, vj, decay * S[4 * i + 3]);
                        o0 = fmaf(S[4 * i + 0], qq.x, o0);
                        o1 = fmaf(S[4 * i + 1], qq.y, o1);
                        o0 = fmaf(S[4 * i + 2], qq.z, o0);
                        o1 = fmaf(S[4 * i + 3], qq.w, o1);
                    }
                } else {
                    const float g = MODE == 1 ? b.g[tt] : 1.f;
                    const float4 *g4 = reinterpret_cast<const float4 *>(&b.gc[MODE == 2 ? tt : 0][MODE == 2 ? s * (DS + 4) : 0]);
                    float r0 = 0.f, r1 = 0.f;
#pragma unroll
                    for (int i = 0; i < DS / 4; i++) {
                        const float4 kk = k4[i];
                        const float4 gg = MODE == 2 ? g4[i] : make_float4(g, g, g, g);
                        S[4 * i + 0] *= gg.x;
                        S[4 * i + 1] *= gg.y;
                        S[4 * i + 2] *= gg.z;
                        S[4 * i + 3] *= gg.w;
                        r0 = fmaf(S[4 * i + 0], kk.x, r0);
                        r1 = fmaf(S[4 * i + 1], kk.y, r1);
                        r0 = fmaf(S[4 * i + 2], kk.z, r0);
                        r1 = fmaf(S[4 * i + 3], kk.w, r1);
                    }
                    float r = r0 + r1;
                    r += __shfl_xor_sync(0xffffffffu, r, 1);
                    r += __shfl_xor_sync(0xffffffffu, r, 2);
                    const float u = b.beta[tt] * (b.v[tt][cl] - r);
#pragma unroll
                    for (int i = 0; i < DS / 4; i++) {
                        const float4 kk = k4[i], qq = q4[i];
                        S[4 * i + 0] = fmaf(kk.x, u, S[4 * i + 0]);
                        S[4 * i + 1] = fmaf(kk.y, u, S[4 * i + 1]);
                        S[4 * i + 2] = fmaf(kk.z, u, S[4 * i + 2]);
                        S[4 * i + 3] = fmaf(kk.w, u, S[4 * i + 3]);
                        o0 = fmaf(S[4 * i + 0], qq.x, o0);
                        o1 = fmaf(S[4 * i + 1], qq.y, o1);
                        o0 = fmaf(S[4 * i + 2], qq.z, o0);
                        o1 = fmaf(S[4 * i + 3], qq.w, o1);
                    }
                }
                float o = o0 + o1;
                o += __shfl_xor_sync(0xffffffffu, o, 1);
                o += __shfl_xor_sync(0xffffffffu, o, 2);
                if (s == 0 && live) p.o[(t0 + tt) * p.ldo + (int64_t)h * p.Dv + col] = o;
            }
        }
        __syncthreads(); // the chunk is consumed and the next one is staged
    }
#pragma unroll
    for (int i = 0; i < DS; i++) {
        const int d = s * DS + i;
        if (live && d < p.D) sp[(int64_t)d * p.Dv] = S[i];
    }
}

// ------------------------------------------------------------------------------------------------ the recurrences, eight tokens at a time
// With S the state before a chunk of eight tokens, G_t the product of the chunk's decays up to token t and u_t the step
// of token t, all reads of S of the chunk are independent of one another:
//   u_t = beta_t (v_t - G_t S^T k_t - sum_{s<t} (G_t / G_s) (k_s . k_t) u_s)        (lightning: u_t = v_t)
//   o_t = G_t S^T q_t + sum_{s<=t} (G_t / G_s) (k_s . q_t) u_s
//   S  <- G_8 S + sum_s (G_8 / G_s) k_s u_s^T
// (the ratios are computed as products of decays: nothing is divided and nothing overflows).  The same fp32 multiply-adds
// as token by token plus 64 small dots a chunk, but the chain of a chunk is one sum over lanes and one triangular solve
// instead of eight of each, and what a lane reads of k and q serves two columns.
//
// Two kernels.  The first, parallel over chunks, does what does not depend on S: activations, unit norms, decays, the dots between a
// chunk's tokens.  In the second a CTA owns one head and 16 value columns and walks the chunks, whose blocks one lane requests
// ahead (cp.async.bulk, kRing buffers); eight warps run the recurrence, two columns each, without a barrier between them: a lane
// keeps DP / 32 rows of both columns, two rows to a packed multiply-add.
//
// Bound by the chain of a chunk in the two warps a scheduler has (16 heads x 8 slices are 128 CTAs; four warps of four columns
// each issue a fifth less but wait two thirds of the time), and by their instruction issue.
// 1024 tokens x 16 heads of 128 x 128: 262 us token by token, 130 us.
constexpr int kTok = 8, kCols = 16, kRecWarps = 8, kRing = 4;
constexpr int kRecThreads = 32 * (kRecWarps + 1);

// place of pair (s, t), s < t, of a triangle that is kept column by column
__host__ __device__ constexpr int below_diagonal(int s, int t) { return s * 7 - s * (s - 1) / 2 + (t - s - 1); }

// numbers of one chunk and head that are not rows
struct chunk_coef {
    float2 nbk[28];       // -beta_t (G_t / G_s) (k_s . k_t), twice
    float qk[kTok][kTok]; // [t][s <= t]: (G_t / G_s) (k_s . q_t)
    float G[kTok], bG[kTok], gam[kTok], beta[kTok]; // G_t, beta_t G_t (one decay per channel: beta_t), G_8 / G_t, beta_t
    float pad[8];
};
// The rows of one chunk.  One decay per head: of a key head, k and q; one decay per channel: of a head, G_t k_t, G_t q_t, (G_8 / G_t) k_t, G_8.
template <int DP, bool CH> struct chunk_rows {
    float k[kTok][DP], q[kTok][DP];
    float kh[CH ? kTok : 0][DP], gall[CH ? DP : 0];
};
template <int DP, bool CH> struct chunk_block { // what one step of the recurrence reads
    chunk_rows<DP, CH> rows;
    chunk_coef coef;
    float v[kTok][kCols];
};
struct chunk_space { // the first kernel's output: [head or key head][chunk], [head][chunk], [head][slice][chunk]
    unsigned char *rows, *coef, *v;
    int chunks;
};

// 16 values a lane, summed over all lanes: lane l ends with value l / 2.  Two sets at once.
__device__ __forceinline__ void fold16(float (&v)[16], float (&w)[16], int lane) {
#pragma unroll
    for (int n = 8, off = 16; n >= 1; n >>= 1, off >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < n; i++) {
            v[i] = (up ? v[n + i] : v[i]) + __shfl_xor_sync(0xffffffffu, up ? v[i] : v[n + i], off);
            w[i] = (up ? w[n + i] : w[i]) + __shfl_xor_sync(0xffffffffu, up ? w[i] : w[n + i], off);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    w[0] += __shfl_xor_sync(0xffffffffu, w[0], 1);
}

// CTA (chunk, key head; with one decay per channel: head): a warp a token for the rows, then a warp a token s for its dots with the tokens t >= s,
// then a warp a head for the head's own numbers.  Bound by latency: what is read is requested before anything waits.
template <int DP, int MODE>
__global__ void __launch_bounds__(32 * kTok) recurrence_prepare_kernel(rec_args p, chunk_space ws) {
    constexpr bool CH = MODE == 2;
    constexpr int PL = DP / 32;
    __shared__ float s_k[kTok][DP], s_q[kTok][DP], s_g[CH ? kTok : 1][CH ? DP : 1];
    __shared__ float s_dot[2][kTok][kTok]; // [with k, with q][s][t]
    step_wait();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = blockIdx.x, y = blockIdx.y;
    const int per = MODE == 1 ? p.H / p.G : 1, hk = CH ? y / (p.H / p.G) : y; // heads of this CTA: y * per ..; their key head
    const int64_t t = (int64_t)c * kTok + w;
    const bool live = t < p.T;
    chunk_rows<DP, CH> &rows = reinterpret_cast<chunk_rows<DP, CH> *>(ws.rows)[(int64_t)y * ws.chunks + c];
    // what head y * per + w of the last part reads (lane u: token u), and what the head's channels share
    const int hw = y * per + min(w, per - 1), u8 = lane & (kTok - 1);
    const int64_t tu = (int64_t)c * kTok + u8;
    float a_in = MODE == 1 && tu < p.T ? p.a[tu * p.ld_a + hw] : 0.f, b_in = MODE != 0 && tu < p.T ? p.b[tu * p.ld_b + hw] : 0.f;
    const float rate_in = MODE == 0 ? p.decay[hw] : p.A_log && !(CH && p.decays) ? p.A_log[hw] : 0.f, dtb_in = MODE == 1 ? p.dt_bias[hw] : 0.f;
    { // token w of the chunk; one past the end is zeros with a decay of 1
        const float *qr = p.q + t * p.ld + (int64_t)hk * p.D, *kr = p.k + t * p.ld + (int64_t)hk * p.D;
        float q[PL], k[PL], g[PL], gb[PL];
#pragma unroll
        for (int i = 0; i < PL; i++) {
            const int d = lane + 32 * i;
            const bool in = live && d < p.D;
            q[i] = in ? qr[d] : 0.f;
            k[i] = in ? kr[d] : 0.f;
            g[i] = CH && in ? p.a[t * p.ld_a + (int64_t)y * p.D + d] : 0.f;
            gb[i] = CH && in && !p.decays ? p.dt_bias[(int64_t)y * p.D + d] : 0.f;
        }
        // the values of its heads, as they are
        const int slices = (p.Dv + kCols - 1) / kCols, wide = slices * kCols;
        float *vo = reinterpret_cast<float *>(ws.v);
        for (int e0 = lane; e0 < per * wide; e0 += 128) {
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int e = e0 + 32 * i, r = e / wide, x = e - r * wide;
                v[i] = live && r < per && x < p.Dv ? p.v[t * p.ld + (int64_t)(y * per + r) * p.Dv + x] : 0.f;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int e = e0 + 32 * i, r = e / wide, x = e - r * wide;
                if (r < per) vo[((((int64_t)(y * per + r) * slices + x / kCols) * ws.chunks + c) * kTok + w) * kCols + x % kCols] = MODE == 0 ? silu_f32(v[i]) : v[i];
            }
        }
        float qm = 1.f, km = 1.f;
        if (MODE == 0) {
#pragma unroll
            for (int i = 0; i < PL; i++) {
                q[i] = silu_f32(q[i]);
                k[i] = silu_f32(k[i]);
            }
        } else {
            float qs = 0.f, ks = 0.f;
#pragma unroll
            for (int i = 0; i < PL; i++) {
                qs = fmaf(q[i], q[i], qs);
                ks = fmaf(k[i], k[i], ks);
            }
            qm = (1.0f / sqrtf((float)p.D)) / sqrtf(warp_sum_f32(qs) + 1e-6f);
            km = 1.0f / sqrtf(warp_sum_f32(ks) + 1e-6f);
        }
        const float a_rate = CH ? expf(rate_in) : 0.f;
#pragma unroll
        for (int i = 0; i < PL; i++) {
            const int d = lane + 32 * i;
            s_q[w][d] = q[i] * qm;
            s_k[w][d] = k[i] * km;
            if (CH) s_g[CH ? w : 0][CH ? d : 0] = !live || d >= p.D ? 1.f : p.decays ? g[i] : expf(-a_rate * softplus_f32(g[i] + gb[i]));
            else {
                rows.q[w][d] = q[i] * qm;
                rows.k[w][d] = k[i] * km;
            }
        }
    }
    __syncthreads();
    { // s = w: its dots with k_t, q_t, t >= s, decayed from s to t
        float kk[kTok], qk[kTok];
#pragma unroll
        for (int u = 0; u < kTok; u++) kk[u] = qk[u] = 0.f;
#pragma unroll
        for (int i = 0; i < PL; i++) {
            const int d = lane + 32 * i;
            float x = s_k[w][d];
#pragma unroll
            for (int u = 0; u < kTok; u++) {
                if (u < w) continue;
                if (CH && u > w) x *= s_g[CH ? u : 0][CH ? d : 0];
                if (u > w && MODE != 0) kk[u] = fmaf(x, s_k[u][d], kk[u]);
                qk[u] = fmaf(x, s_q[u][d], qk[u]);
            }
        }
        float v[16], unused[16] = {};
#pragma unroll
        for (int u = 0; u < kTok; u++) v[u] = kk[u], v[kTok + u] = qk[u];
        fold16(v, unused, lane);
        if (!(lane & 1)) s_dot[lane >> 4][w][(lane >> 1) & (kTok - 1)] = v[0];
        if (CH) { // token w's rows with the decays of the chunk's tokens up to it and behind it
#pragma unroll
            for (int i = 0; i < PL; i++) {
                const int d = lane + 32 * i;
                float up = 1.f, behind = 1.f;
#pragma unroll
                for (int u = 0; u < kTok; u++) {
                    const float g = s_g[CH ? u : 0][CH ? d : 0];
                    if (u <= w) up *= g;
                    else behind *= g;
                }
                rows.k[w][d] = s_k[w][d] * up;
                rows.q[w][d] = s_q[w][d] * up;
                rows.kh[CH ? w : 0][d] = s_k[w][d] * behind;
                if (w == kTok - 1) rows.gall[CH ? d : 0] = up;
            }
        }
    }
    __syncthreads();
    for (int r = w; r < per; r += kTok) { // the heads' own numbers
        const int h = y * per + r;
        float rate = rate_in, dtb = dtb_in;
        if (r != w) { // more heads to a key head than warps
            a_in = MODE == 1 && tu < p.T ? p.a[tu * p.ld_a + h] : 0.f, b_in = MODE != 0 && tu < p.T ? p.b[tu * p.ld_b + h] : 0.f;
            rate = MODE == 1 ? p.A_log[h] : 0.f, dtb = MODE == 1 ? p.dt_bias[h] : 0.f;
        }
        const float g = CH || tu >= p.T ? 1.f : MODE == 0 ? rate : expf(-expf(rate) * softplus_f32(a_in + dtb)); // decay and step of token u8
        const float beta = tu >= p.T ? 0.f : MODE == 0 ? 1.f : sigmoid_f32(b_in);
        chunk_coef &co = reinterpret_cast<chunk_coef *>(ws.coef)[(int64_t)h * ws.chunks + c];
        float gs[kTok], G = 1.f, gam = 1.f;
#pragma unroll
        for (int i = 0; i < kTok; i++) {
            gs[i] = __shfl_sync(0xffffffffu, g, i);
            if (i <= u8) G *= gs[i];
            else gam *= gs[i];
        }
        if (lane < kTok) co.G[lane] = G, co.gam[lane] = gam, co.bG[lane] = beta * G, co.beta[lane] = beta;
#pragma unroll
        for (int e = 0; e < 2; e++) { // pair (s, t)
            const int s = u8, u = (lane >> 3) + 4 * e;
            float ratio = 1.f;
#pragma unroll
            for (int i = 0; i < kTok; i++)
                if (i > s && i <= u) ratio *= gs[i];
            const float bt = __shfl_sync(0xffffffffu, beta, u);
            co.qk[u][s] = s <= u ? s_dot[1][s][u] * ratio : 0.f;
            if (MODE != 0 && s < u) {
                const float x = -bt * (s_dot[0][s][u] * ratio);
                co.nbk[below_diagonal(s, u)] = make_float2(x, x);
            }
        }
    }
}

template <int DP, int MODE>
__global__ void __launch_bounds__(kRecThreads, 1) recurrence_chunk_kernel(rec_args p, chunk_space ws, int *failed) {
    constexpr bool CH = MODE == 2;
    extern __shared__ __align__(16) unsigned char rec_raw[];
    constexpr int R2 = DP / 64; // pairs of rows of a lane
    typedef chunk_block<DP, CH> block_t;
    block_t *ring = reinterpret_cast<block_t *>(rec_raw);
    __shared__ __align__(16) float s_x[kRecWarps][kTok][2];
    __shared__ __align__(8) unsigned long long s_bar[2 * kRing]; // full, free
    __shared__ int s_dead;
    const int h = blockIdx.x, col0 = blockIdx.y * kCols, chunks = ws.chunks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    volatile int *dead = &s_dead;
    const uint32_t full = smem_u32(s_bar), fre = full + 8 * kRing;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kRing; s++) {
            mbar_init(full + 8 * s, 1);
            mbar_init(fre + 8 * s, kRecWarps);
        }
        s_dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    early_wait();
    if (warp == kRecWarps) { // the blocks of the chunks
        const int hk = CH || MODE == 0 ? h : h / (p.H / p.G);
        const unsigned char *rows = ws.rows + (size_t)hk * chunks * sizeof(block_t::rows), *coef = ws.coef + (size_t)h * chunks * sizeof(chunk_coef);
        const unsigned char *v = ws.v + ((size_t)h * gridDim.y + blockIdx.y) * chunks * sizeof(block_t::v);
        for (int c = 0; c < chunks; c++) {
            const int s = c % kRing;
            if (!mbar_wait_warp(fre + 8 * s, (c / kRing & 1) ^ 1, dead)) break;
            if (lane == 0) {
                mbar_expect_tx(full + 8 * s, sizeof(block_t));
                bulk_load(smem_u32(&ring[s].rows), rows + (size_t)c * sizeof(block_t::rows), sizeof(block_t::rows), full + 8 * s);
                bulk_load(smem_u32(&ring[s].coef), coef + (size_t)c * sizeof(chunk_coef), sizeof(chunk_coef), full + 8 * s);
                bulk_load(smem_u32(&ring[s].v), v + (size_t)c * sizeof(block_t::v), sizeof(block_t::v), full + 8 * s);
            }
        }
        __syncwarp();
    } else {
        // a lane's rows: DP 64: 2 l, + 1; else 128 b + 4 l + i
        f32x2 S[R2][2]; // pairs of rows, column
        float *sp = p.state + (int64_t)h * p.D * p.Dv + col0 + 2 * warp;
        const int cols = p.Dv - (col0 + 2 * warp); // live columns of this warp
        auto row = [&](int i) { return R2 == 1 ? 2 * lane : 128 * (i >> 1) + 4 * lane + 2 * (i & 1); };
        auto pairs = [&](const float *x, f32x2 (&v)[R2]) { // this lane's part of a row
            if constexpr (R2 == 1) {
                v[0] = *reinterpret_cast<const f32x2 *>(x + 2 * lane);
            } else {
#pragma unroll
                for (int i = 0; i < R2; i += 2) {
                    const ulonglong2 y = *reinterpret_cast<const ulonglong2 *>(x + 64 * i + 4 * lane);
                    v[i] = y.x, v[i + 1] = y.y;
                }
            }
        };
#pragma unroll
        for (int i = 0; i < R2; i++)
#pragma unroll
            for (int cc = 0; cc < 2; cc++) {
                const int d = row(i);
                S[i][cc] = pack2(d < p.D && cc < cols ? sp[(int64_t)d * p.Dv + cc] : 0.f, d + 1 < p.D && cc < cols ? sp[(int64_t)(d + 1) * p.Dv + cc] : 0.f);
            }
        const int vt = lane >> 2, vc = (lane >> 1) & 1; // token and column of the value that a fold leaves in this lane and its neighbour
        float *op = p.o + (int64_t)vt * p.ldo + (int64_t)h * p.Dv + col0 + 2 * warp + vc;
        for (int c = 0; c < chunks; c++) {
            const block_t &b = ring[c % kRing];
            const int n = (int)min((int64_t)kTok, p.T - (int64_t)c * kTok);
            mbar_wait_warp(full + 8 * (c % kRing), (c / kRing) & 1, dead);
            float vk[16], vq[16];
            {
                f32x2 ak[kTok][2], aq[kTok][2];
#pragma unroll
                for (int t = 0; t < kTok; t++) {
                    ak[t][0] = ak[t][1] = aq[t][0] = aq[t][1] = 0;
                    f32x2 x[R2], y[R2];
                    pairs(b.rows.q[t], y);
                    if (MODE != 0) pairs(b.rows.k[t], x);
#pragma unroll
                    for (int i = 0; i < R2; i++)
#pragma unroll
                        for (int cc = 0; cc < 2; cc++) {
                            if (MODE != 0) ak[t][cc] = fma2(S[i][cc], x[i], ak[t][cc]);
                            aq[t][cc] = fma2(S[i][cc], y[i], aq[t][cc]);
                        }
                }
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const float2 x = unpack2(ak[i >> 1][i & 1]), y = unpack2(aq[i >> 1][i & 1]);
                    vk[i] = x.x + x.y;
                    vq[i] = y.x + y.y;
                }
            }
            fold16(vk, vq, lane);
            float2 u[kTok];
            if (MODE == 0) {
#pragma unroll
                for (int t = 0; t < kTok; t++) u[t] = *reinterpret_cast<const float2 *>(&b.v[t][2 * warp]);
            } else {
                const float x = fmaf(-b.coef.bG[vt], vk[0], b.coef.beta[vt] * b.v[vt][2 * warp + vc]);
                s_x[warp][vt][vc] = vt < n ? x : 0.f;
                __syncwarp();
                f32x2 y[kTok];
#pragma unroll
                for (int t = 0; t < kTok; t += 2) {
                    const ulonglong2 z = *reinterpret_cast<const ulonglong2 *>(&s_x[warp][t][0]);
                    y[t] = z.x, y[t + 1] = z.y;
                }
                const ulonglong2 *cf = reinterpret_cast<const ulonglong2 *>(b.coef.nbk);
#pragma unroll
                for (int s = 0; s < kTok; s++)
#pragma unroll
                    for (int t = s + 1; t < kTok; t++) {
                        const int e = below_diagonal(s, t);
                        y[t] = fma2(e & 1 ? cf[e >> 1].y : cf[e >> 1].x, y[s], y[t]);
                    }
#pragma unroll
                for (int t = 0; t < kTok; t++) u[t] = unpack2(y[t]);
                __syncwarp(); // the next chunk writes s_x
            }
#pragma unroll
            for (int i = 0; i < R2; i++) {
                const f32x2 g = CH ? *reinterpret_cast<const f32x2 *>(&b.rows.gall[CH ? row(i) : 0]) : pack2(b.coef.G[kTok - 1], b.coef.G[kTok - 1]);
#pragma unroll
                for (int cc = 0; cc < 2; cc++) S[i][cc] = mul2(S[i][cc], g);
            }
#pragma unroll
            for (int t = 0; t < kTok; t++) {
                const float gam = CH ? 1.f : b.coef.gam[t];
                const float ux = CH ? u[t].x : u[t].x * gam, uy = CH ? u[t].y : u[t].y * gam;
                const f32x2 u0 = pack2(ux, ux), u1 = pack2(uy, uy);
                f32x2 x[R2];
                pairs((CH ? &b.rows.kh[0][0] : &b.rows.k[0][0]) + t * DP, x);
#pragma unroll
                for (int i = 0; i < R2; i++) {
                    S[i][0] = fma2(x[i], u0, S[i][0]);
                    S[i][1] = fma2(x[i], u1, S[i][1]);
                }
            }
            float o = CH ? vq[0] : b.coef.G[vt] * vq[0];
            const float4 c0 = *reinterpret_cast<const float4 *>(&b.coef.qk[vt][0]), c1 = *reinterpret_cast<const float4 *>(&b.coef.qk[vt][4]);
            const float cf[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
            for (int s = 0; s < kTok; s++) {
                const float w = fmaf(cf[s], vc ? u[s].y : u[s].x, o);
                o = s <= vt ? w : o; // what is past this token (an infinity, too) stays out
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(fre + 8 * (c % kRing));
            if (!(lane & 1) && vt < n && vc < cols) *op = o;
            op += (int64_t)kTok * p.ldo;
        }
#pragma unroll
        for (int i = 0; i < R2; i++)
#pragma unroll
            for (int cc = 0; cc < 2; cc++) {
                const int d = row(i);
                const float2 s2 = unpack2(S[i][cc]);
                if (d < p.D && cc < cols) sp[(int64_t)d * p.Dv + cc] = s2.x;
                if (d + 1 < p.D && cc < cols) sp[(int64_t)(d + 1) * p.Dv + cc] = s2.y;
            }
    }
    __syncthreads();
    if (warp == 0) {
        settle(dead);
        if (lane == 0 && s_dead) *failed = 1;
    }
}

// ------------------------------------------------------------------------------------------------ second halves of two low-rank projections
// x rows hold the first halves [a1 (Ka) | g1 (Kg)] in fp32; CTA (x, y) owns 128 outputs of one of the two matrices and 16
// tokens: the tokens' rows wait in shared memory rounded through the matrices' type, a thread owns one output for all 16 tokens
// and streams its matrix row once in 16-byte pieces (every piece feeds 16 x 8 or 16 x 4 multiply-adds against broadcast reads).
// The decay's outputs leave as exp(-exp(A_log[head]) softplus(. + dt_bias)), the gate's as they are.
constexpr int kLrTokens = 16, kLrOut = 128;

template <typename E>
__global__ void __launch_bounds__(kLrOut) lowrank_pair_kernel(const float *__restrict__ x, int64_t ldx, int64_t T, const E *__restrict__ w_a, int64_t Na,
                                                              int Ka, const E *__restrict__ w_g, int64_t Ng, int Kg, const float *__restrict__ A_log,
                                                              const float *__restrict__ dt_bias, int D, float *__restrict__ a,
                                                              float *__restrict__ g, int vec) {
    extern __shared__ __align__(16) float lr_x[]; // [kLrTokens][Kp]
    constexpr int VE = 16 / (int)sizeof(E);
    const int blocks_a = (int)((Na + kLrOut - 1) / kLrOut);
    const bool is_a = (int)blockIdx.x < blocks_a;
    const int64_t n = (int64_t)(is_a ? blockIdx.x : blockIdx.x - blocks_a) * kLrOut + threadIdx.x, N = is_a ? Na : Ng;
    const int K = is_a ? Ka : Kg, koff = is_a ? 0 : Ka, Kp = (K + 3) & ~3;
    const int64_t t0 = (int64_t)blockIdx.y * kLrTokens;
    const int nt = (int)min((int64_t)kLrTokens, T - t0);
    for (int e = threadIdx.x; e < kLrTokens * Kp; e += blockDim.x) {
        const int tt = e / Kp, k = e - tt * Kp;
        lr_x[e] = (tt < nt && k < K) ? to_f32(from_f32<E>(x[(t0 + tt) * ldx + koff + k])) : 0.f;
    }
    __syncthreads();
    if (n >= N) return;
    const E *wr = (is_a ? w_a : w_g) + n * K;
    float acc[kLrTokens];
#pragma unroll
    for (int tt = 0; tt < kLrTokens; tt++) acc[tt] = 0.f;
    if (vec) { // K a multiple of the 16-byte piece, rows aligned
        for (int k = 0; k < K; k += VE) {
            const uint4 wv = *reinterpret_cast<const uint4 *>(wr + k);
            const E *we = reinterpret_cast<const E *>(&wv);
            float wf[VE];
#pragma unroll
            for (int u = 0; u < VE; u++) wf[u] = to_f32(we[u]);
#pragma unroll
            for (int tt = 0; tt < kLrTokens; tt++) {
#pragma unroll
                for (int u = 0; u < VE; u += 4) {
                    const float4 xv = *reinterpret_cast<const float4 *>(lr_x + tt * Kp + k + u);
                    acc[tt] = fmaf(wf[u], xv.x, acc[tt]);
                    acc[tt] = fmaf(wf[u + 1], xv.y, acc[tt]);
                    acc[tt] = fmaf(wf[u + 2], xv.z, acc[tt]);
                    acc[tt] = fmaf(wf[u + 3], xv.w, acc[tt]);
                }
            }
        }
    } else {
        for (int k = 0; k < K; k++) {
            const float wf = to_f32(wr[k]);
#pragma unroll
            for (int tt = 0; tt < kLrTokens; tt++) acc[tt] = fmaf(wf, lr_x[tt * Kp + k], acc[tt]);
        }
    }
    if (is_a && A_log) {
        const float rate = expf(A_log[n / D]), bias = dt_bias[n];
#pragma unroll
        for (int tt = 0; tt < kLrTokens; tt++) acc[tt] = expf(-rate * softplus_f32(acc[tt] + bias));
    }
    float *out = is_a ? a : g;
#pragma unroll
    for (int tt = 0; tt < kLrTokens; tt++)
        if (tt < nt) out[(t0 + tt) * N + n] = acc[tt];
}

template <int DS, int CV, int MODE>
int recurrence_launch_cv(const rec_args &p) {
    const dim3 grid((unsigned)p.H, (unsigned)((p.Dv + CV - 1) / CV));
    const size_t smem = 2 * sizeof(rec_smem<DS, CV, MODE == 2>);
    auto k = recurrence_kernel<DS, CV, MODE>;
    if (smem > 48 * 1024) GGB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k<<<grid, CV * kNS + 32 * kStageWarps, smem, ggb_cuda_stream()>>>(p);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

// value columns per CTA: 16 while that leaves a CTA per SM at most (the kernel is bound by instruction issue of the one
// CTA an SM holds, so more SMs per head is what helps), else 32
template <int DS, int MODE>
int recurrence_launch_ds(const rec_args &p) {
    if ((int64_t)p.H * ((p.Dv + 15) / 16) <= ggb_sm_count()) return recurrence_launch_cv<DS, 16, MODE>(p);
    return recurrence_launch_cv<DS, 32, MODE>(p);
}

// Tokens in segments whose prepared chunks fit the workspace (the state carries over from segment to segment).  The workspace has one size, so that
// it stays where it is: a graph holds its address.  Where it cannot be had - it does not exist yet and a graph is being captured - or one
// chunk would not fit it, the token by token form runs.
constexpr size_t kChunkSpace = (size_t)32 << 20;
template <int DP, int MODE>
int recurrence_launch_chunks(rec_args p, bool *done) {
    constexpr bool CH = MODE == 2;
    typedef chunk_block<DP, CH> block_t;
    const int slices = (p.Dv + kCols - 1) / kCols, rows_of = CH ? p.H : MODE == 1 ? p.G : p.H;
    const size_t per_chunk = rows_of * sizeof(block_t::rows) + p.H * (sizeof(chunk_coef) + slices * sizeof(block_t::v));
    const int64_t total = (p.T + kTok - 1) / kTok, most = (int64_t)(kChunkSpace / per_chunk);
    *done = most > 0 && ggb_workspace_fits(GGB_WS_RECURRENCE, kChunkSpace);
    if (!*done) return GGB_OK;
    const size_t smem = kRing * sizeof(block_t);
    auto k = recurrence_chunk_kernel<DP, MODE>;
    void *space;
    int rc = ggb_allow_smem(k, smem);
    if (!rc) rc = ggb_workspace(GGB_WS_RECURRENCE, kChunkSpace, &space);
    for (int64_t c0 = 0; c0 < total && !rc; c0 += most) {
        const int chunks = (int)std::min(total - c0, most);
        chunk_space ws{(unsigned char *)space, nullptr, nullptr, chunks};
        ws.coef = ws.rows + (size_t)rows_of * chunks * sizeof(block_t::rows);
        ws.v = ws.coef + (size_t)p.H * chunks * sizeof(chunk_coef);
        rec_args q = p;
        const int64_t t0 = c0 * kTok;
        q.q += t0 * p.ld, q.k += t0 * p.ld, q.v += t0 * p.ld, q.o += t0 * p.ldo, q.T = std::min<int64_t>(p.T - t0, (int64_t)chunks * kTok);
        if (q.b) q.b += t0 * p.ld_b;
        if (q.a) q.a += t0 * p.ld_a;
        GGB_CUDA(ggb_launch_step(recurrence_prepare_kernel<DP, MODE>, dim3((unsigned)chunks, (unsigned)rows_of), dim3(32 * kTok), 0, q, ws));
        GGB_LAUNCH_CHECK();
        GGB_CUDA(ggb_launch_early(k, ggb_cluster{1, 1, 1}, dim3((unsigned)p.H, (unsigned)slices), dim3(kRecThreads), smem, q, ws, ggb_wait_error_flag()));
        GGB_LAUNCH_CHECK();
    }
    return rc;
}

template <int MODE>
int recurrence_launch(const rec_args &p) {
    if (p.T >= 2 * kTok) {
        bool done;
        const int rc = p.D <= 64    ? recurrence_launch_chunks<64, MODE>(p, &done)
                       : p.D <= 128 ? recurrence_launch_chunks<128, MODE>(p, &done)
                                    : recurrence_launch_chunks<256, MODE>(p, &done);
        if (rc || done) return rc;
    }
    const int ds = (p.D + kNS - 1) / kNS;
    if (ds <= 8) return recurrence_launch_ds<8, MODE>(p);
    if (ds <= 16) return recurrence_launch_ds<16, MODE>(p);
    if (ds <= 32) return recurrence_launch_ds<32, MODE>(p);
    return recurrence_launch_ds<64, MODE>(p);
}

} // namespace

extern "C" {

int ggb_op_causal_conv(int dt, const float *x, int64_t ldx, int64_t T, int64_t C, const float *w, int taps, int add_input, int act,
                       float *tail, float *y_f32, int64_t ldy, void *y_dt) {
    return ggb_op_causal_conv_bias(dt, x, ldx, T, C, w, nullptr, taps, add_input, act, tail, y_f32, ldy, y_dt);
}

int ggb_op_causal_conv_bias(int dt, const float *x, int64_t ldx, int64_t T, int64_t C, const float *w, const float *bias, int taps,
                            int add_input, int act, float *tail, float *y_f32, int64_t ldy, void *y_dt) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(dt == GGB_TYPE_BF16 || dt == GGB_TYPE_F32, "causal_conv: dtype %d is neither bf16 nor f32", dt);
    GGB_CHECK_ARG(x && w && T > 0 && C > 0 && ldx >= C && taps >= 1 && taps <= kConvMaxTaps && (taps == 1 || tail) && (y_f32 || y_dt) &&
                      (!y_f32 || ldy >= C),
                  "causal_conv: bad arguments (taps %d, at most %d)", taps, kConvMaxTaps);
    const dim3 grid((unsigned)((C + 127) / 128), (unsigned)((T + kConvTokens - 1) / kConvTokens));
    if (dt == GGB_TYPE_BF16)
        causal_conv_kernel<<<grid, 128, 0, ggb_cuda_stream()>>>(x, ldx, T, C, w, bias, taps, add_input, act, tail, y_f32, ldy, (__nv_bfloat16 *)y_dt);
    else
        causal_conv_kernel<<<grid, 128, 0, ggb_cuda_stream()>>>(x, ldx, T, C, w, bias, taps, add_input, act, tail, y_f32, ldy, (float *)y_dt);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_lowrank_pair_fits(int dt, int Ka, int Kg) { return (size_t)kLrTokens * (size_t)(std::max(Ka, Kg) + 3) * 4 <= 48 * 1024; }

int ggb_op_lowrank_pair(int dt, const float *x, int64_t ldx, int64_t T, const void *w_a, int64_t Na, int Ka, const void *w_g, int64_t Ng, int Kg,
                        const float *A_log, const float *dt_bias, int D, float *a, float *g) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(dt == GGB_TYPE_BF16 || dt == GGB_TYPE_F32, "lowrank_pair: dtype %d is neither bf16 nor f32", dt);
    GGB_CHECK_ARG(x && w_a && w_g && a && g && T > 0 && Na > 0 && Ng > 0 && Ka > 0 && Kg > 0 && ldx >= Ka + Kg && (!A_log || (dt_bias && D > 0 && Na % D == 0)),
                  "lowrank_pair: bad arguments");
    GGB_CHECK_ARG(ggb_lowrank_pair_fits(dt, Ka, Kg), "lowrank_pair: inner sizes %d / %d do not fit shared memory", Ka, Kg);
    const int ve = dt == GGB_TYPE_BF16 ? 8 : 4;
    const int vec = Ka % ve == 0 && Kg % ve == 0 && (((uintptr_t)w_a | (uintptr_t)w_g) & 15) == 0;
    const size_t smem = (size_t)kLrTokens * (size_t)((std::max(Ka, Kg) + 3) & ~3) * 4;
    const dim3 grid((unsigned)((Na + kLrOut - 1) / kLrOut + (Ng + kLrOut - 1) / kLrOut), (unsigned)((T + kLrTokens - 1) / kLrTokens));
    if (dt == GGB_TYPE_BF16)
        lowrank_pair_kernel<<<grid, kLrOut, smem, ggb_cuda_stream()>>>(x, ldx, T, (const __nv_bfloat16 *)w_a, Na, Ka, (const __nv_bfloat16 *)w_g, Ng, Kg, A_log,
                                                                      dt_bias, D, a, g, vec);
    else
        lowrank_pair_kernel<<<grid, kLrOut, smem, ggb_cuda_stream()>>>(x, ldx, T, (const float *)w_a, Na, Ka, (const float *)w_g, Ng, Kg, A_log, dt_bias, D, a, g,
                                                                      vec);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_op_lightning_attn(const float *q, const float *k, const float *v, int64_t ld, int64_t T, int H, int D, int Dv, const float *decay,
                          float *state, float *o, int64_t ldo) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(q && k && v && decay && state && o && T > 0 && H > 0 && D > 0 && D <= 64 * kNS && Dv > 0 && ldo >= (int64_t)H * Dv,
                  "lightning_attn: bad arguments (key size %d, at most %d)", D, 64 * kNS);
    rec_args p{q, k, v, nullptr, nullptr, ld, 0, 0, T, H, H, D, Dv, decay, nullptr, nullptr, state, o, ldo, 0};
    return recurrence_launch<0>(p);
}

int ggb_op_gated_delta(const float *q, const float *k, const float *v, int64_t ld, const float *b, const float *a, int64_t ld_ba, int64_t T,
                       int H, int G, int D, int Dv, const float *A_log, const float *dt_bias, float *state, float *o, int64_t ldo) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(q && k && v && b && a && A_log && dt_bias && state && o && T > 0 && H > 0 && G > 0 && H % G == 0 && D > 0 && D <= 64 * kNS &&
                      Dv > 0 && ldo >= (int64_t)H * Dv,
                  "gated_delta: bad arguments (heads %d over %d key heads, key size %d)", H, G, D);
    rec_args p{q, k, v, b, a, ld, ld_ba, ld_ba, T, H, G, D, Dv, nullptr, A_log, dt_bias, state, o, ldo, 0};
    return recurrence_launch<1>(p);
}

int ggb_op_channel_delta(const float *q, const float *k, const float *v, int64_t ld, const float *b, int64_t ld_b, const float *a, int64_t ld_a,
                         int decays, int64_t T, int H, int G, int D, int Dv, const float *A_log, const float *dt_bias, float *state, float *o,
                         int64_t ldo) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(q && k && v && b && a && (decays || (A_log && dt_bias)) && state && o && T > 0 && H > 0 && G > 0 && H % G == 0 && D > 0 &&
                      D <= 64 * kNS && Dv > 0 && ldo >= (int64_t)H * Dv && ld_a >= (int64_t)H * D && ld_b >= H,
                  "channel_delta: bad arguments (heads %d over %d key heads, key size %d)", H, G, D);
    rec_args p{q, k, v, b, a, ld, ld_b, ld_a, T, H, G, D, Dv, nullptr, A_log, dt_bias, state, o, ldo, decays};
    return recurrence_launch<2>(p);
}

} // extern "C"
