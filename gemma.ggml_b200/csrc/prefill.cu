// prefill.cu — the one genuinely dense contraction of the path: mul_mat with col_num = T > 1
// (ref: src/hpc.cpp:216-277 called with ne11 = T; graph nodes at src/gemma_model.cpp:692-696, 493, 446-450,
// 740).  Decode (T = 1) is 2 flop per weight byte and HBM-bound; prefill re-uses every weight T times, so it
// belongs on the 5th-generation tensor cores:
//
//   C[T][N] (fp32) = A[T][K] (bf16 activations) x dequant(W[N][K] Q4_0 | Q8_0)^T       (+ residual)
//
// Large products of more than 256 rows: two CTAs of a cluster compute a tile (cta_group::2) of 512 or 256 rows x up to 256 columns; each holds half of the
// rows of A and dequantises half of the tile's weight rows, so a prompt of 512 tokens dequantises every weight once.  Others: one
// CTA, 256 or 128 rows x up to 128 columns.  Per 64-wide K block
//   * one thread requests the CTA's A rows by TMA, another one the raw codes (a ring of their own: they are needed a dequantisation earlier);
//   * two groups of eight warps (four of four, eight of two where the tile has fewer weight rows) take the K blocks in turn and DEQUANTISE the W rows (int8 / int4 codes x fp16 block scale -> bf16, exact
//     product rounded once) from shared memory into shared memory, canonical K-major 128-byte-swizzled UMMA layout;
//   * one warp (of the pair's first CTA) issues the tcgen05.mma (K = 16, kind::f16, bf16 x bf16 -> fp32) whose accumulators live in TENSOR
//     MEMORY, up to all 512 columns; tcgen05.commit releases the buffers of both CTAs;
//   * after the last K block the sixteen warps become the EPILOGUE: 32 x 32 pieces turned in shared memory, residual added, whole lines stored.
//     gate | up of a feed-forward: each CTA dequantises rows of one of the two matrices, so both products of an output stand in the same row
//     of tensor memory and leave as gelu(gate) * up in bf16; the 128 KB gelu table is brought into the ring behind the last MMA.
// A product along a long K is summed in pieces of K (as many as a split over the SMs in 256 x 256 tiles needs): several accumulators a
// CTA in tensor memory, added in order by the epilogue, and, where SMs are left, several CTAs, whose pieces all meet in a workspace and are
// added in order by a second kernel: the same bits whichever tile is chosen.
//
// What bounds it.  Large products: the MMAs (140 cycles each of the 128 that a pair's 256 x 256 x 16 takes at least) and what no other tile
// hides, 3 us up to the first MMA and 7 us from the last one to the end, at clocks that fall under the power limit.  A K block has one barrier
// that its A rows and all its dequantising warps arrive on, of both CTAs, and one commit: a wait or commit costs the issuing warp 100 to 200
// cycles whether it has to wait or not (three waits and two commits a block: 900 cycles a block of any tile).  Small products: that start
// and end.  512 tokens, Q8_0: gate | up with gelu 65 us (1060 TFLOP/s; 72 with three waits and two commits a K block; 115 in two launches before),
// 2048 x 16384 in 8 pieces 45 -> 40 to 42 us with its sums, 2048 x 2048 20 -> 16 us, q | k | v 22.5 -> 17 us.
//
// Numerics: weights q*d are exact in fp32 (8 x 11 bits) and rounded once to bf16; activations are rounded
// to bf16 instead of being re-quantised to Q8_0 per 32 (the reference's INIT stage), so prefill agrees with
// the reference within a tolerance (tests/test_prefill_gpu.py), not bit for bit — the decode path is the
// bit-exact one.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "dense.cuh"
#include "prefill_attention.cuh"
#include "tc.cuh"

namespace {

constexpr int BK = 64;
constexpr int kWorkWarps = 16, kTmaWarp = 16, kMmaWarp = 17, kCodesWarp = 18, kGemmThreads = 32 * 19;
constexpr uint32_t kRing = 224 * 1024;
constexpr int kMaxStages = 8;
constexpr size_t kGemmSmem = 1024 + kRing + 512;
static_assert(kGemmSmem >= kOneCtaSmem, "pairs of CTAs");
constexpr uint32_t kTiles = 256 * 128; // bytes of the buffers of dequantised weights, one a group
constexpr int kMaxCodeStages = 16;
enum { FULL = 0, FREE = 64, C_FULL = 128, C_FREE = 256, DONE = 384, SLOT = 392, DEAD = 400, TABLE_FULL = 408 }; // FULL, FREE: of a K block, by its stage of A
constexpr uint32_t kGeluBytes = 65536 * 2, kGeluAt = 64 * 1024; // the gelu table, behind the epilogue's 16 x 4 KB, in the ring, which the last MMA has left

// up to 3 weight matrices that share the A operand run as ONE launch (Q | K | V, gate | up): a segment = one matrix, its first row is a
// multiple of 256, so a tile belongs to exactly one segment
constexpr int kMaxSegs = 3;
struct GemmSeg {
    const __half *d;     // weight scale plane [rows][nb]
    float *c;            // [T][ldc] output of this matrix
    int ldc;
    int n_begin, rows;   // first row of the segment in the concatenated N, its row count
};
struct GemmArgs {
    GemmSeg seg[kMaxSegs];
    int n_seg;
    int N, nb, kblocks;  // N = concatenated rows (padded between segments), nb = K / 32, kblocks = K / 64
    int T, MT, BN;       // a CTA's rows: MT x 128; a tile's columns
    int groups;                                // of warps, that take the K blocks in turn
    int chunks, chunk_kb, stages, code_stages; // stages of A rows, of codes (a multiple of the groups)
    uint32_t a_tx;       // bytes of a stage of A that are loaded: a single row tile leaves out what lies 8 rows and more past the last
    int vec;             // rows of every C and of resid start on 16 bytes
    float *ws;           // workspace [pieces of K][T][N] or null (one CTA along K: tiles go straight to seg.c)
    const float *resid;  // [T][seg[0].ldc] or null (single segment, no workspace)
    __nv_bfloat16 *geglu; // two segments, gate and up, of which every tile takes BN / 2 rows each: [T][rows] gelu(gate) * up
    const uint16_t *gelu; // the fp16 table of gelu
    int *wait_error;
};
struct GemmMaps {
    CUtensorMap a, w[kMaxSegs];
};

// int8 / int4 codes -> bf16 weights without the conversion pipe.  A byte permute puts the biased code into the mantissa of 2^15, and one
// multiply-add of two numbers takes the bias out and applies the block scale: (2^15 + bias + code) d - (2^15 + bias) d, exact, since d has 11
// significant bits and 2^15 + 128 has 9 of them, 2^15 + 8 has 13; the product, exact in fp32 (8 x 11 bits), is rounded once to bf16.  A scale
// that is infinite is applied behind the bias.  Bound by the permutes and roundings, which issue every other cycle: 32 weights of a lane are 110
// instructions (170 with an addition and a multiplication each).
struct block_scale {
    f32x2 d, c;
    float last; // an infinite scale
    __device__ __forceinline__ block_scale(float scale, float bias) {
        const bool odd = fabsf(scale) > 65504.f;
        last = odd ? scale : 1.f;
        const float f = odd ? 1.f : scale;
        d = pack2(f, f), c = pack2(__fmul_rn(-bias, f), __fmul_rn(-bias, f));
    }
};
__device__ __forceinline__ void codes_to_bf16x16(const uint32_t (&w)[4], const block_scale &b, uint32_t (&o)[8]) {
    float2 v[8];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        v[2 * i] = unpack2(fma2(pack2(__uint_as_float(__byte_perm(w[i], 0x47000000u, 0x7404)), __uint_as_float(__byte_perm(w[i], 0x47000000u, 0x7414))), b.d, b.c));
        v[2 * i + 1] = unpack2(fma2(pack2(__uint_as_float(__byte_perm(w[i], 0x47000000u, 0x7424)), __uint_as_float(__byte_perm(w[i], 0x47000000u, 0x7434))), b.d, b.c));
    }
    if (b.last != 1.f)
#pragma unroll
        for (int i = 0; i < 8; i++) v[i].x *= b.last, v[i].y *= b.last;
#pragma unroll
    for (int i = 0; i < 8; i++) o[i] = pack_bf16x2(v[i].x, v[i].y);
}
// 16 bf16 of dequantised weights (two 16-byte chunks of the swizzled row) from 16 int8 codes; b of 32896
__device__ __forceinline__ void dequant16_q8(const uint4 w, const block_scale &b, uint4 &lo, uint4 &hi) {
    const uint32_t u[4] = {w.x ^ 0x80808080u, w.y ^ 0x80808080u, w.z ^ 0x80808080u, w.w ^ 0x80808080u}; // code + 128
    uint32_t out[8];
    codes_to_bf16x16(u, b, out);
    lo = make_uint4(out[0], out[1], out[2], out[3]);
    hi = make_uint4(out[4], out[5], out[6], out[7]);
}
// one Q4_0 block (16 payload bytes -> 32 weights, nibble - 8): elements 0..15 are the low nibbles, 16..31 the high ones; b of 32776
__device__ __forceinline__ void dequant32_q4(const uint4 w, const block_scale &b, uint4 (&o)[4]) {
    const uint32_t l[4] = {w.x & 0x0F0F0F0Fu, w.y & 0x0F0F0F0Fu, w.z & 0x0F0F0F0Fu, w.w & 0x0F0F0F0Fu};
    const uint32_t h[4] = {(w.x >> 4) & 0x0F0F0F0Fu, (w.y >> 4) & 0x0F0F0F0Fu, (w.z >> 4) & 0x0F0F0F0Fu, (w.w >> 4) & 0x0F0F0F0Fu};
    uint32_t lo[8], hi[8];
    codes_to_bf16x16(l, b, lo);
    codes_to_bf16x16(h, b, hi);
    o[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    o[1] = make_uint4(lo[4], lo[5], lo[6], lo[7]);
    o[2] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    o[3] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
}

__device__ __forceinline__ void sts_u4(uint32_t addr, const uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 lds_u4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ float4 load4(const float *p, int vec) { return vec ? *reinterpret_cast<const float4 *>(p) : make_float4(p[0], p[1], p[2], p[3]); }
__device__ __forceinline__ void store4(float *p, const float4 v, int vec) {
    if (vec) *reinterpret_cast<float4 *>(p) = v;
    else p[0] = v.x, p[1] = v.y, p[2] = v.z, p[3] = v.w;
}

template <int TYPE, bool PAIR>
__global__ void __launch_bounds__(kGemmThreads, 1) gemm_quant_kernel(const __grid_constant__ GemmMaps maps, const GemmArgs A) {
    extern __shared__ uint8_t gemm_smem_raw[];
    constexpr int PB = TYPE == GGB_TYPE_Q8_0 ? 32 : 16; // payload bytes of a block of 32 weights
    const uint32_t raw0 = smem_u32(gemm_smem_raw), smem0 = (raw0 + 1023u) & ~1023u, bars = smem0 + kRing;
    uint8_t *gbase = gemm_smem_raw + (smem0 - raw0);
    volatile int *dead = reinterpret_cast<volatile int *>(gbase + kRing + DEAD);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int rank = PAIR ? (int)cluster_rank() : 0, CTAS = PAIR ? 2 : 1;
    const int n0 = blockIdx.y * A.BN, m0 = (PAIR ? blockIdx.x / 2 * 2 + rank : blockIdx.x) * A.MT * 128, split = blockIdx.z, BR = A.BN / CTAS;
    int si = 0;
    if (A.geglu) si = rank;
    else if (A.n_seg > 1 && n0 >= A.seg[1].n_begin) si = (A.n_seg > 2 && n0 >= A.seg[2].n_begin) ? 2 : 1;
    const GemmSeg &sg = A.seg[si];
    const int sn0 = A.geglu ? n0 / 2 : n0 - sg.n_begin; // first row of this tile inside its matrix
    const int w_row0 = A.geglu ? sn0 : sn0 + rank * BR; // first weight row of this CTA
    const int kb0 = split * A.chunks * A.chunk_kb, kb1 = min(kb0 + A.chunks * A.chunk_kb, A.kblocks);
    if (sn0 >= sg.rows) return; // padding between matrices: all CTAs of the tile, before any barrier or tensor memory exists
    const uint32_t b_bytes = (uint32_t)BR * 128, a_bytes = (uint32_t)A.MT * 16384, c_bytes = (uint32_t)BR * 2 * PB;
    const uint32_t codes = smem0 + kTiles, ring = codes + A.code_stages * c_bytes; // dequantised tiles | codes | A rows

    const int group_warps = kWorkWarps / A.groups;
    if (tid == 0) {
        for (int s = 0; s < A.stages; s++) {
            mbar_init(bars + FULL + 8 * s, 1 + CTAS * group_warps); // the bytes of A and the warps that dequantise, of both CTAs
            mbar_init(bars + FREE + 8 * s, 1);
        }
        for (int s = 0; s < A.code_stages; s++) {
            mbar_init(bars + C_FULL + 8 * s, 1);
            mbar_init(bars + C_FREE + 8 * s, group_warps);
        }
        mbar_init(bars + DONE, 1);
        mbar_init(bars + TABLE_FULL, 1);
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        if (PAIR) tmem_alloc512_pair(bars + SLOT);
        else tmem_alloc512(bars + SLOT);
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<uint32_t *>(gbase + kRing + SLOT), 0);

    const uint32_t full = PAIR ? cluster_addr(bars + FULL, 0) : bars + FULL; // the issuing CTA's

    if (warp < kWorkWarps) {
        // ================= the groups take the K blocks in turn; thread t of one owns ONE quant block (32 weights): row w_row0 + (t >> 1), block 2 kb + (t & 1)
        const int G = A.groups, grp = warp / group_warps, gt = tid & (32 * group_warps - 1), wr = gt >> 1, whalf = gt & 1, wrow = w_row0 + wr;
        const bool live = wrow < sg.rows;
        const __half *dp = sg.d + (size_t)wrow * A.nb + whalf;
        const uint32_t dst = smem0 + grp * b_bytes + wr * 128;
        __half cur[4], nxt[4]; // scales of the group's next four K blocks, requested while the four before are used
        auto scales = [&](int kb, __half (&d)[4]) {
#pragma unroll
            for (int u = 0; u < 4; u++) d[u] = live && kb + G * u < kb1 ? __ldg(dp + 2 * (kb + G * u)) : __float2half(0.f);
        };
        scales(kb0 + grp, nxt);
        int s = grp, as = grp, before = -1; // stages of codes and of A; that of A of the group's block before
        uint32_t ph = 0, aph = 0, bph = 0;
        for (int kbase = kb0 + grp; kbase < kb1; kbase += 4 * G) {
#pragma unroll
            for (int u = 0; u < 4; u++) cur[u] = nxt[u];
            scales(kbase + 4 * G, nxt);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (kbase + G * u >= kb1) break;
                mbar_wait_warp(bars + C_FULL + 8 * s, ph, dead);
                uint4 o[4];
                // rows past the matrix: zero codes (TMA) and zero scales
                const block_scale d0(__half2float(cur[u]), TYPE == GGB_TYPE_Q8_0 ? 32896.f : 32776.f);
                const uint32_t src = codes + s * c_bytes + gt * PB;
                if (TYPE == GGB_TYPE_Q8_0) {
                    // the two 16-byte pieces in an order in which eight lanes meet eight groups of banks
                    const uint32_t first = (lane >> 2) & 1;
                    const uint4 x = lds_u4(src + 16 * first), y = lds_u4(src + 16 * (first ^ 1));
                    dequant16_q8(first ? y : x, d0, o[0], o[1]);
                    dequant16_q8(first ? x : y, d0, o[2], o[3]);
                } else {
                    dequant32_q4(lds_u4(src), d0, o);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bars + C_FREE + 8 * s); // the codes are in registers
                if (before >= 0) mbar_wait_warp(bars + FREE + 8 * before, bph, dead); // the group's buffer
#pragma unroll
                for (int q = 0; q < 4; q++) sts_u4(dst + (((4 * whalf + q) ^ (wr & 7)) << 4), o[q]);
                fence_async_smem();
                __syncwarp();
                if (lane == 0) {
                    if (PAIR) mbar_arrive_cluster(full + 8 * as);
                    else mbar_arrive(full + 8 * as);
                }
                before = as, bph = aph;
                as += G;
                if (as >= A.stages) as -= A.stages, aph ^= 1u;
                s += G;
                if (s >= A.code_stages) s -= A.code_stages, ph ^= 1u;
            }
        }
        // ================= epilogue: pieces of 32 rows x 32 columns, dealt to the four warps of a lane quarter
        mbar_wait_warp(bars + DONE, 0, dead);
        tc_fence_after();
        const int chunks = kb1 > kb0 ? (kb1 - kb0 + A.chunk_kb - 1) / A.chunk_kb : 0, lq = warp & 3, cols = (A.geglu ? A.BN / 2 : A.BN) / 32;
        const int planes = A.ws ? chunks : 1; // in a workspace every piece along K stands alone: they are added in order, whichever CTA summed them
        float *cbase = A.ws ? A.ws + (size_t)split * A.chunks * A.T * A.N + n0 : sg.c + sn0;
        const int cld = A.ws ? A.N : sg.ldc;
        const uint32_t my = smem0 + warp * 4096; // the ring is no longer used
        if (A.geglu) mbar_wait_warp(bars + TABLE_FULL, 0, dead);
        auto gelu = [&](uint32_t g) { // of an fp16 number, rounded to fp16: the table, as ggb_op_geglu_bf16 reads it
            uint16_t h;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(smem0 + kGeluAt + 2u * float_to_half_bits(__uint_as_float(g))) : "memory");
            return half_bits_to_float(h);
        };
        for (int piece = warp >> 2; piece < A.MT * cols; piece += kWorkWarps / 4) {
            const int mt = piece / cols, c0 = (piece - mt * cols) * 32, row0 = m0 + mt * 128 + lq * 32;
            if (row0 >= A.T || sn0 + c0 >= sg.rows) continue;
            uint32_t v[32];
            const uint32_t col = tmem + ((uint32_t)(lq * 32) << 16) + (uint32_t)(mt * A.chunks * A.BN + c0);
            auto add_columns = [&](uint32_t at) {
#pragma unroll
                for (int hf = 0; hf < 2; hf++) {
                    uint32_t u[16];
                    tmem_load16(at + 16 * hf, u);
#pragma unroll
                    for (int q = 0; q < 16; q++) v[16 * hf + q] = __float_as_uint(__uint_as_float(v[16 * hf + q]) + __uint_as_float(u[q]));
                }
            };
            for (int plane = 0; plane < planes; plane++) {
                tmem_load32(col + plane * A.BN, v);
                if (!A.ws)
                    for (int ch = 1; ch < chunks; ch++) add_columns(col + ch * A.BN);
                if (A.geglu) { // the other half of the tile's columns is up (one K piece)
#pragma unroll
                    for (int hf = 0; hf < 2; hf++) {
                        uint32_t u[16];
                        tmem_load16(col + A.BN / 2 + 16 * hf, u);
#pragma unroll
                        for (int q = 0; q < 16; q++) v[16 * hf + q] = __float_as_uint(__fmul_rn(gelu(v[16 * hf + q]), __uint_as_float(u[q])));
                    }
                }
                __syncwarp();
#pragma unroll
                for (int p = 0; p < 8; p++) sts_u4(my + lane * 128 + ((p ^ (lane & 7)) << 4), make_uint4(v[4 * p], v[4 * p + 1], v[4 * p + 2], v[4 * p + 3]));
                __syncwarp();
                const int p = lane & 7;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const int r = 4 * q + (lane >> 3), row = row0 + r;
                    const uint4 w = lds_u4(my + r * 128 + ((p ^ (r & 7)) << 4));
                    if (row >= A.T) continue; // rows of a matrix are a multiple of 32
                    float4 o = make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w));
                    if (A.geglu) {
                        *reinterpret_cast<uint2 *>(A.geglu + (size_t)row * sg.rows + sn0 + c0 + 4 * p) = make_uint2(pack_bf16x2(o.x, o.y), pack_bf16x2(o.z, o.w));
                        continue;
                    }
                    if (A.resid) {
                        const float4 r4 = load4(A.resid + (size_t)row * sg.ldc + sn0 + c0 + 4 * p, A.vec);
                        o.x += r4.x, o.y += r4.y, o.z += r4.z, o.w += r4.w;
                    }
                    store4(cbase + ((size_t)plane * A.T + row) * cld + c0 + 4 * p, o, A.ws || A.vec);
                }
            }
        }
        tc_fence_before();
    } else if (warp == kTmaWarp || warp == kCodesWarp) {
        // ================= A rows wait for the MMAs of their stage, codes, requested further ahead, for the warps that read them
        if (lane == 0) {
            const bool is_a = warp == kTmaWarp;
            const int n = is_a ? A.stages : A.code_stages, fre = is_a ? FREE : C_FREE;
            // A is what the kernel before wrote, and everything stored here waits for A; weights stand since a launch before that one at least
            if (is_a) early_wait(), step_next();
            int s = 0;
            uint32_t ph = 0;
            for (int kb = kb0; kb < kb1; kb++) {
                if (!mbar_wait_bounded(bars + fre + 8 * s, ph ^ 1u, dead)) break;
                if (is_a) {
                    if (rank == 0) mbar_expect_tx(bars + FULL + 8 * s, CTAS * A.a_tx);
                    if (PAIR) tma_load_2d_pair(ring + s * a_bytes, &maps.a, kb * BK, m0, full + 8 * s);
                    else tma_load_2d(ring + s * a_bytes, &maps.a, kb * BK, m0, full + 8 * s);
                } else {
                    const uint32_t bar = bars + C_FULL + 8 * s;
                    mbar_expect_tx(bar, c_bytes);
                    tma_load_2d(codes + s * c_bytes, &maps.w[si], kb * 2 * PB, w_row0, bar);
                }
                if (++s == n) s = 0, ph ^= 1u;
            }
            if (A.geglu && is_a) { // the MMAs have read the ring: the gelu table takes its place
                if (mbar_wait_bounded(bars + DONE, 0, dead)) {
                    mbar_expect_tx(bars + TABLE_FULL, kGeluBytes);
                    for (uint32_t o = 0; o < kGeluBytes; o += 32768)
                        bulk_load(smem0 + kGeluAt + o, reinterpret_cast<const uint8_t *>(A.gelu) + o, 32768, bars + TABLE_FULL);
                }
            }
        }
        __syncwarp();
    } else if (rank == 0) {
        // ================= MMA issuer: one wait, asked for a K block ahead, and one commit a K block
        const uint32_t idesc = umma_idesc(128 * CTAS, A.BN);
        int s = 0, chunk = 0, left = A.chunk_kb, grp = 0;
        uint32_t ph = 0;
        bool ready = false;
        for (int kb = kb0; kb < kb1; kb++) {
            const uint32_t first = left == A.chunk_kb ? 0u : 1u;
            if (!ready) mbar_wait_bounded(bars + FULL + 8 * s, ph, dead);
            tc_fence_after();
            const bool wrap = s + 1 == A.stages;
            ready = mbar_test(bars + FULL + 8 * (wrap ? 0 : s + 1), wrap ? ph ^ 1u : ph); // of a block past the last: not done
            const uint32_t a_lo = umma_desc_lo(ring + s * a_bytes, 16), b_lo = umma_desc_lo(smem0 + grp * b_bytes, 16);
            for (int mt = 0; mt < A.MT; mt++) {
                const uint32_t d = tmem + (mt * A.chunks + chunk) * A.BN;
                if (PAIR) umma_ss_pair_k4(d, a_lo + mt * (128 * 128 >> 4), b_lo, idesc, first);
                else umma_ss_k4(d, a_lo + mt * (128 * 128 >> 4), b_lo, idesc, first);
            }
            if (PAIR) umma_arrive_pair(bars + FREE + 8 * s);
            else umma_arrive(bars + FREE + 8 * s);
            if (--left == 0) chunk++, left = A.chunk_kb;
            if (++grp == A.groups) grp = 0;
            s = wrap ? 0 : s + 1;
            ph ^= wrap ? 1u : 0u;
        }
        if (PAIR) umma_arrive_pair(bars + DONE);
        else umma_arrive(bars + DONE);
    }
    __syncthreads();
    if (warp == kMmaWarp) settle(dead);
    if (PAIR) cluster_sync(); // neither leaves while the other one's MMAs or arrivals may still reach it
    if (warp == kMmaWarp) {
        tc_fence_after();
        if (PAIR) tmem_free512_pair(tmem);
        else tmem_free512(tmem);
        if (lane == 0 && *dead) *A.wait_error = 1;
    }
}

// Products that are not cut along K (the logits; gate | up of up to 256 tokens): two CTAs a tile of 256 x 256, persistent.  A tile takes half of
// tensor memory, so that four warps store one tile (or take gelu(gate) * up) while the tensor cores are on the next; sixteen others dequantise, each
// CTA its 128 of the tile's weight rows, into the stage of the ring whose other half TMA fills with A rows.
//
// What bounds it: the way of a K block through the ring (A rows from L2, codes, dequantisation, MMAs: 800 cycles a block where the MMAs take 560)
// at clocks that fall under the power limit.  Q8_0: 512 x 65536 x 2048 144 -> 123 us (1117 TFLOP/s; tiles of 512 x 256 that end before the next
// begins), gate | up of 256 tokens, 2 x 16384 x 2048, 52 -> 40 us.
constexpr int kStreamThreads = 32 * 24, kStreamStages = 5, kStreamCodes = 6, kStreamEpi = 4, kStreamDeq = 8, kStreamGroups = 4; // warps 4..7 store, 8..23 dequantise
enum { Q_FULL = 0, Q_EMPTY = 40, Q_C_FULL = 80, Q_C_FREE = 128, Q_ACC_FULL = 176, Q_ACC_FREE = 192, Q_SLOT = 208, Q_DEAD = 212 };

// gelu of an fp16 number, rounded to fp16: the numbers of the table that ggb_op_geglu_bf16 reads, computed as the table was (equal for every fp16
// number, test_gelu_of_every_fp16_number: a lookup would take shared memory's bandwidth)
__device__ __forceinline__ float gelu_f16(float g) {
    const float x = __half2float(__float2half_rn(g));
    const float inner = __fmul_rn(__fmul_rn(0.79788456080286535587989211986876f, x), __fadd_rn(1.0f, __fmul_rn(__fmul_rn(0.044715f, x), x)));
    return __half2float(__float2half_rn(__fmul_rn(__fmul_rn(0.5f, x), __fadd_rn(1.0f, tanhf(inner)))));
}

template <int TYPE, bool GEGLU>
__global__ void __launch_bounds__(kStreamThreads, 1) gemm_quant_stream_kernel(const __grid_constant__ GemmMaps maps, const GemmArgs A) {
    extern __shared__ uint8_t gemm_smem_raw[];
    constexpr int PB = TYPE == GGB_TYPE_Q8_0 ? 32 : 16; // payload bytes of a block of 32 weights
    constexpr uint32_t kHalf = 128 * 128, kStage = 2 * kHalf, kCodes = 128 * 2 * PB;
    const uint32_t raw0 = smem_u32(gemm_smem_raw), smem0 = (raw0 + 1023u) & ~1023u, bars = smem0 + kRing;
    const uint32_t codes = smem0 + kStreamStages * kStage, turn = codes + kStreamCodes * 8192;
    uint8_t *ctl = gemm_smem_raw + (bars - raw0);
    volatile int *dead = reinterpret_cast<volatile int *>(ctl + Q_DEAD);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int rank = (int)cluster_rank();
    const uint32_t bars0 = cluster_addr(bars, 0);
    if (tid == 0) {
        for (int s = 0; s < kStreamStages; s++) {
            mbar_init(bars + Q_FULL + 8 * s, 1 + 2 * 4); // the bytes of A and the warps that dequantise, of both CTAs
            mbar_init(bars + Q_EMPTY + 8 * s, 1);
        }
        for (int s = 0; s < kStreamCodes; s++) {
            mbar_init(bars + Q_C_FULL + 8 * s, 1);
            mbar_init(bars + Q_C_FREE + 8 * s, 4);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(bars + Q_ACC_FULL + 8 * s, 1);
            mbar_init(bars + Q_ACC_FREE + 8 * s, 8);
        }
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 3) tmem_alloc512_pair(bars + Q_SLOT);
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<uint32_t *>(ctl + Q_SLOT), 0);

    const int pairs = gridDim.x / 2, me = blockIdx.x / 2, m_tiles = (A.T + 255) / 256, total = m_tiles * ((A.N + 255) / 256), kblocks = A.kblocks;
    struct place {
        int m0, si, sn0, w_row0; // first row of A of the pair, matrix, first output column and first weight row of this CTA inside it
    };
    auto locate = [&](int t) { // row tiles first: those that share a piece of W run together
        place r;
        r.m0 = t % m_tiles * 256;
        const int n0 = t / m_tiles * 256;
        r.si = 0;
        if (GEGLU) r.si = rank;
        else if (A.n_seg > 1 && n0 >= A.seg[1].n_begin) r.si = (A.n_seg > 2 && n0 >= A.seg[2].n_begin) ? 2 : 1;
        r.sn0 = GEGLU ? n0 / 2 : n0 - A.seg[r.si].n_begin;
        r.w_row0 = GEGLU ? r.sn0 : r.sn0 + rank * 128;
        return r;
    };

    if (warp == 0 || warp == 2) {
        if (lane == 0) { // warp 0: A rows, counted on the first CTA's barrier; warp 2: codes
            const bool is_a = warp == 0;
            const int n = is_a ? kStreamStages : kStreamCodes, fre = is_a ? Q_EMPTY : Q_C_FREE;
            int s = 0;
            uint32_t ph = 0;
            if (is_a) early_wait(), step_next(); // as gemm_quant_kernel
            for (int t = me; t < total; t += pairs) {
                const place at = locate(t);
                for (int kb = 0; kb < kblocks; kb++) {
                    if (!mbar_wait_bounded(bars + fre + 8 * s, ph ^ 1u, dead)) break;
                    if (is_a) {
                        if (rank == 0) mbar_expect_tx(bars + Q_FULL + 8 * s, 2 * kHalf);
                        tma_load_2d_pair(smem0 + s * kStage, &maps.a, kb * BK, at.m0 + rank * 128, bars0 + Q_FULL + 8 * s);
                    } else {
                        mbar_expect_tx(bars + Q_C_FULL + 8 * s, kCodes);
                        tma_load_2d(codes + s * kCodes, &maps.w[at.si], kb * 2 * PB, at.w_row0, bars + Q_C_FULL + 8 * s);
                    }
                    if (++s == n) s = 0, ph ^= 1u;
                }
            }
        }
        __syncwarp();
    } else if (warp == 1 && rank == 0) {
        const uint32_t idesc = umma_idesc(256, 256);
        int s = 0, it = 0;
        uint32_t ph = 0;
        bool ready = false; // asked for a K block ahead
        for (int t = me; t < total; t += pairs, it++) {
            const int buf = it & 1;
            mbar_wait_bounded(bars + Q_ACC_FREE + 8 * buf, ((it >> 1) & 1) ^ 1, dead);
            for (int kb = 0; kb < kblocks; kb++) {
                if (!ready) mbar_wait_bounded(bars + Q_FULL + 8 * s, ph, dead);
                tc_fence_after();
                const uint32_t at = smem0 + s * kStage;
                if (++s == kStreamStages) s = 0, ph ^= 1u;
                ready = mbar_test(bars + Q_FULL + 8 * s, ph);
                umma_ss_pair_k4(tmem + buf * 256, umma_desc_lo(at, 16), umma_desc_lo(at + kHalf, 16), idesc, kb > 0);
                umma_arrive_pair(bars + Q_EMPTY + (at - smem0) / kStage * 8);
            }
            umma_arrive_pair(bars + Q_ACC_FULL + 8 * buf);
        }
    } else if (warp >= kStreamDeq) {
        // Four groups of four warps take the K blocks of all tiles in turn: a block is 1400 to 2000 cycles in the hands of one, mostly latency, and
        // the MMAs want one every 560.  A thread owns a row of the CTA's 128: 64 weights, two scales.  It takes the four pieces of 16 codes in
        // the order q ^ turn, in which eight neighbouring rows meet eight groups of banks, where the codes lie (64 bytes a row) and where the
        // weights go (the 128-byte swizzle): turn = w * (r >> 1) in the field of four elements, whose w and 1 + w both have inverses.
        const int grp = (warp - kStreamDeq) >> 2, wr = tid & 127, r2 = (wr >> 2) & 1, r1 = (wr >> 1) & 1, turn_of = ((r2 ^ r1) << 1) | r2;
        const float bias = TYPE == GGB_TYPE_Q8_0 ? 32896.f : 32776.f;
        int ft = me, fkb = grp; // whose scales are asked for next: four of the group's blocks ahead
        const __half *dp = nullptr;
        auto row_of = [&]() { // rows past the matrix: zero codes (TMA), any scale
            const place at = locate(ft);
            dp = A.seg[at.si].d + (size_t)min(at.w_row0 + wr, A.seg[at.si].rows - 1) * A.nb;
        };
        auto ask = [&]() {
            if (fkb >= kblocks || !dp) {
                while (fkb >= kblocks) fkb -= kblocks, ft += pairs;
                if (ft < total) row_of();
            }
            const __half2 d = ft < total ? __ldg(reinterpret_cast<const __half2 *>(dp + 2 * fkb)) : __float2half2_rn(0.f);
            fkb += kStreamGroups;
            return d;
        };
        __half2 sc[4];
#pragma unroll
        for (int u = 0; u < 4; u++) sc[u] = ask();
        const int n_blocks = (total - me + pairs - 1) / pairs * kblocks;
        int s = grp, cs = grp;
        uint32_t ph = 0, cph = 0;
        for (int b0 = grp; b0 < n_blocks; b0 += 4 * kStreamGroups) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (b0 + kStreamGroups * u >= n_blocks) break;
                const float2 d = __half22float2(sc[u]);
                sc[u] = ask();
                const block_scale d0(d.x, bias), d1(d.y, bias);
                mbar_wait_warp(bars + Q_C_FULL + 8 * cs, cph, dead);
                const uint32_t src = codes + cs * kCodes + wr * 2 * PB, dst = smem0 + s * kStage + kHalf + wr * 128;
                uint4 x[4];
                if (TYPE == GGB_TYPE_Q8_0) {
#pragma unroll
                    for (int q = 0; q < 4; q++) x[q] = lds_u4(src + 16 * (q ^ turn_of));
                } else { // 32 bytes a row: the two pieces in an order in which eight rows meet eight groups of banks; low nibbles, then high ones
                    x[0] = lds_u4(src + 16 * r2), x[1] = lds_u4(src + 16 * (r2 ^ 1));
                }
                mbar_wait_warp(bars + Q_EMPTY + 8 * s, ph ^ 1u, dead);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int p = q ^ turn_of;
                    uint32_t c[4], o[8];
                    block_scale b = d0;
                    if (p >> 1) b = d1;
                    if (TYPE == GGB_TYPE_Q8_0) {
                        const uint4 w = x[q];
                        c[0] = w.x ^ 0x80808080u, c[1] = w.y ^ 0x80808080u, c[2] = w.z ^ 0x80808080u, c[3] = w.w ^ 0x80808080u;
                    } else {
                        const uint4 w = (p >> 1) == r2 ? x[0] : x[1];
                        const int sh = (p & 1) * 4;
                        c[0] = (w.x >> sh) & 0x0F0F0F0Fu, c[1] = (w.y >> sh) & 0x0F0F0F0Fu, c[2] = (w.z >> sh) & 0x0F0F0F0Fu, c[3] = (w.w >> sh) & 0x0F0F0F0Fu;
                    }
                    codes_to_bf16x16(c, b, o);
                    sts_u4(dst + (((2 * p) ^ (wr & 7)) << 4), make_uint4(o[0], o[1], o[2], o[3]));
                    sts_u4(dst + (((2 * p + 1) ^ (wr & 7)) << 4), make_uint4(o[4], o[5], o[6], o[7]));
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(bars + Q_C_FREE + 8 * cs);
                    mbar_arrive_cluster(bars0 + Q_FULL + 8 * s);
                }
                s += kStreamGroups;
                if (s >= kStreamStages) s -= kStreamStages, ph ^= 1u;
                cs += kStreamGroups;
                if (cs >= kStreamCodes) cs -= kStreamCodes, cph ^= 1u;
            }
        }
    } else if (warp >= kStreamEpi) {
        const int lq = warp & 3, p = lane & 7;
        const uint32_t my = turn + lq * 4096;
        int it = 0;
        for (int t = me; t < total; t += pairs, it++) {
            const place at = locate(t);
            const GemmSeg &sg = A.seg[at.si];
            const int buf = it & 1, row0 = at.m0 + rank * 128 + lq * 32;
            mbar_wait_warp(bars + Q_ACC_FULL + 8 * buf, (it >> 1) & 1, dead);
            tc_fence_after();
            if (row0 < A.T)
                for (int c0 = 0; c0 < (GEGLU ? 128 : 256) && at.sn0 + c0 < sg.rows; c0 += 32) {
                    const uint32_t col = tmem + ((uint32_t)(lq * 32) << 16) + buf * 256 + c0;
                    uint32_t v[32];
                    tmem_load32(col, v);
                    if (GEGLU) { // the other half of the tile's columns is up
#pragma unroll
                        for (int hf = 0; hf < 2; hf++) {
                            uint32_t u[16];
                            tmem_load16(col + 128 + 16 * hf, u);
#pragma unroll
                            for (int q = 0; q < 16; q++) v[16 * hf + q] = __float_as_uint(__fmul_rn(gelu_f16(__uint_as_float(v[16 * hf + q])), __uint_as_float(u[q])));
                        }
                    }
                    // row = lane -> eight lanes a row: 16-byte piece p of row r at place p ^ (r & 7)
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < 8; q++) sts_u4(my + lane * 128 + ((q ^ (lane & 7)) << 4), make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const int r = 4 * q + (lane >> 3), row = row0 + r;
                        const uint4 w = lds_u4(my + r * 128 + ((p ^ (r & 7)) << 4));
                        if (row >= A.T) continue; // rows of a matrix are a multiple of 32
                        float4 o = make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w));
                        const int n = at.sn0 + c0 + 4 * p;
                        if (GEGLU) {
                            *reinterpret_cast<uint2 *>(A.geglu + (size_t)row * sg.rows + n) = make_uint2(pack_bf16x2(o.x, o.y), pack_bf16x2(o.z, o.w));
                            continue;
                        }
                        if (A.resid) {
                            const float4 r4 = load4(A.resid + (size_t)row * sg.ldc + n, A.vec);
                            o.x += r4.x, o.y += r4.y, o.z += r4.z, o.w += r4.w;
                        }
                        store4(sg.c + (size_t)row * sg.ldc + n, o, A.vec);
                    }
                }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(bars0 + Q_ACC_FREE + 8 * buf);
        }
    }
    __syncthreads();
    if (warp == 3) settle(dead);
    cluster_sync(); // neither leaves while the other one's MMAs or arrivals may still reach it
    if (warp == 3) {
        tc_fence_after();
        tmem_free512_pair(tmem);
        if (lane == 0 && *dead) *A.wait_error = 1;
    }
}

// the pieces of a product that several CTAs summed along K, in order (+ residual)
__global__ void splitk_reduce_kernel(const GemmArgs A, int pieces) {
    step_wait();
    step_next();
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4, T = A.T, N = A.N; // N and the segments: multiples of 32
    if (i >= T * N) return;
    const int64_t t = i / N;
    const int n = (int)(i - t * N);
    int si = 0;
    if (A.n_seg > 1 && n >= A.seg[1].n_begin) si = (A.n_seg > 2 && n >= A.seg[2].n_begin) ? 2 : 1;
    const GemmSeg &sg = A.seg[si];
    const int col = n - sg.n_begin;
    if (col >= sg.rows) return; // tile padding between segments
    float4 acc = *reinterpret_cast<const float4 *>(A.ws + i);
    auto add = [&](const float *p, int vec) {
        const float4 v = load4(p, vec);
        acc.x += v.x, acc.y += v.y, acc.z += v.z, acc.w += v.w;
    };
    for (int s = 1; s < pieces; s++) add(A.ws + (int64_t)s * T * N + i, 1);
    if (A.resid) add(A.resid + t * sg.ldc + col, A.vec);
    store4(sg.c + t * sg.ldc + col, acc, A.vec);
}

// rms_norm * w -> bf16 (the A operand of the next GEMM): same double-sum order as rms_norm_kernel (elementwise.cu)
__global__ void __launch_bounds__(GGB_DEV_NORM_THREADS)
rms_norm_bf16_kernel(const float *x, const float *w, float eps, int64_t E, __nv_bfloat16 *y) {
    __shared__ double s_w[GGB_DEV_NORM_THREADS / 32];
    step_wait();
    step_next();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float *xr = x + (int64_t)blockIdx.x * E;
    double acc = 0.0;
    for (int64_t i = tid; i < E; i += GGB_DEV_NORM_THREADS) {
        const float v = xr[i];
        acc = __dadd_rn(acc, (double)__fmul_rn(v, v));
    }
    acc = warp_sum_f64(acc);
    if (lane == 0) s_w[warp] = acc;
    __syncthreads();
    double sum = s_w[0];
#pragma unroll
    for (int i = 1; i < GGB_DEV_NORM_THREADS / 32; i++) sum = __dadd_rn(sum, s_w[i]);
    const float mean = __double2float_rn(__ddiv_rn(sum, (double)E));
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, eps)));
    for (int64_t i = tid; i < E; i += GGB_DEV_NORM_THREADS)
        y[(int64_t)blockIdx.x * E + i] = __float2bfloat16_rn(__fmul_rn(__fmul_rn(xr[i], scale), w[i]));
}

// What follows a product that several CTAs summed along K, with the adding of its pieces: the sums as splitk_reduce_kernel takes them, then the
// arithmetic of the kernel that would read them, to the bit, without a launch and a pass over memory between.  512 x 2048 in 8 pieces: 10.2 + 4.9 us
// for sums and norm, 12.8 us; 512 x 2560 in 4 pieces: 8 + 6.5 us for sums and rotation, 11.8 us (all cold).  Bound by reading the pieces.
__device__ __forceinline__ float pieces_sum(const float *ws, int64_t plane, int pieces) {
    float v[8], s;
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = i < pieces ? ws[i * plane] : 0.f;
    s = v[0];
#pragma unroll
    for (int i = 1; i < 8; i++)
        if (i < pieces) s += v[i];
    return s;
}

// c = pieces (+ residual); y = rms_norm(c) * w in bf16 (rms_norm_bf16_kernel)
__global__ void __launch_bounds__(GGB_DEV_NORM_THREADS) splitk_norm_kernel(const GemmArgs A, int pieces, const float *w, float eps, __nv_bfloat16 *y) {
    __shared__ double s_w[GGB_DEV_NORM_THREADS / 32];
    extern __shared__ float s_row[];
    step_wait();
    step_next();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, E = A.N;
    const int64_t t = blockIdx.x, plane = (int64_t)A.T * E;
    const GemmSeg &sg = A.seg[0];
    double acc = 0.0;
#pragma unroll 2
    for (int i = tid; i < E; i += GGB_DEV_NORM_THREADS) {
        float v = pieces_sum(A.ws + t * E + i, plane, pieces);
        if (A.resid) v += A.resid[t * sg.ldc + i];
        sg.c[t * sg.ldc + i] = v;
        s_row[i] = v;
        acc = __dadd_rn(acc, (double)__fmul_rn(v, v));
    }
    acc = warp_sum_f64(acc);
    if (lane == 0) s_w[warp] = acc;
    __syncthreads();
    double sum = s_w[0];
#pragma unroll
    for (int i = 1; i < GGB_DEV_NORM_THREADS / 32; i++) sum = __dadd_rn(sum, s_w[i]);
    const float mean = __double2float_rn(__ddiv_rn(sum, (double)E));
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, eps)));
    for (int i = tid; i < E; i += GGB_DEV_NORM_THREADS) y[t * E + i] = __float2bfloat16_rn(__fmul_rn(__fmul_rn(s_row[i], scale), w[i]));
}

// q | k | v: the rotation of q (times q_scale, to seg[0].c) and k, k and v to the cache (rope_kv_store_batch_kernel)
struct rope_args {
    const int32_t *pos;
    int H, Hkv, d, table_ctx;
    float q_scale;
    const float *cosT, *sinT;
    __half *kcache, *vcache;
};
__global__ void splitk_rope_kernel(const GemmArgs A, int pieces, const rope_args r) {
    step_wait();
    step_next();
    const int half = r.d / 2, nq = r.H * half, nk = r.Hkv * half, nv = r.Hkv * r.d, idx = blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t t = blockIdx.y, plane = (int64_t)A.T * A.N;
    int pos = r.pos[t];
    pos = pos < 0 ? 0 : (pos >= r.table_ctx ? r.table_ctx - 1 : pos);
    const float *row = A.ws + t * A.N;
    if (idx < nq + nk) {
        const bool is_q = idx < nq;
        const int j = is_q ? idx : idx - nq, h = j / half, i = j % half;
        const float c = r.cosT[(int64_t)pos * half + i], s = r.sinT[(int64_t)pos * half + i];
        const float *src = row + A.seg[is_q ? 0 : 1].n_begin + h * r.d + i;
        const float x0 = pieces_sum(src, plane, pieces), x1 = pieces_sum(src + half, plane, pieces);
        const float r0 = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s)), r1 = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
        if (is_q) {
            float *qt = A.seg[0].c + t * A.seg[0].ldc + h * r.d + i;
            qt[0] = __fmul_rn(r0, r.q_scale);
            qt[half] = __fmul_rn(r1, r.q_scale);
        } else {
            __half *kr = r.kcache + (int64_t)pos * r.Hkv * r.d + h * r.d + i;
            kr[0] = __float2half_rn(r0);
            kr[half] = __float2half_rn(r1);
        }
    } else if (idx < nq + nk + nv) {
        const int j = idx - nq - nk;
        r.vcache[(int64_t)pos * r.Hkv * r.d + j] = __float2half_rn(pieces_sum(row + A.seg[2].n_begin + j, plane, pieces));
    }
}

// gelu(gate) * up -> bf16 (fp16 gelu table like the reference's ggml_gelu; ref: src/gemma_model.cpp:448-449)
__global__ void geglu_bf16_kernel(const float *gate, const float *up, int64_t n, const uint16_t *__restrict__ table,
                                  __nv_bfloat16 *y) {
    // four elements per thread: 128-bit loads of gate / up, four table lookups in flight, one 64-bit store
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i + 3 < n) {
        const float4 g = *reinterpret_cast<const float4 *>(gate + i), u = *reinterpret_cast<const float4 *>(up + i);
        const uint16_t t0 = table[float_to_half_bits(g.x)], t1 = table[float_to_half_bits(g.y)];
        const uint16_t t2 = table[float_to_half_bits(g.z)], t3 = table[float_to_half_bits(g.w)];
        __nv_bfloat162 lo = __floats2bfloat162_rn(__fmul_rn(half_bits_to_float(t0), u.x), __fmul_rn(half_bits_to_float(t1), u.y));
        __nv_bfloat162 hi = __floats2bfloat162_rn(__fmul_rn(half_bits_to_float(t2), u.z), __fmul_rn(half_bits_to_float(t3), u.w));
        uint2 o;
        o.x = *reinterpret_cast<uint32_t *>(&lo);
        o.y = *reinterpret_cast<uint32_t *>(&hi);
        *reinterpret_cast<uint2 *>(y + i) = o;
    } else {
        for (int64_t j = i; j < n; j++) y[j] = __float2bfloat16_rn(__fmul_rn(half_bits_to_float(table[float_to_half_bits(gate[j])]), up[j]));
    }
}

__global__ void cvt_f32_bf16_kernel(const float *x, int64_t n, __nv_bfloat16 *y) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __float2bfloat16_rn(x[i]);
}

// Causal attention of T query tokens at positions pos0 .. pos0+T-1 over the fp16 KV cache (position-major
// [n_ctx][Hkv*d]).  One warp per (token, GH query heads that share a KV head), the reference's node order
// (ref: src/gemma_model.cpp:454-489): kq = K . f16(q) (fp32 accumulate), soft_max_ext with the fp16 exp table and
// a double sum, P rounded to fp16, kqv = V^T . P.  q is already roped and scaled.  A K / V row is loaded once for
// the GH heads, and the 8 lane partials of a step (8 / GH positions x GH heads) are reduced with ONE folded
// butterfly (9 shuffles instead of 40; the same additions as the plain xor-butterfly).  CUDA cores.
constexpr int kAttnWarps = 4;
template <int GH>
__global__ void __launch_bounds__(kAttnWarps * 32)
attn_prefill_kernel(const float *__restrict__ q, const __half *__restrict__ kc, const __half *__restrict__ vc, int T,
                    int pos0, int H, int Hkv, int d, const uint16_t *__restrict__ exp_table, float *__restrict__ out,
                    __nv_bfloat16 *__restrict__ out_bf16, int n_kv_max) {
    constexpr int NP = 8 / GH; // positions per step
    extern __shared__ float attn_s[]; // [kAttnWarps][GH][n_kv_max]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int HG = H / GH; // head groups per token
    const int item = blockIdx.x * kAttnWarps + warp;
    if (item >= T * HG) return;
    const int t = item / HG, h0 = (item % HG) * GH, g = h0 / (H / Hkv);
    const int n_kv = pos0 + t + 1;
    float *s = attn_s + (size_t)warp * GH * n_kv_max;
    const size_t stride = (size_t)Hkv * d;
    const bool in = 8 * lane < d;
    float qf[GH][8];
#pragma unroll
    for (int u = 0; u < GH; u++)
#pragma unroll
        for (int e = 0; e < 8; e++)
            qf[u][e] = in ? __half2float(__float2half_rn(q[((size_t)t * H + h0 + u) * d + 8 * lane + e])) : 0.f;
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    // after the fold a lane holds value index 4 b4 + 2 b3 + b2 of the step: value = position * GH + head
    const int vi = (b4 ? 4 : 0) + (b3 ? 2 : 0) + (b2 ? 1 : 0);
    const int my_p = vi / GH, my_u = vi % GH;
    float mx = -INFINITY; // of head my_u over the positions this lane sees
    for (int j0 = 0; j0 < n_kv; j0 += NP) {
        float v[8];
#pragma unroll
        for (int p = 0; p < NP; p++) {
            uint4 raw = make_uint4(0, 0, 0, 0);
            if (in && j0 + p < n_kv) raw = *reinterpret_cast<const uint4 *>(kc + (size_t)(j0 + p) * stride + (size_t)g * d + 8 * lane);
            const __half2 *h2 = reinterpret_cast<const __half2 *>(&raw);
            float kf[8];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float2 f = __half22float2(h2[e]);
                kf[2 * e] = f.x;
                kf[2 * e + 1] = f.y;
            }
#pragma unroll
            for (int u = 0; u < GH; u++) {
                float acc = 0.f;
#pragma unroll
                for (int e = 0; e < 8; e++) acc = fmaf(kf[e], qf[u][e], acc);
                v[p * GH + u] = acc;
            }
        }
        float k4[4], k2[2];
#pragma unroll
        for (int i = 0; i < 4; i++) k4[i] = (b4 ? v[4 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, b4 ? v[i] : v[4 + i], 16);
#pragma unroll
        for (int i = 0; i < 2; i++) k2[i] = (b3 ? k4[2 + i] : k4[i]) + __shfl_xor_sync(0xffffffffu, b3 ? k4[i] : k4[2 + i], 8);
        float k1 = (b2 ? k2[1] : k2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? k2[0] : k2[1], 4);
        k1 += __shfl_xor_sync(0xffffffffu, k1, 2);
        k1 += __shfl_xor_sync(0xffffffffu, k1, 1);
        if (j0 + my_p < n_kv) {
            if ((lane & 3) == 0) s[(size_t)my_u * n_kv_max + j0 + my_p] = k1;
            mx = fmaxf(mx, k1);
        }
    }
    // the maximum of every head: lanes with the same head index hold its positions' maxima
    float mxu[GH];
#pragma unroll
    for (int u = 0; u < GH; u++) mxu[u] = warp_max_f32(my_u == u ? mx : -INFINITY);
    __syncwarp();
    float inv[GH];
#pragma unroll
    for (int u = 0; u < GH; u++) {
        float *su = s + (size_t)u * n_kv_max;
        double sum = 0.0;
        for (int j = lane; j < n_kv; j += 32) {
            const float e = half_bits_to_float(exp_table[float_to_half_bits(su[j] - mxu[u])]);
            su[j] = e;
            sum += (double)e;
        }
        sum = warp_sum_f64(sum);
        inv[u] = (float)(1.0 / sum);
    }
    __syncwarp();
    float o[GH][8];
#pragma unroll
    for (int u = 0; u < GH; u++)
#pragma unroll
        for (int e = 0; e < 8; e++) o[u][e] = 0.f;
    for (int j = 0; j < n_kv; j++) { // (unrolling this loop by 8 measured slower: 3.1 vs 2.5 ms per prefill)
        float vf[8];
        if (in) {
            const uint4 raw = *reinterpret_cast<const uint4 *>(vc + (size_t)j * stride + (size_t)g * d + 8 * lane);
            const __half2 *h2 = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float2 f = __half22float2(h2[e]);
                vf[2 * e] = f.x;
                vf[2 * e + 1] = f.y;
            }
        }
#pragma unroll
        for (int u = 0; u < GH; u++) {
            const float p = __half2float(__float2half_rn(s[(size_t)u * n_kv_max + j] * inv[u])); // ggml converts P to fp16 for the V mat-mul
            if (in) {
#pragma unroll
                for (int e = 0; e < 8; e++) o[u][e] = fmaf(vf[e], p, o[u][e]);
            }
        }
    }
    if (in) {
#pragma unroll
        for (int u = 0; u < GH; u++) {
            const size_t at = ((size_t)t * H + h0 + u) * d + 8 * lane;
            if (out) {
#pragma unroll
                for (int e = 0; e < 8; e++) out[at + e] = o[u][e];
            }
            if (out_bf16) { // the o-projection's A operand, rounded exactly as ggb_op_cvt_f32_bf16 would
                uint4 pk;
                __nv_bfloat162 p0 = __floats2bfloat162_rn(o[u][0], o[u][1]), p1 = __floats2bfloat162_rn(o[u][2], o[u][3]);
                __nv_bfloat162 p2 = __floats2bfloat162_rn(o[u][4], o[u][5]), p3 = __floats2bfloat162_rn(o[u][6], o[u][7]);
                pk.x = *reinterpret_cast<uint32_t *>(&p0); pk.y = *reinterpret_cast<uint32_t *>(&p1);
                pk.z = *reinterpret_cast<uint32_t *>(&p2); pk.w = *reinterpret_cast<uint32_t *>(&p3);
                *reinterpret_cast<uint4 *>(out_bf16 + at) = pk;
            }
        }
    }
}

} // namespace

// The MQA / GQA form: ONE CTA (4 warps) per (token, 4 query heads of one KV head).  The attention above is bound by
// L2 bandwidth (every warp re-reads the K / V rows: 1 GB per layer at T = 512); here a K / V row is loaded once for the
// 4 heads and the positions are dealt to the 4 warps, so the traffic drops 4x at the same number of warps.  Scores:
// 2 positions x 4 heads per folded butterfly; max / sum / P.V partials are combined across the warps in shared memory.
__global__ void __launch_bounds__(128)
attn_prefill_gqa_kernel(const float *__restrict__ q, const __half *__restrict__ kc, const __half *__restrict__ vc, int T,
                        int pos0, int H, int Hkv, int d, const uint16_t *__restrict__ exp_table, float *__restrict__ out,
                        __nv_bfloat16 *__restrict__ out_bf16, int n_kv_max) {
    constexpr int GH = 4, NW = 4;
    extern __shared__ float attn_s[]; // s[GH][n_kv_max] | red[NW][GH][256] | wmax[NW][GH] | wsum double[NW][GH]
    float *s = attn_s;
    float *red = attn_s + (size_t)GH * n_kv_max;
    float *wmax = red + NW * GH * 256;
    double *wsum = reinterpret_cast<double *>(wmax + NW * GH);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const int HG = H / GH;
    const int t = blockIdx.x / HG, h0 = (blockIdx.x % HG) * GH, g = h0 / (H / Hkv);
    const int n_kv = pos0 + t + 1;
    const size_t stride = (size_t)Hkv * d;
    const bool in = 8 * lane < d;
    float qf[GH][8];
#pragma unroll
    for (int u = 0; u < GH; u++)
#pragma unroll
        for (int e = 0; e < 8; e++)
            qf[u][e] = in ? __half2float(__float2half_rn(q[((size_t)t * H + h0 + u) * d + 8 * lane + e])) : 0.f;
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    const int my_p = b4 ? 1 : 0, my_u = (b3 ? 2 : 0) + (b2 ? 1 : 0); // value index = position * GH + head
    float mx = -INFINITY;
    for (int j0 = 2 * warp; j0 < n_kv; j0 += 2 * NW) {
        float v[8];
#pragma unroll
        for (int p = 0; p < 2; p++) {
            uint4 raw = make_uint4(0, 0, 0, 0);
            if (in && j0 + p < n_kv) raw = *reinterpret_cast<const uint4 *>(kc + (size_t)(j0 + p) * stride + (size_t)g * d + 8 * lane);
            const __half2 *h2 = reinterpret_cast<const __half2 *>(&raw);
            float kf[8];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float2 f = __half22float2(h2[e]);
                kf[2 * e] = f.x;
                kf[2 * e + 1] = f.y;
            }
#pragma unroll
            for (int u = 0; u < GH; u++) {
                float acc = 0.f;
#pragma unroll
                for (int e = 0; e < 8; e++) acc = fmaf(kf[e], qf[u][e], acc);
                v[p * GH + u] = acc;
            }
        }
        float k4[4], k2[2];
#pragma unroll
        for (int i = 0; i < 4; i++) k4[i] = (b4 ? v[4 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, b4 ? v[i] : v[4 + i], 16);
#pragma unroll
        for (int i = 0; i < 2; i++) k2[i] = (b3 ? k4[2 + i] : k4[i]) + __shfl_xor_sync(0xffffffffu, b3 ? k4[i] : k4[2 + i], 8);
        float k1 = (b2 ? k2[1] : k2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? k2[0] : k2[1], 4);
        k1 += __shfl_xor_sync(0xffffffffu, k1, 2);
        k1 += __shfl_xor_sync(0xffffffffu, k1, 1);
        if (j0 + my_p < n_kv) {
            if ((lane & 3) == 0) s[(size_t)my_u * n_kv_max + j0 + my_p] = k1;
            mx = fmaxf(mx, k1);
        }
    }
#pragma unroll
    for (int u = 0; u < GH; u++) {
        const float m = warp_max_f32(my_u == u ? mx : -INFINITY);
        if (lane == 0) wmax[warp * GH + u] = m;
    }
    __syncthreads();
    float inv[GH];
#pragma unroll
    for (int u = 0; u < GH; u++) {
        const float m = fmaxf(fmaxf(wmax[u], wmax[GH + u]), fmaxf(wmax[2 * GH + u], wmax[3 * GH + u]));
        float *su = s + (size_t)u * n_kv_max;
        double sum = 0.0;
        for (int j = tid; j < n_kv; j += 128) {
            const float e = half_bits_to_float(exp_table[float_to_half_bits(su[j] - m)]);
            su[j] = e;
            sum += (double)e;
        }
        sum = warp_sum_f64(sum);
        if (lane == 0) wsum[warp * GH + u] = sum;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < GH; u++) inv[u] = (float)(1.0 / (wsum[u] + wsum[GH + u] + wsum[2 * GH + u] + wsum[3 * GH + u]));
    float o[GH][8];
#pragma unroll
    for (int u = 0; u < GH; u++)
#pragma unroll
        for (int e = 0; e < 8; e++) o[u][e] = 0.f;
    for (int j = warp; j < n_kv; j += NW) {
        float vf[8];
        if (in) {
            const uint4 raw = *reinterpret_cast<const uint4 *>(vc + (size_t)j * stride + (size_t)g * d + 8 * lane);
            const __half2 *h2 = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float2 f = __half22float2(h2[e]);
                vf[2 * e] = f.x;
                vf[2 * e + 1] = f.y;
            }
        }
#pragma unroll
        for (int u = 0; u < GH; u++) {
            const float p = __half2float(__float2half_rn(s[(size_t)u * n_kv_max + j] * inv[u])); // P as fp16, like ggml
            if (in) {
#pragma unroll
                for (int e = 0; e < 8; e++) o[u][e] = fmaf(vf[e], p, o[u][e]);
            }
        }
    }
    if (in) {
#pragma unroll
        for (int u = 0; u < GH; u++)
#pragma unroll
            for (int e = 0; e < 8; e++) red[(warp * GH + u) * 256 + 8 * lane + e] = o[u][e];
    }
    __syncthreads();
    if (in) { // warp w finishes head h0 + w: the four warps' partial rows in warp order
        float r[8];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const int c = 8 * lane + e;
            r[e] = ((red[(0 * GH + warp) * 256 + c] + red[(1 * GH + warp) * 256 + c]) + red[(2 * GH + warp) * 256 + c]) +
                   red[(3 * GH + warp) * 256 + c];
        }
        const size_t at = ((size_t)t * H + h0 + warp) * d + 8 * lane;
        if (out) {
#pragma unroll
            for (int e = 0; e < 8; e++) out[at + e] = r[e];
        }
        if (out_bf16) {
            uint4 pk;
            __nv_bfloat162 p0 = __floats2bfloat162_rn(r[0], r[1]), p1 = __floats2bfloat162_rn(r[2], r[3]);
            __nv_bfloat162 p2 = __floats2bfloat162_rn(r[4], r[5]), p3 = __floats2bfloat162_rn(r[6], r[7]);
            pk.x = *reinterpret_cast<uint32_t *>(&p0); pk.y = *reinterpret_cast<uint32_t *>(&p1);
            pk.z = *reinterpret_cast<uint32_t *>(&p2); pk.w = *reinterpret_cast<uint32_t *>(&p3);
            *reinterpret_cast<uint4 *>(out_bf16 + at) = pk;
        }
    }
}

extern "C" {

size_t ggb_gemm_workspace_bytes(int64_t T, int64_t N, int64_t K) {
    (void)K;
    return (size_t)8 * (size_t)T * (size_t)N * 4; // up to 8 K-splits
}

// until every SM has a piece of a 256 x 256 tile
int ggb_gemm_pieces(int64_t T, int64_t N, int64_t K) {
    const int64_t big = (N + 255) / 256 * ((T + 255) / 256), sms = ggb_sm_count(), kblocks = K / BK;
    int pieces = 1;
    while (pieces < 8 && big * pieces * 2 <= sms && kblocks / (pieces * 2) >= 4) pieces *= 2;
    return pieces;
}

int ggb_op_cvt_f32_bf16(const float *x, int64_t n, void *y_bf16) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(x && y_bf16 && n > 0, "bad cvt args");
    cvt_f32_bf16_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ggb_cuda_stream()>>>(x, n, (__nv_bfloat16 *)y_bf16);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_op_rms_norm_bf16(const float *x, const float *w, float eps, int64_t E, int64_t T, void *y_bf16) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(x && w && y_bf16 && E > 0 && T > 0, "bad rms_norm_bf16 args");
    GGB_CUDA(ggb_launch_step(rms_norm_bf16_kernel, dim3((unsigned)T), dim3(GGB_DEV_NORM_THREADS), 0, x, w, eps, E, (__nv_bfloat16 *)y_bf16));
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int ggb_op_geglu_bf16(const float *gate, const float *up, int64_t n, void *y_bf16) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(gate && up && y_bf16 && n > 0, "bad geglu_bf16 args");
    geglu_bf16_kernel<<<(unsigned)((n + 1023) / 1024), 256, 0, ggb_cuda_stream()>>>(gate, up, n, ggb_gelu_table_dev(), (__nv_bfloat16 *)y_bf16);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

// what the sums of a split product go through; `done` says that they did (a product that is not split leaves it to its caller)
struct gemm_tail {
    const float *norm_w = nullptr;
    float eps = 0.f;
    __nv_bfloat16 *y = nullptr;
    const rope_args *rope = nullptr;
    bool done = false;
};

static int gemm_launch(int n, const ggb_weight *const *w, const void *a_bf16, int64_t T, float *const *c, const int64_t *ldc,
                       const float *resid, void *workspace, size_t workspace_bytes, void *geglu = nullptr, gemm_tail *tail = nullptr) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(n >= 1 && n <= kMaxSegs && w && a_bf16 && c && ldc && T > 0, "bad gemm args");
    GGB_CHECK_ARG(n == 1 || !resid, "gemm: a residual needs a single matrix");
    const int64_t K = w[0]->cols;
    const int type = w[0]->type;
    GGB_CHECK_ARG(type == GGB_TYPE_Q4_0 || type == GGB_TYPE_Q8_0, "gemm: weight type %d", type);
    GemmArgs A{};
    GemmMaps maps{};
    int64_t N = 0;
    uintptr_t at16 = (uintptr_t)resid;
    for (int i = 0; i < n; i++) {
        at16 |= (uintptr_t)c[i];
        GGB_CHECK_ARG(w[i] && (c[i] || geglu) && w[i]->cols == K && w[i]->type == type, "gemm: matrices of one launch share K and the type");
        const int64_t rows = w[i]->rows;
        GGB_CHECK_ARG(K % 64 == 0 && rows % 32 == 0 && ldc[i] >= rows && ldc[i] % 4 == 0,
                      "gemm needs K %% 64 == 0, N %% 32 == 0 (N=%lld K=%lld)", (long long)rows, (long long)K);
        A.seg[i] = GemmSeg{w[i]->d, c[i], (int)ldc[i], (int)N, (int)rows};
        N += i + 1 < n ? (rows + 255) / 256 * 256 : rows;
    }
    A.n_seg = n;
    A.vec = at16 % 16 == 0; // row pitches are whole 16-byte pieces
    GGB_CHECK_ARG((uintptr_t)geglu % 8 == 0, "gemm_geglu: y starts on 8 bytes");
    const int kblocks = (int)(K / BK), sms = ggb_sm_count(), pb = ggb_payload_bytes(type);
    int pieces = ggb_gemm_pieces(T, N, K);
    if (pieces > 1 && (!workspace || workspace_bytes < (size_t)pieces * T * N * 4)) pieces = 1;
    GGB_CHECK_ARG(!geglu || (T > 128 && n == 2 && w[0]->rows == w[1]->rows && w[0]->rows % 256 == 0), "gemm_geglu: two matrices of as many rows and more than 128 tokens");
    if (geglu) pieces = 1, N = 2 * w[0]->rows;
    A.gelu = ggb_gelu_table_dev();
    // The tile (of one CTA or of a pair), and the CTAs along K, with the least estimated time (cycles).  A K block takes what its MMAs (130 each by a
    // pair of 256 columns, 100 of fewer, 80 by one CTA of 128, 40 of 64, and 100 for the wait and the commit), the bytes through shared memory
    // (written by TMA, read and written by the dequantisation, read for the MMAs), the bytes from L2 or the dequantisation take (2.7 a row: a fit, as
    // all of these), and no less than a group's way with it, 2000, over the groups.  The constants choose the
    // fastest of all tiles for 28 shapes from 16 x 2048 x 2048 to 512 x 65536 x 2048 and 2048 x 16384, all of which were timed.
    auto stages_of = [&](bool pr, int MT, int br, int *codes) { // of A rows (a K block's also tell of the group's buffer: no fewer than groups), of codes
        const int cs = br == 32 ? kMaxCodeStages : MT == 1 ? 12 : pr ? 4 : 8;
        if (codes) *codes = cs;
        return std::min<int>(kMaxStages, (int)((kRing - kTiles - cs * br * 2 * pb) / (MT * 16384)));
    };
    double best = -1.0;
    int splits = 1;
    bool pair = false;
    for (int pr = geglu ? 1 : 0; pr <= (geglu || T > 256 ? 1 : 0); pr++)
        for (int MT = 1; MT <= (T > (pr ? 256 : 128) ? 2 : 1); MT++)
            for (int bn = pr ? 256 : 128; bn >= (geglu ? 256 : 64); bn /= 2)
                for (int sp = 1; sp <= pieces; sp *= 2) {
                    const int chunks = pieces / sp, chunk_kb = (kblocks + pieces - 1) / pieces, br = pr ? bn / 2 : bn, rows = MT * (pr ? 256 : 128);
                    if (MT * chunks * bn > 512 || stages_of(pr, MT, br, nullptr) < 256 / br) continue;
                    const int64_t tiles = (N + bn - 1) / bn * ((T + rows - 1) / rows) * sp, slots = pr ? sms / 2 : sms, busy = std::min(tiles, slots) * (pr ? 2 : 1);
                    const double mma = MT * 4.0 * (pr ? (bn == 256 ? 130.0 : 100.0) : (bn == 128 ? 80.0 : 41.0)) + 100.0;
                    const double smem = (MT * 16384.0 + br * (4.0 * pb + 128.0) + MT * 4 * (4096.0 + br * 32.0)) / 190.0;
                    const double l2 = (MT * 16384.0 + br * 2.0 * pb) / std::min(90.0, 7450.0 / busy);
                    const double stage = std::max(std::max(std::max(mma, smem), l2), std::max(br * 2.7, 2030.0 * br / 256.0));
                    const double store = MT * 128.0 * bn / (geglu ? 20.0 : 10.0) * (sp > 1 ? chunks : 1);
                    double cost = (double)((tiles + slots - 1) / slots) * (chunks * chunk_kb * stage + store + (pr ? 12000.0 : 6150.0));
                    if (sp > 1) cost += 3240.0 + (double)pieces * T * N * 8.0 / (60.0 * sms);
                    if (best < 0.0 || cost < best) {
                        best = cost;
                        splits = sp, pair = pr;
                        A.MT = MT, A.BN = bn, A.chunks = chunks, A.chunk_kb = chunk_kb;
                    }
                }
    // Persistent pairs with tiles of 256 x 256, which dequantise every weight once per 256 tokens and store a tile behind the next one's MMAs: 800 cycles a K
    // block.  gate | up, 2 x 16384 x 2048 Q8_0: 256 tokens 40 us (52), but 512 tokens 72 us (65 in tiles of 512 rows); 65536 x 2048, 512 tokens 123 us (144)
    const int64_t big = (N + 255) / 256 * ((T + 255) / 256);
    const bool stream = geglu ? T <= 256 : pieces == 1 && T > 256 && (double)((big + sms / 2 - 1) / (sms / 2)) * kblocks * 800.0 + 14000.0 < best;
    if (stream) pair = true, splits = 1, A.MT = 1, A.BN = 256;
    const int br = pair ? A.BN / 2 : A.BN;
    A.groups = 256 / br;
    A.N = (int)N, A.nb = (int)w[0]->nb, A.kblocks = kblocks, A.T = (int)T;
    // Codes come from memory, A rows from L2: what is in flight of the codes bounds a product of few rows (256000 x 2048, Q4_0, 33 to 128 rows:
    // 4 stages 276 to 289 us, 12 stages 263 to 275), the MMAs and shared memory one of 512 rows a tile.
    A.stages = stages_of(pair, A.MT, br, &A.code_stages);
    const int a_rows = !pair && T <= A.MT * 128 ? (int)(T + 7) / 8 * 8 : A.MT * 128;
    A.a_tx = (uint32_t)a_rows * 128;
    A.ws = splits > 1 ? (float *)workspace : nullptr;
    A.resid = splits > 1 ? nullptr : resid; // added by the reducer
    A.geglu = (__nv_bfloat16 *)geglu;
    A.wait_error = ggb_wait_error_flag();
    int rc = ggb_tensor_map_bf16(&maps.a, a_bf16, T, K, K, a_rows);
    for (int i = 0; i < n && !rc; i++) rc = ggb_tensor_map_bytes(&maps.w[i], w[i]->qs, w[i]->rows, K / 32 * pb, 2 * pb, br);
    if (rc) return rc;
    const bool q4 = type == GGB_TYPE_Q4_0;
    auto kfn = pair ? (q4 ? gemm_quant_kernel<GGB_TYPE_Q4_0, true> : gemm_quant_kernel<GGB_TYPE_Q8_0, true>)
                    : (q4 ? gemm_quant_kernel<GGB_TYPE_Q4_0, false> : gemm_quant_kernel<GGB_TYPE_Q8_0, false>);
    if (stream)
        kfn = geglu ? (q4 ? gemm_quant_stream_kernel<GGB_TYPE_Q4_0, true> : gemm_quant_stream_kernel<GGB_TYPE_Q8_0, true>)
                    : (q4 ? gemm_quant_stream_kernel<GGB_TYPE_Q4_0, false> : gemm_quant_stream_kernel<GGB_TYPE_Q8_0, false>);
    if ((rc = ggb_allow_smem(kfn, kGemmSmem))) return rc;
    // row tiles first: those that share a piece of W run together
    const int rows = A.MT * (pair ? 256 : 128);
    dim3 grid((unsigned)((T + rows - 1) / rows * (pair ? 2 : 1)), (unsigned)((N + A.BN - 1) / A.BN), (unsigned)splits);
    if (stream) grid = dim3((unsigned)(2 * std::min<int64_t>(big, sms / 2)));
    GGB_CUDA(ggb_launch_early(kfn, ggb_cluster{pair ? 2u : 1u, 1, 1}, grid, dim3(stream ? kStreamThreads : kGemmThreads), kGemmSmem, maps, A));
    GGB_LAUNCH_CHECK();
    if (splits > 1) {
        A.resid = resid;
        const int64_t cnt = T * N;
        const int planes = (kblocks + A.chunk_kb - 1) / A.chunk_kb;
        if (tail && tail->rope) {
            const rope_args &r = *tail->rope;
            const int total = (r.H + r.Hkv) * (r.d / 2) + r.Hkv * r.d;
            GGB_CUDA(ggb_launch_step(splitk_rope_kernel, dim3((unsigned)((total + 255) / 256), (unsigned)T), dim3(256), 0, A, planes, r));
        } else if (tail) {
            const size_t row = (size_t)N * 4;
            if ((rc = ggb_allow_smem(splitk_norm_kernel, row))) return rc;
            GGB_CUDA(ggb_launch_step(splitk_norm_kernel, dim3((unsigned)T), dim3(GGB_DEV_NORM_THREADS), row, A, planes, tail->norm_w, tail->eps, tail->y));
        } else {
            GGB_CUDA(ggb_launch_step(splitk_reduce_kernel, dim3((unsigned)((cnt / 4 + 255) / 256)), dim3(256), 0, A, planes));
        }
        if (tail) tail->done = true;
        GGB_LAUNCH_CHECK();
    }
    return GGB_OK;
}

int ggb_op_gemm_bf16(const ggb_weight *w, const void *a_bf16, int64_t T, float *c, int64_t ldc, const float *resid,
                     void *workspace, size_t workspace_bytes) {
    const ggb_weight *ws[1] = {w};
    float *cs[1] = {c};
    const int64_t ls[1] = {ldc};
    GGB_CHECK_ARG(w != nullptr, "bad gemm args");
    return gemm_launch(1, ws, a_bf16, T, cs, ls, resid, workspace, workspace_bytes);
}

int ggb_op_gemm_bf16_multi(int n, const ggb_weight *const *w, const void *a_bf16, int64_t T, float *const *c, const int64_t *ldc,
                           void *workspace, size_t workspace_bytes) {
    return gemm_launch(n, w, a_bf16, T, c, ldc, nullptr, workspace, workspace_bytes);
}

int ggb_op_gemm_norm_bf16(const ggb_weight *w, const void *a_bf16, int64_t T, float *c, const float *resid, void *workspace, size_t workspace_bytes,
                          const float *norm_w, float eps, void *y_bf16) {
    GGB_CHECK_ARG(w && norm_w && y_bf16, "bad gemm_norm args");
    const ggb_weight *ws[1] = {w};
    float *cs[1] = {c};
    const int64_t ls[1] = {w->rows};
    gemm_tail tail{norm_w, eps, (__nv_bfloat16 *)y_bf16};
    const bool fits = (size_t)w->rows * 4 <= 200 * 1024; // a row in shared memory
    const int rc = gemm_launch(1, ws, a_bf16, T, cs, ls, resid, workspace, workspace_bytes, nullptr, fits ? &tail : nullptr);
    return rc || tail.done ? rc : ggb_op_rms_norm_bf16(c, norm_w, eps, w->rows, T, y_bf16);
}

int ggb_op_gemm_rope_store_bf16(const ggb_weight *const *w, const void *a_bf16, int64_t T, float *const *c, void *workspace, size_t workspace_bytes,
                                const int32_t *pos, int H, int Hkv, int d, float q_scale, void *kcache, void *vcache) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(w && w[0] && w[1] && w[2] && c && c[0] && c[1] && c[2] && pos && kcache && vcache && T > 0 && T <= 65535, "bad gemm_rope_store args");
    GGB_CHECK_ARG(w[0]->rows == (int64_t)H * d && w[1]->rows == (int64_t)Hkv * d && w[2]->rows == (int64_t)Hkv * d, "gemm_rope_store: rows of q, k, v");
    GGB_CHECK_ARG(ggb_rope_cos_dev() && ggb_rope_n_dims() == d, "rope table not initialised for head_dim %d", d);
    const rope_args r{pos, H, Hkv, d, ggb_rope_n_ctx(), q_scale, ggb_rope_cos_dev(), ggb_rope_sin_dev(), (__half *)kcache, (__half *)vcache};
    const int64_t ls[3] = {w[0]->rows, w[1]->rows, w[2]->rows};
    gemm_tail tail;
    tail.rope = &r;
    const int rc = gemm_launch(3, w, a_bf16, T, c, ls, nullptr, workspace, workspace_bytes, nullptr, &tail);
    return rc || tail.done ? rc : ggb_op_rope_kv_store_batch(c[0], c[1], c[2], pos, T, H, Hkv, d, q_scale, kcache, vcache);
}

int ggb_op_gemm_geglu_bf16(const ggb_weight *gate, const ggb_weight *up, const void *a_bf16, int64_t T, void *y_bf16) {
    GGB_CHECK_ARG(gate && up && y_bf16, "bad gemm_geglu args");
    const ggb_weight *ws[2] = {gate, up};
    float *cs[2] = {nullptr, nullptr};
    const int64_t ls[2] = {gate->rows, up->rows};
    return gemm_launch(2, ws, a_bf16, T, cs, ls, nullptr, nullptr, 0, y_bf16);
}

int ggb_op_attn_prefill(const float *q, const void *kcache, const void *vcache, int64_t T, int pos0, int H, int Hkv, int d,
                        float *out, void *out_bf16) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(q && kcache && vcache && (out || out_bf16) && T > 0 && d % 8 == 0 && d <= 256 && H % Hkv == 0, "bad attn_prefill args");
    // GGB_PREFILL_ATTN_SIMPLE: a warp a (token, head), with GGB_PREFILL_ATTN_GH4 a warp a token and four heads, whatever the sizes
    const bool simple = getenv("GGB_PREFILL_ATTN_SIMPLE") != nullptr;
    if (!simple && ggb_attn_prefill_fits(q, kcache, vcache, T, pos0, H, Hkv, d, out, out_bf16))
        return ggb_attn_prefill_tiles(q, kcache, vcache, T, pos0, H, Hkv, d, out, out_bf16);
    const int n_kv_max = pos0 + (int)T;
    if ((H / Hkv) % 4 == 0 && !simple) { // MQA / GQA: one CTA per (token, 4 heads of one KV head)
        const size_t smem4 = ((size_t)4 * n_kv_max + 4 * 4 * 256 + 16) * 4 + 16 * 8;
        GGB_CHECK_ARG(smem4 <= 200 * 1024, "attn_prefill: context %d too long for the score buffer", n_kv_max);
        if (smem4 > 48 * 1024) GGB_CUDA(cudaFuncSetAttribute(attn_prefill_gqa_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem4));
        attn_prefill_gqa_kernel<<<(unsigned)(T * (H / 4)), 128, smem4, ggb_cuda_stream()>>>(
            q, (const __half *)kcache, (const __half *)vcache, (int)T, pos0, H, Hkv, d, ggb_exp_table_dev(), out,
            (__nv_bfloat16 *)out_bf16, n_kv_max);
        GGB_LAUNCH_CHECK();
        return GGB_OK;
    }
    // query heads per warp: sharing the K/V loads between 4 heads (gh = 4) measured SLOWER for Gemma-2B at T = 512 (3.9 vs
    // 3.3 ms per prefill: a quarter of the warps, each with 4x the serial work), so one head per warp it is
    const int gh = getenv("GGB_PREFILL_ATTN_GH4") && (H / Hkv) % 4 == 0 ? 4 : 1;
    const size_t smem = (size_t)kAttnWarps * gh * n_kv_max * 4;
    GGB_CHECK_ARG(smem <= 200 * 1024, "attn_prefill: context %d too long for the score buffer", n_kv_max);
    const unsigned blocks = (unsigned)((T * (H / gh) + kAttnWarps - 1) / kAttnWarps);
    if (gh == 4) {
        if (smem > 48 * 1024) GGB_CUDA(cudaFuncSetAttribute(attn_prefill_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attn_prefill_kernel<4><<<blocks, kAttnWarps * 32, smem, ggb_cuda_stream()>>>(q, (const __half *)kcache, (const __half *)vcache,
                                                                                    (int)T, pos0, H, Hkv, d, ggb_exp_table_dev(), out, (__nv_bfloat16 *)out_bf16, n_kv_max);
    } else {
        if (smem > 48 * 1024) GGB_CUDA(cudaFuncSetAttribute(attn_prefill_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attn_prefill_kernel<1><<<blocks, kAttnWarps * 32, smem, ggb_cuda_stream()>>>(q, (const __half *)kcache, (const __half *)vcache,
                                                                                    (int)T, pos0, H, Hkv, d, ggb_exp_table_dev(), out, (__nv_bfloat16 *)out_bf16, n_kv_max);
    }
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

} // extern "C"
