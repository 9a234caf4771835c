// gemm_any.cu — C[T][N] = A[T][K] W[N][K]^T on the tensor cores (tcgen05) for fp32 matrices, and for the bf16 matrices that gemm.cu's TMA form does
// not take (fewer than 64 rows of A, odd sizes, strides and addresses).  Results and accuracy are those of fp32 multiply-adds.
//
// A tile is 128 rows of W (the M of an MMA: one lane of tensor memory each) x BT rows of A, so that few tokens cost few columns and a store of
// one token's 32 features is one line.  Sixteen warps bring both operands from memory, K in stages of 64, and write them as swizzled bf16
// tiles; nothing is asked of sizes or alignment (VEC: 16-byte loads, else numbers one by one).  One warp issues the MMAs, eight drain.
//
// fp32: a number is the sum of three bf16 numbers, x = xh + xm + xl (exact), and a product is xh yh + (xh ym + xm yh) + (xh yl + xm ym + xl yh),
// what is left out is below 2^-24 of it.  xm and xl are kept as 2^8 xm and 2^16 xl, and the sums of the two brackets come 2^8 and 2^16 times as
// large: so a number keeps its bits down to 2^-128, not only to 2^-110 (the smallest bf16 number is 2^-133, and below that the first
// part is no longer the largest: numbers of 2^-140, which have ten bits, come out to 12 bits).  The three parts of A lie behind one another as one operand of 3 BT columns, so that a part
// of W is read from shared memory once for all of its products: Wh [Ah Am Al], Wm [Ah Am], Wl [Ah], into columns for xh yh, first-order and
// second-order terms.  The tensor cores truncate their running sum, so every stage has an accumulator of its own (two, in turn), which the
// draining warps add to registers, rounding to nearest: the error against 64 bits is smaller than that of one chain of multiply-adds
// (K = 1000: 1.0e-7 against 5.7e-7).  A result that is not finite is computed once more by plain multiply-adds (plain_tile: an infinity is
// not the sum of its parts).
//
// A product of few tiles is cut along K over the CTAs of a cluster (up to 8), whose sums meet in shared memory and are added in order.
//
// What bounds it: fp32, shared memory (written and read: BT = 64: 170 KB a stage, 1330 cycles of 128 bytes); bf16, the loads in flight.
// 333 x 2816 x 1000 fp32: 98.4 -> 30.5 us (64 x 64 tiles of FMAs).
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "dense.cuh"
#include "gemm_any.cuh"
#include "tc.cuh"

namespace {

constexpr int kM = 128, kBK = 64;
constexpr int kDrain = 8, kLoad = 16, kMmaWarp = kDrain, kThreads = 32 * (kDrain + 1 + kLoad);
constexpr int kMaxBT = 64, kMaxSplits = 8;
enum { FULL = 0, EMPTY = 32, ACC_FULL = 64, ACC_FREE = 80, SLOT = 96, DEAD = 100, kCtl = 128 };

template <typename E> struct parts_of { static constexpr int n = sizeof(E) == 4 ? 3 : 1, stages_per_acc = 1, stages = sizeof(E) == 4 ? 2 : 4; };
template <typename E> __host__ __device__ inline uint32_t stage_bytes(int BT) { return (uint32_t)parts_of<E>::n * (kM + BT) * 128; }

struct any_args {
    const void *w, *a;
    int64_t N, K, T, lda, ldc;
    float *c;
    void *c_act; // when set: act(c) in the matrices' type instead of c
    int act, BT, splits, kblocks;
    int *wait_error;
};

__device__ __forceinline__ void tmem_load8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\ntcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_load8x3(uint32_t ta, uint32_t tb, uint32_t tc, uint32_t (&u)[8], uint32_t (&v)[8], uint32_t (&w)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%24];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%25];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%26];\n"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]),
                   "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                 : "r"(ta), "r"(tb), "r"(tc)
                 : "memory");
}

// Two fp32 numbers as three pairs of bf16 numbers: h + 2^-8 m + 2^-16 l, each remainder exact
__device__ __forceinline__ void split3_scaled(f32x2 v, uint32_t &h, uint32_t &m, uint32_t &l) {
    const f32x2 minus = pack2(-1.f, -1.f), up = pack2(256.f, 256.f);
    float2 x = unpack2(v);
    h = pack_bf16x2(x.x, x.y);
    v = mul2(fma2(pack2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u)), minus, v), up);
    x = unpack2(v);
    m = pack_bf16x2(x.x, x.y);
    v = mul2(fma2(pack2(__uint_as_float(m << 16), __uint_as_float(m & 0xffff0000u)), minus, v), up);
    x = unpack2(v);
    l = pack_bf16x2(x.x, x.y);
}

// The results of a tile that are not finite (odd: of a row of W, a bit a token) once more by plain multiply-adds, by all threads: 4 x 4 results a thread
// of the first 16 warps, K in steps of 32 through shared memory.  smem: where the stages were.  A portion of NaN takes 150 us where
// finite numbers take 22 (333 x 1408 x 1000; each result by a walk of its own along K: 1040).
template <typename E, typename PUT> __device__ __noinline__ void plain_tile(const any_args &g, int64_t n0, int64_t t0, int BT, const uint64_t *odd, float *smem, PUT put) {
    constexpr int KB = 32, PITCH = KB + 1, NL = ((kM + kMaxBT) * KB + kThreads - 1) / kThreads;
    const int tid = threadIdx.x, rg = tid & 31, cg = tid >> 5;
    float *sw = smem, *sa = smem + kM * PITCH, acc[4][4], next[NL];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    auto fetch = [&](int64_t k0) {
#pragma unroll
        for (int u = 0; u < NL; u++) {
            const int i = tid + kThreads * u, r = i / KB;
            const int64_t k = k0 + i % KB, row = r < kM ? n0 + r : t0 + r - kM;
            next[u] = 0.f;
            if (r < kM + BT && k < g.K && row < (r < kM ? g.N : g.T))
                next[u] = to_f32(r < kM ? static_cast<const E *>(g.w)[row * g.K + k] : static_cast<const E *>(g.a)[row * g.lda + k]);
        }
    };
    fetch(0);
    for (int64_t k0 = 0; k0 < g.K; k0 += KB) {
        const int ks = (int)min((int64_t)KB, g.K - k0);
        __syncthreads();
#pragma unroll
        for (int u = 0; u < NL; u++) {
            const int i = tid + kThreads * u;
            if (i < (kM + BT) * KB) smem[i / KB * PITCH + i % KB] = next[u];
        }
        __syncthreads();
        fetch(k0 + KB);
        if (cg < 16)
            for (int k = 0; k < ks; k++) {
                float w[4], x[4];
#pragma unroll
                for (int i = 0; i < 4; i++) w[i] = sw[(rg + 32 * i) * PITCH + k], x[i] = cg + 16 * i < BT ? sa[(cg + 16 * i) * PITCH + k] : 0.f;
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] = fmaf(w[i], x[j], acc[i][j]);
            }
    }
    if (cg < 16)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int row = rg + 32 * i;
            const uint64_t again = odd[row] | odd[kM + row];
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (again >> (cg + 16 * j) & 1) put(cg + 16 * j, row, acc[i][j]);
        }
}

// 16 bytes of a row from column k on: whole, or what lies inside K number by number
template <typename E, bool VEC> __device__ __forceinline__ uint4 load_piece(const E *row, int64_t k, int64_t K) {
    constexpr int V = 16 / (int)sizeof(E);
    if (VEC) return k < K ? ld_stream_u4(row + k) : make_uint4(0, 0, 0, 0); // K is a multiple of V
    union {
        E e[V];
        uint4 u;
    } p;
    p.u = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int i = 0; i < V; i++)
        if (k + i < K) p.e[i] = row[k + i];
    return p.u;
}

template <typename E, bool VEC>
__global__ void __launch_bounds__(kThreads, 1) gemm_any_kernel(const __grid_constant__ any_args g) {
    constexpr int P = parts_of<E>::n, SPA = parts_of<E>::stages_per_acc, STAGES = parts_of<E>::stages;
    extern __shared__ uint8_t ga_raw[];
    __shared__ uint64_t s_odd[P == 3 ? 2 * kM : 1]; // of a draining thread: tokens of its row whose results are not finite
    const uint32_t raw0 = smem_u32(ga_raw), base = (raw0 + 1023u) & ~1023u;
    uint8_t *gbase = ga_raw + (base - raw0);
    const int BT = g.BT;
    const uint32_t st_bytes = stage_bytes<E>(BT), part_a = P * kM * 128, bars = base + STAGES * st_bytes;
    uint8_t *ctl = gbase + STAGES * st_bytes;
    volatile int *dead = reinterpret_cast<volatile int *>(ctl + DEAD);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int rank = g.splits > 1 ? (int)cluster_rank() : 0;
    const int64_t tile = blockIdx.x / g.splits, m_tiles = (g.T + BT - 1) / BT;
    const int64_t t0 = tile % m_tiles * BT, n0 = tile / m_tiles * kM; // those that share rows of W run together
    const int per = (g.kblocks + g.splits - 1) / g.splits, kb0 = min(rank * per, g.kblocks), kb1 = min(kb0 + per, g.kblocks), nkb = kb1 - kb0;
    if (tid == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(bars + FULL + 8 * s, kLoad);
            mbar_init(bars + EMPTY + 8 * s, 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(bars + ACC_FULL + 8 * s, 1);
            mbar_init(bars + ACC_FREE + 8 * s, kDrain);
        }
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) tmem_alloc512(bars + SLOT);
    early_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    step_next();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<uint32_t *>(ctl + SLOT), 0);
    const uint32_t acc_cols = P * BT; // of one accumulator; two of them: at most 384

    if (warp > kMmaWarp) {
        // ---- a thread owns one 16-byte piece of every RS-th row of the stage: rows of W, then rows of A
        constexpr int V = 16 / (int)sizeof(E), PCS = kBK / V, RS = 32 * kLoad / PCS, NI = (kM + kMaxBT + RS - 1) / RS, NW = kM / RS;
        const int lt = tid - 32 * (kMmaWarp + 1), pc = lt % PCS, r0 = lt / PCS;
        const E *wp = static_cast<const E *>(g.w) + (n0 + r0) * g.K, *ap = static_cast<const E *>(g.a) + (t0 + r0) * g.lda;
        uint32_t live = 0; // bit i: row r0 + RS i of the stage exists
#pragma unroll
        for (int i = 0; i < NI; i++) {
            const int r = r0 + RS * i;
            if (i < NW ? n0 + r < g.N : (r - kM < BT && t0 + r - kM < g.T)) live |= 1u << i;
        }
        uint4 v[NI];
        auto fetch = [&](int i, int kb) {
            const E *row = i < NW ? wp + (int64_t)(RS * i) * g.K : ap + (int64_t)(RS * i - kM) * g.lda;
            v[i] = live >> i & 1 ? load_piece<E, VEC>(row, (int64_t)kb * kBK + pc * V, g.K) : make_uint4(0, 0, 0, 0);
        };
        if (nkb > 0)
#pragma unroll
            for (int i = 0; i < NI; i++) fetch(i, kb0);
        int s = 0;
        uint32_t ph = 1;
        for (int kb = kb0; kb < kb1; kb++) {
            if (!mbar_wait_warp(bars + EMPTY + 8 * s, ph, dead)) break;
            uint8_t *st = gbase + s * st_bytes;
#pragma unroll
            for (int i0 = 0; i0 < NI; i0 += 4) { // four pieces at a time: their chains of instructions side by side
                uint2 h[4], m[4], l[4];
                if (P == 3)
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (i0 + u < NI) {
                            const uint4 x = v[i0 + u];
                            split3_scaled(pack2(__uint_as_float(x.x), __uint_as_float(x.y)), h[u].x, m[u].x, l[u].x);
                            split3_scaled(pack2(__uint_as_float(x.z), __uint_as_float(x.w)), h[u].y, m[u].y, l[u].y);
                        }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int i = i0 + u;
                    if (i >= NI) continue;
                    const int r = r0 + RS * i, ra = r - kM; // row of W's or A's tile
                    const bool is_w = i < NW;
                    uint8_t *dst = is_w ? st + r * 128 : st + part_a + ra * 128;
                    const int pitch = (is_w ? kM : BT) * 128; // between the parts
                    if (is_w || ra < BT) {
                        if (P == 1) *reinterpret_cast<uint4 *>(dst + ((pc ^ (r & 7)) << 4)) = v[i];
                        else {
                            uint8_t *d = dst + (((pc >> 1) ^ (r & 7)) << 4) + 8 * (pc & 1);
                            *reinterpret_cast<uint2 *>(d) = h[u];
                            *reinterpret_cast<uint2 *>(d + pitch) = m[u];
                            *reinterpret_cast<uint2 *>(d + 2 * pitch) = l[u];
                        }
                    }
                    if (kb + 1 < kb1) fetch(i, kb + 1); // its way from memory is the rest of this stage and the wait for the next
                }
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + FULL + 8 * s);
            if (++s == STAGES) s = 0, ph ^= 1u;
        }
    } else if (warp == kMmaWarp) {
        int s = 0;
        uint32_t ph = 0;
        for (int kb = kb0; kb < kb1; kb++) {
            const int q = kb - kb0, acc = q / SPA, buf = acc & 1;
            if (q % SPA == 0) mbar_wait_bounded(bars + ACC_FREE + 8 * buf, ((acc >> 1) & 1) ^ 1, dead);
            mbar_wait_bounded(bars + FULL + 8 * s, ph, dead);
            tc_fence_after();
            const uint32_t d = tmem + buf * acc_cols, w_lo = umma_desc_lo(base + s * st_bytes, 16), a_lo = umma_desc_lo(base + s * st_bytes + part_a, 16);
#pragma unroll
            for (int k = 0; k < kBK / 16; k++) { // 16 numbers are 2 descriptor units
                umma_ss(d, w_lo + 2 * k, a_lo + 2 * k, umma_idesc(kM, P * BT), k > 0 || q % SPA != 0);
                if (P == 3) {
                    umma_ss(d + BT, w_lo + kM * 8 + 2 * k, a_lo + 2 * k, umma_idesc(kM, 2 * BT), 1);
                    umma_ss(d + 2 * BT, w_lo + 2 * kM * 8 + 2 * k, a_lo + 2 * k, umma_idesc(kM, BT), 1);
                }
            }
            umma_arrive(bars + EMPTY + 8 * s);
            if (q % SPA == SPA - 1 || kb == kb1 - 1) umma_arrive(bars + ACC_FULL + 8 * buf);
            if (++s == STAGES) s = 0, ph ^= 1u;
        }
    }
    constexpr int kCols = kMaxBT / 2; // of a draining warp: one half of the tile's tokens, 32 rows of W
    float sum[kCols];
    const int lq = warp & 3, half = warp >> 2, hc = BT / 2, row = lq * 32 + lane;
    if (warp < kDrain) {
#pragma unroll
        for (int c = 0; c < kCols; c++) sum[c] = 0.f;
        const int accs = (nkb + SPA - 1) / SPA;
        for (int q = 0; q < accs; q++) {
            const int buf = q & 1;
            mbar_wait_warp(bars + ACC_FULL + 8 * buf, (q >> 1) & 1, dead);
            tc_fence_after();
            const uint32_t col = tmem + ((uint32_t)(lq * 32) << 16) + buf * acc_cols + half * hc;
#pragma unroll
            for (int c0 = 0; c0 < kCols; c0 += 8)
                if (c0 < hc) {
                    uint32_t x[8], y[8], z[8];
                    if (P == 3) tmem_load8x3(col + c0, col + BT + c0, col + 2 * BT + c0, x, y, z);
                    else tmem_load8(col + c0, x);
#pragma unroll
                    for (int c = 0; c < 8; c++) sum[c0 + c] += P == 3 ? fmaf(fmaf(__uint_as_float(z[c]), 0x1p-8f, __uint_as_float(y[c])), 0x1p-8f, __uint_as_float(x[c])) : __uint_as_float(x[c]);
                }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + ACC_FREE + 8 * buf);
        }
    }
    __syncthreads(); // every MMA and every write of a stage is done
    auto put = [&](int c, int row, float v) {
        const int64_t at = (t0 + c) * g.ldc + n0 + row;
        if (g.c_act) static_cast<E *>(g.c_act)[at] = from_f32<E>(act_f32(v, g.act));
        else g.c[at] = v;
    };
    uint64_t odd = 0;
    auto store = [&](int c, float v) { // token column c of the tile
        if (t0 + c >= g.T || n0 + row >= g.N) return;
        if (P == 3 && !isfinite(v)) odd |= 1ull << c;
        put(c, row, v);
    };
    if (g.splits > 1) { // the ranks' sums, [token][row], in order
        float *mine = reinterpret_cast<float *>(gbase);
        if (warp < kDrain) {
#pragma unroll
            for (int c = 0; c < kCols; c++)
                if (c < hc) mine[(half * hc + c) * kM + row] = sum[c];
        }
        cluster_sync();
        if (warp < kDrain)
            for (int c = half + 2 * rank; c < BT; c += 2 * g.splits) {
                float v = 0.f;
                for (int q = 0; q < g.splits; q++) v += ld_cluster_f32(cluster_addr(base + (uint32_t)(c * kM + row) * 4, q));
                store(c, v);
            }
        cluster_sync(); // a rank's sums are read until here
    } else if (warp < kDrain) {
#pragma unroll
        for (int c = 0; c < kCols; c++)
            if (c < hc) store(half * hc + c, sum[c]);
    }
    if (warp == kMmaWarp) {
        settle(dead);
        tc_fence_after();
        tmem_free512(tmem);
        if (lane == 0 && *dead) *g.wait_error = 1;
    }
    if constexpr (P == 3) { // in bf16 the tensor cores' sums are plain arithmetic's
        if (__syncthreads_or(odd != 0 && !*dead)) {
            if (warp < kDrain) s_odd[half * kM + row] = odd;
            plain_tile<E>(g, n0, t0, BT, s_odd, reinterpret_cast<float *>(gbase), put);
        }
    }
}

// ------------------------------------------------------------------------------------------------ the slots of a mixture of experts, bf16
// C[slot][N] = A[row of the slot][K] W[expert of the slot][N][K]^T for a portion of few slots.  A tile is 128 rows of an expert's matrix, by TMA, x up to 64
// of its slots, whose rows of A four warps copy through the slot list (rows past the last stay as they are: they give columns that nobody stores).
// Persistent CTAs; the tile list lies in shared memory.  Every block of 64 along K has an accumulator of its own (four, in turn), which eight warps add up
// in fp32: K = 8192: error against 64 bits 3e-7, one chain of multiply-adds 9.5e-7, one accumulator of the tensor cores 9.2e-6.
//
// Bound by memory.  32 experts, 1408 x 2048: 64 slots 34 us, 256 slots 37 us, 5.0 TB/s of matrices (440 us on the tile kernel; 46 us by gathered rows in
// gemm.cu's tiles of 128).
constexpr int kMaxSlots = 511, kMaxTiles = kMaxSlots + kMaxSlots / kMaxBT;
constexpr int kFewStages = 8, kFewAccs = 4, kCopy = 4, kTmaWarp = kDrain + 1, kFewThreads = 32 * (kTmaWarp + 1 + kCopy);
constexpr int kLag = 3; // stages whose rows of A are under way
constexpr uint32_t kFewStage = (kM + kMaxBT) * 128;
enum { F_FULL = 0, F_EMPTY = 64, F_ACC_FULL = 128, F_ACC_FREE = 160, F_SLOT = 192, F_DEAD = 196, kFewCtl = 256 };

struct few_args {
    const __nv_bfloat16 *a;
    int64_t N, lda, ldc;
    float *c;
    __nv_bfloat16 *c_act;
    int act, kblocks, n, max_tiles; // slots; tiles there may be
    int *wait_error;
    ggb_moe_groups grp;
};
struct few_tile {
    int row0, expert, rows, BT; // first slot, slots, as a multiple of 16
};

__global__ void __launch_bounds__(kFewThreads, 1) gemm_few_slots_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ few_args g) {
    typedef __nv_bfloat16 E;
    extern __shared__ uint8_t ga_raw[];
    __shared__ few_tile tiles[kMaxTiles];
    __shared__ int row_src[kMaxSlots];
    const uint32_t raw0 = smem_u32(ga_raw), base = (raw0 + 1023u) & ~1023u, bars = base + kFewStages * kFewStage;
    uint8_t *ctl = ga_raw + (bars - raw0);
    volatile int *dead = reinterpret_cast<volatile int *>(ctl + F_DEAD);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < kFewStages; s++) {
            mbar_init(bars + F_FULL + 8 * s, 1 + kCopy);
            mbar_init(bars + F_EMPTY + 8 * s, 1);
        }
        for (int s = 0; s < kFewAccs; s++) {
            mbar_init(bars + F_ACC_FULL + 8 * s, 1);
            mbar_init(bars + F_ACC_FREE + 8 * s, kDrain);
        }
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) tmem_alloc512(bars + F_SLOT);
    early_wait();
    const int n_tiles = min(*g.grp.n_tiles, g.max_tiles);
    for (int i = tid; i < n_tiles; i += kFewThreads) {
        const int e = g.grp.tile_expert[i], r0 = g.grp.tile_row0[i], rows = min(kMaxBT, g.grp.offsets[e + 1] - r0);
        tiles[i] = few_tile{r0, e, rows, (rows + 15) / 16 * 16};
    }
    for (int i = tid; i < g.n; i += kFewThreads) row_src[i] = g.grp.row_src ? g.grp.row_src[i] : i;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    step_next();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<uint32_t *>(ctl + F_SLOT), 0);
    const int cols = (int)((g.N + kM - 1) / kM), total = n_tiles * cols; // item: tile item / cols, rows item % cols * 128 of its matrix

    if (warp == kTmaWarp) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 1;
            for (int item = blockIdx.x; item < total; item += gridDim.x) {
                const int row = (int)(tiles[item / cols].expert * g.N) + item % cols * kM;
                for (int kb = 0; kb < g.kblocks; kb++) {
                    if (!mbar_wait_bounded(bars + F_EMPTY + 8 * s, ph, dead)) break;
                    mbar_expect_tx(bars + F_FULL + 8 * s, kM * 128);
                    tma_load_2d(base + s * kFewStage, &map_w, kb * kBK, row, bars + F_FULL + 8 * s);
                    if (++s == kFewStages) s = 0, ph ^= 1u;
                }
            }
        }
        __syncwarp();
    } else if (warp > kTmaWarp) {
        // ---- a thread copies one 16-byte piece of every 16th row; a stage is handed over kLag stages behind its request
        const int lt = tid - 32 * (kTmaWarp + 1), pc = lt & 7, r0 = lt >> 3;
        int s = 0, asked = 0, given = 0;
        uint32_t ph = 1;
        auto give = [&]() {
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + F_FULL + 8 * (given % kFewStages));
            given++;
        };
        for (int item = blockIdx.x; item < total; item += gridDim.x) {
            const few_tile t = tiles[item / cols];
            const E *ap[4];
#pragma unroll
            for (int i = 0; i < 4; i++) ap[i] = g.a + (int64_t)row_src[t.row0 + min(r0 + 16 * i, t.rows - 1)] * g.lda + 8 * pc;
            for (int kb = 0; kb < g.kblocks; kb++) {
                if (!mbar_wait_warp(bars + F_EMPTY + 8 * s, ph, dead)) break;
#pragma unroll
                for (int i = 0; i < 4; i++) // rows 16 apart lie at the same place of the swizzle
                    if (r0 + 16 * i < t.rows) cp_async16(base + s * kFewStage + (kM + r0 + 16 * i) * 128 + ((pc ^ (r0 & 7)) << 4), ap[i] + kb * kBK);
                cp_async_commit();
                if (++s == kFewStages) s = 0, ph ^= 1u;
                if (++asked > kLag) {
                    cp_async_wait<kLag>();
                    give();
                }
            }
        }
        cp_async_wait<0>();
        while (given < asked) give();
    } else if (warp == kMmaWarp) {
        int s = 0;
        uint32_t ph = 0, q = 0;
        for (int item = blockIdx.x; item < total; item += gridDim.x) {
            const uint32_t idesc = umma_idesc(kM, tiles[item / cols].BT);
            for (int kb = 0; kb < g.kblocks; kb++, q++) {
                const uint32_t buf = q % kFewAccs, at = base + s * kFewStage;
                mbar_wait_bounded(bars + F_ACC_FREE + 8 * buf, ((q / kFewAccs) & 1) ^ 1, dead);
                mbar_wait_bounded(bars + F_FULL + 8 * s, ph, dead);
                tc_fence_after();
                umma_ss_k4(tmem + buf * kMaxBT, umma_desc_lo(at, 16), umma_desc_lo(at + kM * 128, 16), idesc, 0);
                umma_arrive(bars + F_EMPTY + 8 * s);
                umma_arrive(bars + F_ACC_FULL + 8 * buf);
                if (++s == kFewStages) s = 0, ph ^= 1u;
            }
        }
    } else {
        constexpr int kCols = kMaxBT / 2; // of a draining warp: one half of the tile's slots, 32 rows of W
        const int lq = warp & 3, half = warp >> 2;
        uint32_t q = 0;
        for (int item = blockIdx.x; item < total; item += gridDim.x) {
            const few_tile t = tiles[item / cols];
            const int hc = t.BT / 2;
            float sum[kCols];
#pragma unroll
            for (int c = 0; c < kCols; c++) sum[c] = 0.f;
            for (int kb = 0; kb < g.kblocks; kb++, q++) {
                const uint32_t buf = q % kFewAccs;
                mbar_wait_warp(bars + F_ACC_FULL + 8 * buf, (q / kFewAccs) & 1, dead);
                tc_fence_after();
                const uint32_t col = tmem + ((uint32_t)(lq * 32) << 16) + buf * kMaxBT + half * hc;
#pragma unroll
                for (int c0 = 0; c0 < kCols; c0 += 8)
                    if (c0 < hc) {
                        uint32_t x[8];
                        tmem_load8(col + c0, x);
#pragma unroll
                        for (int c = 0; c < 8; c++) sum[c0 + c] += __uint_as_float(x[c]);
                    }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bars + F_ACC_FREE + 8 * buf);
            }
            const int64_t n = (int64_t)(item % cols) * kM + lq * 32 + lane;
#pragma unroll
            for (int c = 0; c < kCols; c++) {
                const int r = half * hc + c;
                if (c >= hc || r >= t.rows || n >= g.N) continue;
                const int64_t out = (int64_t)(t.row0 + r) * g.ldc + n;
                if (g.c_act) g.c_act[out] = from_f32<E>(act_f32(sum[c], g.act));
                else g.c[out] = sum[c];
            }
        }
    }
    __syncthreads();
    if (warp == kMmaWarp) {
        settle(dead);
        tc_fence_after();
        tmem_free512(tmem);
        if (lane == 0 && *dead) *g.wait_error = 1;
    }
}

template <typename E>
int launch_any(const void *w, int64_t N, int64_t K, const void *a, int64_t lda, int64_t T, float *c, int64_t ldc, void *c_act, int act) {
    constexpr int P = parts_of<E>::n, V = 16 / (int)sizeof(E);
    any_args g{w, a, N, K, T, lda, ldc, c, c_act, act, 0, 1, (int)((K + kBK - 1) / kBK), ggb_wait_error_flag()};
    // the tile and the split of the least estimate.  Cycles of a stage: the bytes that pass through shared memory at 128 a cycle (written once;
    // read for the MMAs: every part of W once, the parts of A as often as they are multiplied), the loading warps' instructions (about 35 a 16-byte
    // piece and thread), or the bytes from memory at 24 a cycle and SM; a tile: its prologue and its stores
    const int64_t n_tiles = (N + kM - 1) / kM;
    const int sms = ggb_sm_count();
    double best = 0.0;
    for (int bt = 16; bt <= kMaxBT; bt += 16) {
        const int64_t tiles = n_tiles * ((T + bt - 1) / bt);
        for (int splits = 1; splits <= kMaxSplits && splits <= g.kblocks; splits *= 2) {
            const double smem = (P * (kM + bt) * 128.0 + P * kM * 128.0 + (P == 3 ? 6 : 1) * bt * 128.0) / 128.0;
            const double issue = (P == 3 ? 36.0 : 8.0) * (kM + bt) * (kBK / V) / 32.0 / 4.0, bytes = (kM + bt) * kBK * sizeof(E) / 24.0;
            const double stage = std::max(smem, std::max(issue, bytes));
            const double rounds = (double)((tiles * splits + sms - 1) / sms);
            const double cost = rounds * (((g.kblocks + splits - 1) / splits) * stage + 3000.0 + 20.0 * bt) + (splits > 1 ? 3000.0 : 0.0);
            if (!g.BT || cost < best) best = cost, g.BT = bt, g.splits = splits;
        }
    }
    const bool vec = K % V == 0 && lda % V == 0 && ((uintptr_t)w | (uintptr_t)a) % 16 == 0;
    auto kern = vec ? gemm_any_kernel<E, true> : gemm_any_kernel<E, false>;
    size_t smem = 1024 + (size_t)parts_of<E>::stages * stage_bytes<E>(g.BT) + kCtl;
    if (g.splits > 1) smem = std::max(smem, kOneCtaSmem);
    const int rc = ggb_allow_smem(kern, smem);
    if (rc) return rc;
    const int64_t ctas = n_tiles * ((T + g.BT - 1) / g.BT) * g.splits;
    GGB_CHECK_ARG(ctas < (1ll << 31), "linear: %lld tiles", (long long)ctas);
    GGB_CUDA(ggb_launch_early(kern, ggb_cluster{(unsigned)g.splits, 1, 1}, dim3((unsigned)ctas), dim3(kThreads), smem, g));
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

} // namespace

int ggb_gemm_any(int dt, const void *w, int64_t N, int64_t K, const void *a, int64_t lda, int64_t T, float *c, int64_t ldc, void *c_act, int act) {
    return dt == GGB_TYPE_BF16 ? launch_any<__nv_bfloat16>(w, N, K, a, lda, T, c, ldc, c_act, act) : launch_any<float>(w, N, K, a, lda, T, c, ldc, c_act, act);
}

int ggb_gemm_any_grouped(const void *w, int64_t N, int64_t K, const void *a, int64_t lda, int64_t n, int n_exp, float *c, int64_t ldc, void *c_act, int act,
                         const ggb_moe_groups &grp) {
    typedef __nv_bfloat16 E;
    GGB_CHECK_ARG(n <= kMaxSlots && K % kBK == 0 && lda % 8 == 0 && ((uintptr_t)w | (uintptr_t)a) % 16 == 0, "moe_linear: %lld slots, K %lld", (long long)n, (long long)K);
    // the list's tiles, at most: an expert with slots leaves one of its tiles half empty
    const int max_tiles = (int)(n / kMaxBT + std::min<int64_t>(n, n_exp));
    const few_args g{(const E *)a, N, lda, ldc, c, (E *)c_act, act, (int)(K / kBK), (int)n, max_tiles, ggb_wait_error_flag(), grp};
    const int64_t items = (N + kM - 1) / kM * max_tiles;
    GGB_CHECK_ARG(items < (1ll << 31) && n_exp * N < (1ll << 31), "moe_linear: %lld tiles of %lld rows", (long long)items, (long long)(n_exp * N));
    CUtensorMap map_w;
    const size_t smem = 1024 + (size_t)kFewStages * kFewStage + kFewCtl;
    int rc = ggb_allow_smem(gemm_few_slots_kernel, smem);
    if (!rc) rc = ggb_tensor_map_bf16(&map_w, w, n_exp * N, K, K, kM);
    if (rc) return rc;
    GGB_CUDA(ggb_launch_early(gemm_few_slots_kernel, ggb_cluster{1, 1, 1}, dim3((unsigned)std::min<int64_t>(items, ggb_sm_count())), dim3(kFewThreads), smem, map_w, g));
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}
