// gemm.cu — products of plain bf16 matrices on the tensor cores: C[T][N] = A[T][K] W[N][K]^T, and the grouped form for a mixture of experts.
//
// A tile of C is 256 x 256, by two CTAs of a cluster, or 128 x (256, 128, 64), by one; a tile of an expert's slots is gemm_slots_kernel's.  Both operands arrive by TMA (tensor maps, 128-byte swizzle, 64 numbers of K a stage)
// in a ring that takes all of shared memory but the epilogue's corner; one warp issues the MMAs, eight drain tensor memory.  CTAs are
// persistent: where a tile needs half of tensor memory, the next one's products run while the last one's are stored.  The epilogue
// turns 32 x 32 pieces in shared memory, so that a store instruction writes whole 128-byte lines.
//
// A product along a long K is summed in `chunks` pieces of K, each with an accumulator of its own in tensor memory, added up in order by
// the epilogue (the tensor cores truncate a running sum at every step: shorter sums are more exact), and, where that still leaves SMs
// without work, over several CTAs whose sums (each of its own pieces) meet in a workspace and are added in order.  The number of pieces is
// what a split over the SMs in 256 x 256 tiles needs; the tile is then the one with the least estimated time.
//
// What bounds it: 1024 x 8192 x 2048 is 128 tiles of 256 x 256 on 74 pairs of CTAs, two rounds of 32 stages of 512 cycles of the tensor cores,
// the second for 54 pairs; the tensor cores are busy for 61 to 64 % of the cycles.  37.3 us, 921 TFLOP/s (47.6 us with both operands
// copied by cp.async and rows stored by their own lanes; 38.8 us in one round of 256 x 256 tiles a CTA, whose stores nothing hides).
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "dense.cuh"
#include "tc.cuh"

namespace {

constexpr int BK = 64, BM = 128; // a stage of K, the rows of a CTA
constexpr int kThreads = 384; // warp 0: TMA, 1: MMA, 2: tensor memory, 4..11: epilogue
constexpr uint32_t kRing = 192 * 1024, kTurn = 8 * 4096;
constexpr int kMaxStages = 8, kListed = 256; // groups whose first row tiles are kept in shared memory
constexpr size_t kSmem = 1024 + kRing + kTurn + 256;
static_assert(kSmem >= kOneCtaSmem, "pairs of CTAs");
enum { FULL = 0, EMPTY = 64, ACC_FULL = 128, ACC_FREE = 144, SLOT = 160, DEAD = 168 };

struct gemm_args {
    int T, N, kblocks;
    int BN, n_tiles, m_tiles;
    int chunks, chunk_kb, splits; // K pieces a CTA sums, their blocks of 64, CTAs along K
    int stages;
    // grouped: group g has the rows [m_ranges[g], m_ranges[g + 1]) of C, whose rows of a are row_src[.] (or the same, by TMA), and the rows g * N .. of W
    const int32_t *m_ranges, *row_src;
    int n_groups;
    const __nv_bfloat16 *a;
    float *c;
    __nv_bfloat16 *act_out; // when set: bf16 act(c) instead of c
    int act;
    int64_t ldc;
    int vec; // rows of C start on 16 bytes
    float *ws; // [splits][T][N] or null
    int *wait_error;
};

struct pair_maps {
    CUtensorMap w, a[4]; // a: boxes of 128 rows; of a grouped product 32, 64, 96 and 128
};
struct tile_at {
    int m0, m_end, n0, split, group;
};

// a warp's 32 rows x 32 columns of accumulators, K pieces added in order, stored as whole lines
__device__ __forceinline__ void store_piece(const gemm_args &a, uint32_t col, int chunks, uint32_t my, int lane, int row0, int m_end, int n0, int split) {
    uint32_t v[32];
    if (chunks > 0) tmem_load32(col, v);
    else // no block of K is left for this CTA
        for (int q = 0; q < 32; q++) v[q] = 0;
    for (int ch = 1; ch < chunks; ch++) {
        uint32_t u[32];
        tmem_load32(col + ch * a.BN, u);
#pragma unroll
        for (int q = 0; q < 32; q++) v[q] = __float_as_uint(__uint_as_float(v[q]) + __uint_as_float(u[q]));
    }
    // row = lane -> eight lanes a row: 16-byte piece p of row r at place p ^ (r & 7)
    __syncwarp();
#pragma unroll
    for (int p = 0; p < 8; p++)
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(my + lane * 128 + ((p ^ (lane & 7)) << 4)), "r"(v[4 * p]), "r"(v[4 * p + 1]), "r"(v[4 * p + 2]),
                     "r"(v[4 * p + 3])
                     : "memory");
    __syncwarp();
    const int p = lane & 7, n = n0 + 4 * p;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int r = 4 * q + (lane >> 3), row = row0 + r;
        float4 o;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o.x), "=f"(o.y), "=f"(o.z), "=f"(o.w) : "r"(my + r * 128 + ((p ^ (r & 7)) << 4)) : "memory");
        if (row >= m_end || n >= a.N) continue;
        if (a.act_out && !a.ws) { // the next product's operand; N and ldc are multiples of 8
            uint2 y;
            y.x = pack_bf16x2(act_f32(o.x, a.act), act_f32(o.y, a.act));
            y.y = pack_bf16x2(act_f32(o.z, a.act), act_f32(o.w, a.act));
            *reinterpret_cast<uint2 *>(a.act_out + row * a.ldc + n) = y;
        } else { // N is a multiple of 4
            float *dst = a.ws ? a.ws + ((int64_t)split * a.T + row) * a.N + n : a.c + row * a.ldc + n;
            if (a.vec) *reinterpret_cast<float4 *>(dst) = o;
            else dst[0] = o.x, dst[1] = o.y, dst[2] = o.z, dst[3] = o.w;
        }
    }
}

// GROUPED: row tiles of a group's own rows
template <bool GROUPED>
__global__ void __launch_bounds__(kThreads, 1) gemm_tma_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const gemm_args a) {
    extern __shared__ uint8_t gm_raw[];
    __shared__ int first_tile[GROUPED ? kListed + 1 : 1]; // the first row tile of a group
    const uint32_t raw0 = smem_u32(gm_raw), base = (raw0 + 1023u) & ~1023u, turn = base + kRing, bars = turn + kTurn;
    uint8_t *ctl = gm_raw + (bars - raw0);
    volatile int *dead = reinterpret_cast<volatile int *>(ctl + DEAD);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t a_bytes = BM * 128, stage_bytes = a_bytes + (uint32_t)a.BN * 128;
    const int n_acc = a.chunks * a.BN <= 256 ? 2 : 1;
    if (tid == 0) {
        for (int s = 0; s < a.stages; s++) {
            mbar_init(bars + FULL + 8 * s, 1);
            mbar_init(bars + EMPTY + 8 * s, 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(bars + ACC_FULL + 8 * s, 1);
            mbar_init(bars + ACC_FREE + 8 * s, 8);
        }
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) tmem_alloc512(bars + SLOT);
    early_wait();
    const bool listed = GROUPED && a.n_groups <= kListed;
    if (listed && warp == 3) { // prefix sums of the groups' row tiles
        int sum = 0;
        for (int g0 = 0; g0 < a.n_groups; g0 += 32) {
            const int g = g0 + lane;
            int v = g < a.n_groups ? (a.m_ranges[g + 1] - a.m_ranges[g] + BM - 1) / BM : 0;
            for (int off = 1; off < 32; off *= 2) {
                const int o = __shfl_up_sync(0xffffffffu, v, off);
                if (lane >= off) v += o;
            }
            if (g < a.n_groups) first_tile[g + 1] = sum + v;
            sum += __shfl_sync(0xffffffffu, v, 31);
        }
        if (lane == 0) first_tile[0] = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    step_next();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<uint32_t *>(ctl + SLOT), 0);
    int row_tiles = a.m_tiles;
    if (listed) row_tiles = first_tile[a.n_groups];
    else if (GROUPED) {
        row_tiles = 0;
        for (int g = 0; g < a.n_groups; g++) row_tiles += (a.m_ranges[g + 1] - a.m_ranges[g] + BM - 1) / BM;
    }
    const int total = row_tiles * a.n_tiles * a.splits;
    auto locate = [&](int t) {
        tile_at r;
        r.group = 0;
        if (!GROUPED) { // row tiles first: those that share a piece of W run together
            r.m0 = t % a.m_tiles * BM;
            r.m_end = a.T;
            t /= a.m_tiles;
            r.n0 = t % a.n_tiles * a.BN;
            r.split = t / a.n_tiles;
            return r;
        }
        const int rt = t / a.n_tiles;
        r.n0 = (t - rt * a.n_tiles) * a.BN;
        r.split = 0;
        int f;
        if (listed) {
            int lo = 0, hi = a.n_groups - 1; // the last group whose first tile is not behind rt
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (first_tile[mid] <= rt) lo = mid;
                else hi = mid - 1;
            }
            r.group = lo;
            f = first_tile[lo];
        } else {
            f = 0;
            for (;; r.group++) {
                const int n = (a.m_ranges[r.group + 1] - a.m_ranges[r.group] + BM - 1) / BM;
                if (f + n > rt) break;
                f += n;
            }
        }
        r.m0 = a.m_ranges[r.group] + (rt - f) * BM;
        r.m_end = a.m_ranges[r.group + 1];
        return r;
    };
    auto k_range = [&](int split, int &kb0, int &kb1) {
        kb0 = split * a.chunks * a.chunk_kb;
        kb1 = min(kb0 + a.chunks * a.chunk_kb, a.kblocks);
    };

    if (warp == 0) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            for (int t = blockIdx.x; t < total; t += gridDim.x) {
                const tile_at at = locate(t);
                int kb0, kb1;
                k_range(at.split, kb0, kb1);
                for (int kb = kb0; kb < kb1; kb++) {
                    if (!mbar_wait_bounded(bars + EMPTY + 8 * s, ph ^ 1u, dead)) break;
                    const uint32_t sa = base + s * stage_bytes, bar = bars + FULL + 8 * s;
                    mbar_expect_tx(bar, stage_bytes);
                    tma_load_2d(sa, &map_a, kb * BK, at.m0, bar);
                    tma_load_2d(sa + a_bytes, &map_w, kb * BK, at.group * a.N + at.n0, bar);
                    if (++s == a.stages) s = 0, ph ^= 1u;
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        const uint32_t idesc = umma_idesc(128, a.BN);
        int s = 0, it = 0;
        uint32_t ph = 0;
        for (int t = blockIdx.x; t < total; t += gridDim.x, it++) {
            int kb0, kb1, chunk = 0, left = a.chunk_kb;
            k_range(locate(t).split, kb0, kb1);
            const int buf = n_acc == 2 ? it & 1 : 0, use = n_acc == 2 ? it >> 1 : it;
            mbar_wait_bounded(bars + ACC_FREE + 8 * buf, (use & 1) ^ 1, dead);
            tc_fence_after();
            for (int kb = kb0; kb < kb1; kb++) {
                mbar_wait_bounded(bars + FULL + 8 * s, ph, dead);
                tc_fence_after();
                const uint32_t a_lo = umma_desc_lo(base + s * stage_bytes, 16), w_lo = umma_desc_lo(base + s * stage_bytes + a_bytes, 16);
                const uint32_t first = left == a.chunk_kb ? 0u : 1u;
                const uint32_t d = tmem + buf * 256 + chunk * a.BN;
#pragma unroll
                for (int k = 0; k < BK / 16; k++) umma_ss(d, a_lo + 2 * k, w_lo + 2 * k, idesc, k > 0 ? 1u : first);
                umma_arrive(bars + EMPTY + 8 * s);
                if (++s == a.stages) s = 0, ph ^= 1u;
                if (--left == 0) chunk++, left = a.chunk_kb;
            }
            umma_arrive(bars + ACC_FULL + 8 * buf);
        }
    } else if (warp >= 4) {
        const int w8 = warp - 4, lq = warp & 3, half = w8 >> 2;
        const uint32_t my = turn + w8 * 4096;
        int it = 0;
        for (int t = blockIdx.x; t < total; t += gridDim.x, it++) {
            const tile_at at = locate(t);
            int kb0, kb1;
            k_range(at.split, kb0, kb1);
            const int chunks = (kb1 - kb0 + a.chunk_kb - 1) / a.chunk_kb; // the last CTA along K may have fewer
            const int buf = n_acc == 2 ? it & 1 : 0, use = n_acc == 2 ? it >> 1 : it;
            mbar_wait_warp(bars + ACC_FULL + 8 * buf, use & 1, dead);
            tc_fence_after();
            // a warp's 32 rows, every other 32 columns (the two warps of a quarter share them)
            const int row0 = at.m0 + lq * 32;
            if (row0 < at.m_end)
                for (int c0 = 32 * half; c0 < a.BN && at.n0 + c0 < a.N; c0 += 64)
                    store_piece(a, tmem + ((uint32_t)(lq * 32) << 16) + buf * 256 + c0, chunks, my, lane, row0, at.m_end, at.n0 + c0, at.split);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + ACC_FREE + 8 * buf);
        }
    }
    __syncthreads();
    if (warp == 2) {
        settle(dead);
        tc_fence_after();
        tmem_free512(tmem);
        if (lane == 0 && *dead) *a.wait_error = 1;
    }
}

// Two CTAs a tile of 256 rows and 256 columns: each holds 128 rows of A and of the accumulators and half of W's rows.  A single CTA
// reads A and W tiles of 12 KB from shared memory for an MMA of 128 cycles while TMA writes 64 bytes a cycle: 160 of the 128 bytes a cycle that
// shared memory has; a pair needs 112.  2048 x 8192 x 4096: 104 us, 1320 TFLOP/s (107 us single, 131 us before either); 1024 x 32000 x 2048: 109 us
// (125, 190 us).
__global__ void __launch_bounds__(kThreads, 1) gemm_pair_kernel(const __grid_constant__ pair_maps maps, const gemm_args a) {
    extern __shared__ uint8_t gm_raw[];
    const uint32_t raw0 = smem_u32(gm_raw), base = (raw0 + 1023u) & ~1023u, turn = base + kRing, bars = turn + kTurn;
    uint8_t *ctl = gm_raw + (bars - raw0);
    volatile int *dead = reinterpret_cast<volatile int *>(ctl + DEAD);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t rank = cluster_rank(), bars0 = cluster_addr(bars, 0);
    constexpr uint32_t a_bytes = BM * 128, stage_bytes = a_bytes + 16384;
    constexpr int kStages = (int)(kRing / stage_bytes);
    const int n_acc = a.chunks == 1 ? 2 : 1;
    if (tid == 0) {
        for (int s = 0; s < kStages; s++) {
            mbar_init(bars + FULL + 8 * s, 1);
            mbar_init(bars + EMPTY + 8 * s, 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(bars + ACC_FULL + 8 * s, 1);
            mbar_init(bars + ACC_FREE + 8 * s, 16); // eight warps of each CTA
        }
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) tmem_alloc512_pair(bars + SLOT);
    early_wait();
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    step_next();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<uint32_t *>(ctl + SLOT), 0);
    const int total = a.m_tiles * a.n_tiles * a.splits, pairs = gridDim.x / 2, me = blockIdx.x / 2;
    // row tiles first: those that share a piece of W run together
    auto locate = [&](int t, int &m0, int &n0, int &split) {
        m0 = t % a.m_tiles * (2 * BM);
        t /= a.m_tiles;
        n0 = t % a.n_tiles * 256;
        split = t / a.n_tiles;
    };
    auto k_range = [&](int split, int &kb0, int &kb1) {
        kb0 = split * a.chunks * a.chunk_kb;
        kb1 = min(kb0 + a.chunks * a.chunk_kb, a.kblocks);
    };
    if (warp == 0) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            for (int t = me; t < total; t += pairs) {
                int m0, n0, split, kb0, kb1;
                locate(t, m0, n0, split);
                k_range(split, kb0, kb1);
                for (int kb = kb0; kb < kb1; kb++) {
                    if (!mbar_wait_bounded(bars + EMPTY + 8 * s, ph ^ 1u, dead)) break;
                    const uint32_t sa = base + s * stage_bytes;
                    if (rank == 0) mbar_expect_tx(bars + FULL + 8 * s, 2 * stage_bytes);
                    tma_load_2d_pair(sa, &maps.a[0], kb * BK, m0 + (int)rank * BM, bars0 + FULL + 8 * s);
                    tma_load_2d_pair(sa + a_bytes, &maps.w, kb * BK, n0 + (int)rank * 128, bars0 + FULL + 8 * s);
                    if (++s == kStages) s = 0, ph ^= 1u;
                }
            }
            for (int k = 0; k < kStages && mbar_wait_bounded(bars + EMPTY + 8 * s, ph ^ 1u, dead); k++) // every arrival of the MMAs is here
                if (++s == kStages) s = 0, ph ^= 1u;
        }
        __syncwarp();
    } else if (warp == 1 && rank == 0) {
        const uint32_t idesc = umma_idesc(256, 256);
        int s = 0, it = 0;
        uint32_t ph = 0;
        for (int t = me; t < total; t += pairs, it++) {
            int m0, n0, split, kb0, kb1, chunk = 0, left = a.chunk_kb;
            locate(t, m0, n0, split);
            k_range(split, kb0, kb1);
            const int buf = n_acc == 2 ? it & 1 : 0, use = n_acc == 2 ? it >> 1 : it;
            mbar_wait_bounded(bars + ACC_FREE + 8 * buf, (use & 1) ^ 1, dead);
            tc_fence_after();
            for (int kb = kb0; kb < kb1; kb++) {
                mbar_wait_bounded(bars + FULL + 8 * s, ph, dead);
                tc_fence_after();
                const uint32_t a_lo = umma_desc_lo(base + s * stage_bytes, 16), w_lo = umma_desc_lo(base + s * stage_bytes + a_bytes, 16);
                const uint32_t first = left == a.chunk_kb ? 0u : 1u;
                const uint32_t d = tmem + buf * 256 + chunk * 256;
#pragma unroll
                for (int k = 0; k < BK / 16; k++) umma_ss_pair(d, a_lo + 2 * k, w_lo + 2 * k, idesc, k > 0 ? 1u : first);
                umma_arrive_pair(bars + EMPTY + 8 * s);
                if (++s == kStages) s = 0, ph ^= 1u;
                if (--left == 0) chunk++, left = a.chunk_kb;
            }
            umma_arrive_pair(bars + ACC_FULL + 8 * buf);
        }
        for (int k = 0; k < n_acc; k++, it++) { // and of the epilogues of both
            const int buf = n_acc == 2 ? it & 1 : 0, use = n_acc == 2 ? it >> 1 : it;
            mbar_wait_bounded(bars + ACC_FREE + 8 * buf, (use & 1) ^ 1, dead);
        }
    } else if (warp >= 4) {
        const int w8 = warp - 4, lq = warp & 3, half = w8 >> 2;
        int it = 0;
        for (int t = me; t < total; t += pairs, it++) {
            int m0, n0, split, kb0, kb1;
            locate(t, m0, n0, split);
            k_range(split, kb0, kb1);
            const int chunks = kb1 > kb0 ? (kb1 - kb0 + a.chunk_kb - 1) / a.chunk_kb : 0;
            const int buf = n_acc == 2 ? it & 1 : 0, use = n_acc == 2 ? it >> 1 : it;
            mbar_wait_warp(bars + ACC_FULL + 8 * buf, use & 1, dead);
            tc_fence_after();
            const int row0 = m0 + (int)rank * BM + lq * 32;
            if (row0 < a.T)
                for (int c0 = 32 * half; c0 < 256 && n0 + c0 < a.N; c0 += 64)
                    store_piece(a, tmem + ((uint32_t)(lq * 32) << 16) + buf * 256 + c0, chunks, turn + w8 * 4096, lane, row0, a.T, n0 + c0, split);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(bars0 + ACC_FREE + 8 * buf);
        }
    }
    warp_meet();
    __syncthreads();
    if (warp == 2) settle(dead);
    cluster_sync(); // neither gives its tensor memory back while the other one's MMAs or arrivals may still reach it
    if (warp == 2) {
        tc_fence_after();
        tmem_free512_pair(tmem);
        if (lane == 0 && *dead) *a.wait_error = 1;
    }
    cluster_sync(); // and neither leaves before the other one has
}

// The slots of a mixture of experts, sorted by group: C[slot][N] = A[slot][K] W[group of the slot][N][K]^T.  A pair of CTAs owns 256 features (the M of an MMA, half
// a CTA) x up to 256 slots of a group in equal tiles of a multiple of 32: so a group's matrix is read once whatever its slots, and no row is computed for nothing but
// the last 31.  A lane of tensor memory is a feature, so that 32 lanes store a line of a slot's row as they are.
//
// Rows of A come by TMA where they lie sorted.  Where they do not (row_src), three groups of four warps copy them through the slot
// list, which takes the stages in turn: a group hands one over when it has asked for its next (asking takes 500 cycles of a stage's 700, arriving 2500).
//
// Bound by memory, the matrices, and by the last round of tiles.  32 experts x 128 +- 11 slots, 1408 x 2048: 44.2 us a product from sorted rows (row tiles of 128
// slots x 256 features, in which half of the groups read their matrix twice: 47.0), 42.9 through the slot list (50.9 gathered ahead of it, 52 gathered ahead of this
// kernel, which is the slower way up to 4096 slots an expert); with GELU 44.6 (64.2).  TMA's gather of four rows takes 80 cycles: 80 us.  Where it is not the
// faster form: ggb_gemm_grouped_bf16_slots.
constexpr uint32_t kSlotStage = BM * 128 + 128 * 128;
constexpr int kSlotStages = 6, kMaxGroups = 8192;
constexpr int kCopyGroups = 3, kCopyWarps = 4, kSlotThreads = kThreads + 32 * kCopyWarps * kCopyGroups; // warps 12..: rows of A through the slot list
static_assert(kSlotStages == 2 * kCopyGroups, "a copying group has two places of the ring");
constexpr size_t kSlotSmem = 1024 + kSlotStages * kSlotStage + 256; // and the list of first tiles
static_assert(kSlotSmem >= kOneCtaSmem && kSlotSmem + 4 * (kMaxGroups + 1) <= 232448, "pairs of CTAs");

__global__ void __launch_bounds__(kSlotThreads, 1) gemm_slots_kernel(const __grid_constant__ pair_maps maps, const gemm_args a) {
    extern __shared__ uint8_t gm_raw[];
    __shared__ int warp_sum[kSlotThreads / 32];
    const uint32_t raw0 = smem_u32(gm_raw), base = (raw0 + 1023u) & ~1023u, bars = base + kSlotStages * kSlotStage;
    uint8_t *ctl = gm_raw + (bars - raw0);
    volatile int *dead = reinterpret_cast<volatile int *>(ctl + DEAD);
    int *first_tile = reinterpret_cast<int *>(ctl + 256); // [n_groups + 1]: the first slot tile of a group
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t rank = cluster_rank(), bars0 = cluster_addr(bars, 0);
    if (tid == 0) {
        for (int s = 0; s < kSlotStages; s++) {
            mbar_init(bars + FULL + 8 * s, a.row_src ? 1 + 2 * kCopyWarps : 1); // TMA, the copying warps of both CTAs
            mbar_init(bars + EMPTY + 8 * s, 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(bars + ACC_FULL + 8 * s, 1);
            mbar_init(bars + ACC_FREE + 8 * s, 16);
        }
        *dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) tmem_alloc512_pair(bars + SLOT);
    early_wait();
    { // prefix sums of the groups' slot tiles: a thread takes `each` neighbouring groups
        const int nt = blockDim.x, each = (a.n_groups + nt - 1) / nt, g0 = min(tid * each, a.n_groups), g1 = min(g0 + each, a.n_groups);
        int own = 0;
        for (int g = g0; g < g1; g++) own += (a.m_ranges[g + 1] - a.m_ranges[g] + 255) / 256;
        int sum = own;
        for (int off = 1; off < 32; off *= 2) {
            const int o = __shfl_up_sync(0xffffffffu, sum, off);
            if (lane >= off) sum += o;
        }
        if (lane == 31) warp_sum[warp] = sum;
        __syncthreads();
        sum -= own;
        for (int w = 0; w < warp; w++) sum += warp_sum[w];
        for (int g = g0; g < g1; g++) {
            first_tile[g] = sum;
            sum += (a.m_ranges[g + 1] - a.m_ranges[g] + 255) / 256;
        }
        if (tid == nt - 1) first_tile[a.n_groups] = sum;
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    step_next();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<uint32_t *>(ctl + SLOT), 0);
    const int total = first_tile[a.n_groups] * a.n_tiles, pairs = gridDim.x / 2, me = blockIdx.x / 2;
    struct slot_tile {
        int group, row0, rows, width, n0; // width: rows as a multiple of 32
    };
    auto locate = [&](int t) { // a group's features follow one another: its rows of A stay in L2
        slot_tile r;
        const int st = t / a.n_tiles;
        r.n0 = (t - st * a.n_tiles) * 256;
        int lo = 0, hi = a.n_groups - 1; // the last group whose first tile is not behind st
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (first_tile[mid] <= st) lo = mid;
            else hi = mid - 1;
        }
        const int f = first_tile[lo], n = first_tile[lo + 1] - f, g0 = a.m_ranges[lo], g1 = a.m_ranges[lo + 1];
        r.group = lo;
        r.width = ((g1 - g0 + n - 1) / n + 31) / 32 * 32;
        r.row0 = g0 + (st - f) * r.width;
        r.rows = min(r.width, g1 - r.row0);
        return r;
    };
    // one copy a stage and CTA for either operand (a thread takes 150 cycles for each): the box of A that covers half a tile, whose last rows may be the next
    // group's or behind the matrix: columns that nobody stores
    auto box_of = [](const slot_tile &at) { return (at.width / 2 + 31) / 32; };
    if (warp == 3) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 1;
            for (int t = me; t < total && !a.row_src; t += pairs) {
                const slot_tile at = locate(t);
                const CUtensorMap *map = &maps.a[box_of(at) - 1];
                const int r0 = at.row0 + (int)rank * (at.width / 2);
                for (int kb = 0; kb < a.kblocks; kb++) {
                    if (!mbar_wait_bounded(bars + EMPTY + 8 * s, ph, dead)) break;
                    tma_load_2d_pair(base + s * kSlotStage + BM * 128, map, kb * BK, r0, bars0 + FULL + 8 * s);
                    if (++s == kSlotStages) s = 0, ph ^= 1u;
                }
            }
        }
        __syncwarp();
    } else if (warp == 0) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 1;
            for (int t = me; t < total; t += pairs) {
                const slot_tile at = locate(t);
                const bool both = at.n0 + BM < a.N, mine = rank == 0 || both; // features behind the last one: not read, not stored
                for (int kb = 0; kb < a.kblocks; kb++) {
                    if (!mbar_wait_bounded(bars + EMPTY + 8 * s, ph, dead)) break;
                    if (rank == 0) mbar_expect_tx(bars + FULL + 8 * s, (both ? 2 * BM * 128 : BM * 128) + (a.row_src ? 0 : 2 * box_of(at) * 32 * 128));
                    if (mine) tma_load_2d_pair(base + s * kSlotStage, &maps.w, kb * BK, at.group * a.N + at.n0 + (int)rank * BM, bars0 + FULL + 8 * s);
                    if (++s == kSlotStages) s = 0, ph ^= 1u;
                }
            }
            for (int k = 0; k < kSlotStages && mbar_wait_bounded(bars + EMPTY + 8 * s, ph, dead); k++) // every arrival of the MMAs is here
                if (++s == kSlotStages) s = 0, ph ^= 1u;
        }
        __syncwarp();
    } else if (warp == 1 && rank == 0) {
        int s = 0, it = 0;
        uint32_t ph = 0;
        for (int t = me; t < total; t += pairs, it++) {
            const uint32_t idesc = umma_idesc(256, locate(t).width), buf = it & 1;
            mbar_wait_bounded(bars + ACC_FREE + 8 * buf, ((it >> 1) & 1) ^ 1, dead);
            tc_fence_after();
            for (int kb = 0; kb < a.kblocks; kb++) {
                mbar_wait_bounded(bars + FULL + 8 * s, ph, dead);
                tc_fence_after();
                const uint32_t at = base + s * kSlotStage;
                umma_ss_pair_k4(tmem + buf * 256, umma_desc_lo(at, 16), umma_desc_lo(at + BM * 128, 16), idesc, kb > 0);
                umma_arrive_pair(bars + EMPTY + 8 * s);
                if (++s == kSlotStages) s = 0, ph ^= 1u;
            }
            umma_arrive_pair(bars + ACC_FULL + 8 * buf);
        }
        for (int k = 0; k < 2; k++, it++) mbar_wait_bounded(bars + ACC_FREE + 8 * (it & 1), ((it >> 1) & 1) ^ 1, dead); // and of the epilogues of both
    } else if (warp >= 12) {
        // stages grp, grp + 3, ... of all of this CTA's, into two places of the ring: a thread copies one 16-byte piece of every 16th row
        const int grp = (warp - 12) / kCopyWarps, lt = (tid - kThreads) % (32 * kCopyWarps), pc = lt & 7, r0 = lt >> 3;
        int next = grp, n = 0; // its next stage, counted from the tile's first; stages asked for
        auto give = [&](int k) {
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(bars0 + FULL + 8 * (grp + kCopyGroups * (k & 1)));
        };
        bool going = true; // a wait that gave up ends all of its tiles: `next` is then no stage of the following one
        for (int t = me; going && t < total; t += pairs, next -= a.kblocks) {
            if (next >= a.kblocks) continue;
            const slot_tile at = locate(t);
            const int h0 = (int)rank * (at.width / 2), mine = min(at.width / 2, at.rows - h0); // this CTA's half of the tile (none: not above 0)
            const __nv_bfloat16 *from[8];
#pragma unroll
            for (int i = 0; i < 8; i++) from[i] = a.a + (int64_t)a.row_src[at.row0 + min(h0 + r0 + 16 * i, at.rows - 1)] * (a.kblocks * BK) + 8 * pc;
            for (; next < a.kblocks; next += kCopyGroups, n++) {
                const int s = grp + kCopyGroups * (n & 1);
                if (!(going = mbar_wait_warp(bars + EMPTY + 8 * s, ((n >> 1) & 1) ^ 1, dead))) break;
#pragma unroll
                for (int i = 0; i < 8; i++) // rows 16 apart lie at the same place of the swizzle; those behind the last stay as they are: columns that nobody stores
                    if (r0 + 16 * i < mine) cp_async16(base + s * kSlotStage + (BM + r0 + 16 * i) * 128 + ((pc ^ (r0 & 7)) << 4), from[i] + next * BK);
                cp_async_commit();
                if (n > 0) {
                    cp_async_wait<1>();
                    give(n - 1);
                }
            }
        }
        cp_async_wait<0>();
        if (going && n > 0) give(n - 1);
    } else if (warp >= 4) {
        const int lq = warp & 3, half = (warp - 4) >> 2;
        int it = 0;
        for (int t = me; t < total; t += pairs, it++) {
            const slot_tile at = locate(t);
            const uint32_t buf = it & 1;
            mbar_wait_warp(bars + ACC_FULL + 8 * buf, (it >> 1) & 1, dead);
            tc_fence_after();
            const int n = at.n0 + (int)rank * BM + lq * 32 + lane; // N is a multiple of 32: a warp's features are all there or none
            if (n < a.N)
                for (int c0 = 32 * half; c0 < at.rows; c0 += 64) {
                    uint32_t v[32];
                    tmem_load32(tmem + ((uint32_t)(lq * 32) << 16) + buf * 256 + c0, v);
                    const int64_t row = at.row0 + c0;
                    if (a.act_out) { // two slots at a time: an even lane stores its and its neighbour's feature of the first one, an odd lane of the second
                        __nv_bfloat16 *dst = a.act_out + (row + (lane & 1)) * a.ldc + (n & ~1);
                        const int left = at.rows - c0 - (lane & 1);
                        if (a.act == GGB_ACT_GELU_ERF) {
#pragma unroll
                            for (int c = 0; c < 32; c++) v[c] = __float_as_uint(act_f32(__uint_as_float(v[c]), GGB_ACT_GELU_ERF));
                        } else {
#pragma unroll
                            for (int c = 0; c < 32; c++) v[c] = __float_as_uint(act_f32(__uint_as_float(v[c]), a.act));
                        }
#pragma unroll
                        for (int c = 0; c < 32; c += 2) {
                            const float x = __uint_as_float(v[c]), y = __uint_as_float(v[c + 1]), o = __shfl_xor_sync(0xffffffffu, lane & 1 ? x : y, 1);
                            if (c < left) *reinterpret_cast<uint32_t *>(dst + c * a.ldc) = lane & 1 ? pack_bf16x2(o, y) : pack_bf16x2(x, o);
                        }
                    } else {
                        float *dst = a.c + row * a.ldc + n;
#pragma unroll
                        for (int c = 0; c < 32; c++)
                            if (c0 + c < at.rows) dst[c * a.ldc] = __uint_as_float(v[c]);
                    }
                }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(bars0 + ACC_FREE + 8 * buf);
        }
    }
    warp_meet();
    __syncthreads();
    if (warp == 2) settle(dead);
    cluster_sync(); // neither gives its tensor memory back while the other one's MMAs or arrivals may still reach it
    if (warp == 2) {
        tc_fence_after();
        tmem_free512_pair(tmem);
        if (lane == 0 && *dead) *a.wait_error = 1;
    }
    cluster_sync(); // and neither leaves before the other one has
}

// the CTAs' sums along K in order
__global__ void splits_add_kernel(const float *__restrict__ ws, int splits, int64_t T, int64_t N, float *__restrict__ c, __nv_bfloat16 *__restrict__ act_out, int act,
                                  int64_t ldc) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4; // N is a multiple of 4
    if (i >= T * N) return;
    const int64_t t = i / N, n = i - t * N;
    float4 s = *reinterpret_cast<const float4 *>(ws + i);
    for (int k = 1; k < splits; k++) {
        const float4 v = *reinterpret_cast<const float4 *>(ws + (int64_t)k * T * N + i);
        s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
    }
    const float o[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int u = 0; u < 4; u++) {
        if (act_out) act_out[t * ldc + n + u] = __float2bfloat16_rn(act_f32(o[u], act));
        else c[t * ldc + n + u] = o[u];
    }
}

int launch_pair(const void *w, int64_t w_rows, int64_t K, const void *a, int64_t a_rows, const gemm_args &g, int pairs) {
    pair_maps maps;
    auto kern = g.m_ranges ? gemm_slots_kernel : gemm_pair_kernel;
    const size_t pair_smem = std::max(kOneCtaSmem, g.m_ranges ? kSlotSmem + 4 * ((size_t)g.n_groups + 1) : kSmem);
    int rc = ggb_allow_smem(kern, g.m_ranges ? kSlotSmem + 4 * (kMaxGroups + 1) : kSmem);
    if (!rc) rc = ggb_tensor_map_bf16(&maps.w, w, w_rows, K, K, 128);
    for (int i = 0; i < (g.row_src ? 0 : g.m_ranges ? 4 : 1) && !rc; i++) rc = ggb_tensor_map_bf16(&maps.a[i], a, a_rows, K, K, g.m_ranges ? 32 * (i + 1) : BM);
    if (rc) return rc;
    GGB_CUDA(ggb_launch_early(kern, ggb_cluster{2, 1, 1}, dim3((unsigned)(2 * std::min(pairs, ggb_sm_count() / 2))), dim3(g.row_src ? kSlotThreads : kThreads), pair_smem, maps, g));
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int launch(const void *w, int64_t w_rows, int64_t K, const void *a, int64_t a_rows, const gemm_args &g, int ctas) {
    CUtensorMap ma, mw;
    auto kern = g.m_ranges ? gemm_tma_kernel<true> : gemm_tma_kernel<false>;
    int rc = ggb_allow_smem(kern, kSmem);
    if (!rc) rc = ggb_tensor_map_bf16(&ma, a, a_rows, K, K, BM);
    if (!rc) rc = ggb_tensor_map_bf16(&mw, w, w_rows, K, K, g.BN);
    if (rc) return rc;
    GGB_CUDA(ggb_launch_early(kern, ggb_cluster{1, 1, 1}, dim3((unsigned)std::min(ctas, ggb_sm_count())), dim3(kThreads), kSmem, ma, mw, g));
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

int stages_of(int BN) { return std::min<int>(kMaxStages, (int)(kRing / (uint32_t)((BM + BN) * 128))); }

} // namespace

static int tensor_map_2d(CUtensorMap *map, CUtensorMapDataType type, CUtensorMapSwizzle swizzle, const void *base, int64_t rows, int64_t cols, int64_t pitch_bytes, int box_cols,
                         int box_rows) {
    typedef CUresult (*encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static encode_fn encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult qr;
        GGB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr));
        GGB_CHECK_ARG(fn && qr == cudaDriverEntryPointSuccess, "cuTensorMapEncodeTiled is not in the driver");
        encode = (encode_fn)fn;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, pitch[1] = {(cuuint64_t)pitch_bytes};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, step[2] = {1, 1};
    const CUresult r = encode(map, type, 2, const_cast<void *>(base), dims, pitch, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    GGB_CHECK_ARG(r == CUDA_SUCCESS, "tensor map of %lld x %lld numbers, pitch %lld bytes: error %d", (long long)rows, (long long)cols, (long long)pitch_bytes, (int)r);
    return GGB_OK;
}
int ggb_tensor_map_bf16(CUtensorMap_st *map, const void *base, int64_t rows, int64_t cols, int64_t ld, int box_rows) {
    return tensor_map_2d(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, CU_TENSOR_MAP_SWIZZLE_128B, base, rows, cols, ld * 2, 64, box_rows);
}
int ggb_tensor_map_bytes(CUtensorMap_st *map, const void *base, int64_t rows, int64_t row_bytes, int box_bytes, int box_rows) {
    return tensor_map_2d(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, CU_TENSOR_MAP_SWIZZLE_NONE, base, rows, row_bytes, row_bytes, box_bytes, box_rows);
}

bool ggb_gemm_dense_bf16_fits(int64_t N, int64_t K, int64_t T, int64_t ldc) {
    return T >= 64 && K % 64 == 0 && N % 32 == 0 && ldc % 4 == 0 && N < (1ll << 31) && K < (1ll << 31) && T < (1ll << 31);
}

// The K-split workspace only grows (one stream).
int ggb_gemm_dense_bf16(const void *w, int64_t N, int64_t K, const void *a, int64_t T, float *c, int64_t ldc, void *c_act, int act) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(w && a && (c || c_act) && ((uintptr_t)w | (uintptr_t)a) % 16 == 0, "gemm: operands start on 16 bytes");
    GGB_CHECK_ARG(!c_act || ldc % 8 == 0, "gemm: an activation takes rows of whole 16-byte pieces");
    const int sms = ggb_sm_count(), kblocks = (int)(K / BK), pieces = ggb_gemm_pieces(T, N, K);
    gemm_args g{};
    double best = 0.0;
    int pair = -1; // two CTAs a tile
    // (256 rows a CTA never have the least estimate: half as many tiles, whose stages take twice as long and more)
    static const struct {
        int bn, pair;
    } shapes[] = {{256, 1}, {256, 0}, {128, 0}, {64, 0}};
    for (const auto &sh : shapes)
        for (int splits = 1; splits <= pieces; splits *= 2) {
            const int chunks = pieces / splits;
            if (chunks * sh.bn > 512) continue;
            const int chunk_kb = (kblocks + pieces - 1) / pieces, cs = 1 + sh.pair, rows = BM * cs;
            const int64_t m_tiles = (T + rows - 1) / rows, n_tiles = (N + sh.bn - 1) / sh.bn, tiles = m_tiles * n_tiles * splits;
            // cycles of a stage: its MMAs, or the bytes that pass through shared memory at 128 a cycle (written by TMA, read for the MMAs); a round of
            // tiles: its stages and, unless the next tile runs meanwhile, its stores
            const double mma = std::max(sh.bn, 96) * 2.0, smem = ((BM + sh.bn / cs) * 128.0 + 4 * (4096.0 + sh.bn * 32.0 / cs)) / 128.0;
            const double stage = std::max(mma, smem), store = BM * sh.bn / 12.0;
            const double rounds = (double)((tiles + sms / cs - 1) / (sms / cs));
            double cost = rounds * (chunks * chunk_kb * stage + (chunks * sh.bn > 256 ? store : 0.0)) + store + 2000.0;
            if (splits > 1) cost += 12000.0 + (double)splits * T * N * 8.0 / (32.0 * sms); // another launch, the sums' way through memory
            cost += sh.pair ? 4000.0 : 0.0;                                               // a cluster's launch
            if (pair < 0 || cost < best) {
                best = cost;
                pair = sh.pair;
                g.BN = sh.bn, g.n_tiles = (int)n_tiles, g.m_tiles = (int)m_tiles, g.chunks = chunks, g.chunk_kb = chunk_kb, g.splits = splits;
            }
        }
    // sized by T and N alone, for every product that some K would cut: where one of them has run, a captured one allocates nothing
    void *ws = nullptr;
    if ((N + 255) / 256 * ((T + 255) / 256) * 2 <= sms) {
        const int e = ggb_workspace(GGB_WS_GEMM_SPLITS, ggb_gemm_workspace_bytes(T, N, K), &ws);
        if (e) return e;
    }
    if (g.splits > 1) g.ws = (float *)ws;
    g.T = (int)T, g.N = (int)N, g.kblocks = kblocks, g.stages = stages_of(g.BN);
    g.c = c, g.act_out = (__nv_bfloat16 *)c_act, g.act = act, g.ldc = ldc;
    g.vec = g.ws || ((uintptr_t)c % 16 == 0 && ldc % 4 == 0);
    g.wait_error = ggb_wait_error_flag();
    const int tiles = g.m_tiles * g.n_tiles * g.splits, rc = pair ? launch_pair(w, N, K, a, T, g, tiles) : launch(w, N, K, a, T, g, tiles);
    if (rc || g.splits == 1) return rc;
    splits_add_kernel<<<(unsigned)((T * N / 4 + 255) / 256), 256, 0, ggb_cuda_stream()>>>(g.ws, g.splits, T, N, c, g.act_out, act, ldc);
    GGB_LAUNCH_CHECK();
    return GGB_OK;
}

static int rows_tile_n(int64_t N) { return N <= 64 ? 64 : N <= 128 ? 128 : 256; }
// The grouped forms: w = [n_exp][N][K], rows of c in sorted-slot order, offsets[e] .. offsets[e + 1] those of expert e (device), row_src their rows of a (or
// null: the same)
bool ggb_gemm_grouped_bf16_fits(int64_t N, int64_t K, int64_t ldc) { return K % 64 == 0 && N % 32 == 0 && ldc % 8 == 0; }

// Which of the two forms, by the least estimated time in microseconds: the rounds of tiles, each K / 64 stages and its stores, or the bytes.  The counts of a router's
// groups are taken to spread by about their square root.  The figures are fitted to 6752 calls (4 to 128 groups of 32 to 2048 rows, N 64 to 2048, K 256 to 2048, sums and GELU, rows sorted or
// not, gates of 2 to 32 equal blocks): the chosen form is 0.5 % above the better one on the average, 11 % at the 99th percentile (always tiles of slots: 17 %, of rows: 9 %).  They
// differ by up to a factor of two either way: a pair of CTAs takes 256 features whatever N is (8 x 2048 rows, 64 x 1024, sorted: tiles of rows 7.4 us, of slots 14.9; 8 x 64 rows,
// 256 x 2048: 15.6, 11.7), half as many tiles leave half of the chip out (8 x 512 rows, 1024 x 2048: 19.8, 29.3) or read a matrix once where two read it (64 x 256
// rows, 1408 x 2048: 159, 116).
bool ggb_gemm_grouped_bf16_slots(int64_t N, int64_t K, int64_t n_rows, int n_exp, bool equal, bool gather, bool act) {
    if (n_exp > kMaxGroups || n_exp * N >= (1ll << 31)) return false;
    // in a capture that the workspace of the copied rows would have to grow in: up to 256 rows a group in the form that needs none, beyond that refused if that is not the faster one
    if (gather && n_rows <= 256 * (int64_t)n_exp && !ggb_workspace_fits(GGB_WS_MOE_GATHER, (size_t)n_rows * (size_t)K * 2)) return true;
    const double per = (double)n_rows / n_exp, spread = equal ? 0 : 0.75 * std::sqrt(per), kb = (double)(K / BK), sms = ggb_sm_count();
    auto tiles = [&](double size) { return (std::max(1.0, std::ceil((per - spread) / size)) + std::max(1.0, std::ceil((per + spread) / size))) / 2; };
    const double BN = rows_tile_n(N), mb = 1e-6 * ((double)n_exp * N * K * 2 + (double)n_rows * N * (act ? 2 : 4));
    const double width = std::min(256.0, 32 * std::ceil(per / tiles(256) / 32));
    const double rounds_r = std::ceil(n_exp * tiles(BM) * std::ceil(N / BN) / sms - 0.02), rounds_s = std::ceil(n_exp * tiles(256) * std::ceil(N / 256.0) / (sms / 2) - 0.02);
    const double rows = std::max(2.6 + rounds_r * (kb * (0.095 + 0.0007 * BN) + (act ? 0.034 : 0.022) * BN), 2.6 + 0.24 * mb) + (gather ? 1.1 + 0.55e-6 * n_rows * K : 0);
    const double slots = (gather ? 5.7 : 5) + std::max(rounds_s * (0.158 * kb + (act ? 0.052 * width : 0.3 + 0.033 * width)), 0.163 * mb);
    return slots < rows;
}
int ggb_gemm_grouped_bf16(bool slots, const void *w, int64_t N, int64_t K, const void *a, int64_t n_rows, int n_exp, const int32_t *offsets, const int32_t *row_src,
                          float *c, void *c_act, int act, int64_t ldc) {
    GGB_REQUIRE_INIT();
    GGB_CHECK_ARG(((uintptr_t)w | (uintptr_t)a) % 16 == 0, "gemm: operands start on 16 bytes");
    gemm_args g{};
    g.T = (int)n_rows, g.N = (int)N, g.kblocks = (int)(K / BK);
    g.m_ranges = offsets, g.n_groups = n_exp;
    g.c = c, g.act_out = (__nv_bfloat16 *)c_act, g.act = act, g.ldc = ldc;
    g.wait_error = ggb_wait_error_flag();
    if (!slots) {
        g.BN = rows_tile_n(N), g.n_tiles = (int)((N + g.BN - 1) / g.BN);
        g.chunks = 1, g.chunk_kb = g.kblocks, g.splits = 1, g.stages = stages_of(g.BN), g.vec = (uintptr_t)c % 16 == 0;
        const int64_t most = ((n_rows + BM - 1) / BM + n_exp) * g.n_tiles;
        return launch(w, (int64_t)n_exp * N, K, a, n_rows, g, (int)std::min<int64_t>(most, 1 << 20));
    }
    g.n_tiles = (int)((N + 255) / 256), g.row_src = row_src, g.a = (const __nv_bfloat16 *)a;
    const int64_t most = (n_rows / 256 + std::min<int64_t>(n_rows, n_exp)) * g.n_tiles;
    return launch_pair(w, (int64_t)n_exp * N, K, a, n_rows, g, (int)std::min<int64_t>(most, 1 << 20));
}
