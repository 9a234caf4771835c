// tc.cuh — tensor-core plumbing of the sm_100a kernels: mbarriers with bounded waits, shared-memory matrix descriptors, tcgen05
// instructions and tensor-memory loads and stores.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

// set by a kernel whose wait ran out (host-mapped, checked by ggb_sync): a wait that ends so is an error in the program, never a
// matter of timing
int *ggb_wait_error_flag();

// a tensor map over a row-major bf16 matrix [rows][cols] with row pitch ld (numbers): boxes of 64 columns x box_rows, 128-byte swizzle
struct CUtensorMap_st;
int ggb_tensor_map_bf16(CUtensorMap_st *map, const void *base, int64_t rows, int64_t cols, int64_t ld, int box_rows);
// over rows of bytes: boxes of box_bytes x box_rows, as they lie
int ggb_tensor_map_bytes(CUtensorMap_st *map, const void *base, int64_t rows, int64_t row_bytes, int box_bytes, int box_rows);

#ifdef __CUDACC__

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.b32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// The same without waiting: asked ahead, so that a warp does not stand for the hundred cycles and more that an answer takes
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.b32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Waits for a phase.  Every wait ends: after kWaitTries tries (seconds) the CTA's `dead` word is set, which ends all of its other
// waits at once; the kernel then requests no more copies, runs through with whatever is in its buffers, gives what it has requested time to
// arrive (settle), gives its tensor memory back and reports the failure.  By one lane, or by a warp that only issues MMAs, whose lanes meet in
// every election (elect.sync), of which one lane goes on:
constexpr int kWaitTries = 1 << 21;
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, volatile int *dead) { // false: given up
    if (mbar_try(bar, parity)) return true;
    for (int i = 0; i < kWaitTries; i++) {
        if (mbar_try(bar, parity)) return true;
        if (*dead) return false;
    }
    *dead = 1;
    return false;
}
// By a warp whose lanes all go on.  Every lane asks and a vote decides, so that the lanes leave the wait together, each with an answer of its own: what a warp
// reads or writes behind it may be handed on by one lane's arrival, and instructions of a converged warp (loads of tensor memory) may follow.  Where
// every lane leaves by its own answer, that rests on no branch ahead having parted the lanes: a kernel that waited so lost numbers, its
// buffers were refilled while the last lanes read them.  Where one lane asks for all, the others come out of the barrier of the warp apart
// from it (in every one of 5100 waits for a late copy, by up to 250 cycles, and the warp stays parted: 429 against 364 cycles an item); with
// the vote never, at 363 cycles.  (In the warps that issue MMAs, too: attention of 1024 tokens 44.0 us; 41.9.)
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *dead) { // false: given up
    if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
    for (int i = 0; i < kWaitTries; i++) {
        if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
        if (__any_sync(0xffffffffu, *dead)) return false;
    }
    *dead = 1;
    return false;
}
// Behind a wait that ran out: copies and MMAs may still be under way, and what they write stays this CTA's for another half second.  By one
// warp, when all of them are done.
__device__ __forceinline__ void settle(volatile int *dead) {
    if (*dead)
        for (int i = 0; i < 500; i++) __nanosleep(1000000);
}

// Shared memory of which an SM has room for one CTA.  The CTAs of a cluster that allocate tensor memory ask for at least this much: with two on an SM, a
// cluster could wait on one SM for the tensor memory that another one holds, which on a second SM waits for what this one holds.
constexpr size_t kOneCtaSmem = 116 * 1024;

// Shared-memory matrix operands, 128-byte swizzle: rows of 128 bytes, 16-byte piece c of row r at place c ^ (r & 7), 1024-byte atoms
// of 8 rows that follow one another.  K-major: rows are M / N.  MN-major: rows are K, a row holds 64 numbers of M / N, and lbo is the
// distance between blocks of 64 numbers of M / N.  A descriptor's upper half (distance of the atoms, version, swizzle) is the same for
// all of them; the lower one holds the address and lbo.
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t saddr, uint32_t lbo) { return ((saddr & 0x3FFFFu) >> 4) | ((lbo >> 4) << 16); }
constexpr uint32_t kUmmaDescHi = (1024u >> 4) | (1u << 14) | (2u << 29); // 1024 bytes between atoms, sm_100, 128-byte swizzle
// instruction descriptor, kind::f16: fp32 accumulators, A and B bf16, A K-major, B K-major or (b_mn) MN-major
__device__ __forceinline__ constexpr uint32_t umma_idesc(int M, int N, bool b_mn = false) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn ? 1u << 16 : 0u) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// MMAs are issued by a whole converged warp, of which the elected lane acts: descriptors and addresses then stay in uniform registers
// (an `if (lane == 0)` around the loop costs a move per operand and MMA, more than a small MMA takes)
#define GGB_ELECT "elect.sync _|e, 0xffffffff;\n"
__device__ __forceinline__ void umma_ss(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p, e;\n.reg .b64 a, b;\n" GGB_ELECT "setp.ne.b32 p, %4, 0;\nmov.b64 a, {%1, %5};\nmov.b64 b, {%2, %5};\n"
                 "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n}\n" ::"r"(tmem_d),
                 "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(kUmmaDescHi)
                 : "memory");
}
// The four steps of a block of 64 along K (K-major operands: 32 bytes further each) under one election
#define GGB_K4(G) "{\n.reg .pred p, q, e;\n.reg .b64 a, b;\n" GGB_ELECT "setp.ne.b32 p, %4, 0;\nsetp.eq.b32 q, %4, %4;\nmov.b64 a, {%1, %5};\nmov.b64 b, {%2, %5};\n" \
    "@e tcgen05.mma.cta_group::" G ".kind::f16 [%0], a, b, %3, p;\nadd.s64 a, a, 2;\nadd.s64 b, b, 2;\n" \
    "@e tcgen05.mma.cta_group::" G ".kind::f16 [%0], a, b, %3, q;\nadd.s64 a, a, 2;\nadd.s64 b, b, 2;\n" \
    "@e tcgen05.mma.cta_group::" G ".kind::f16 [%0], a, b, %3, q;\nadd.s64 a, a, 2;\nadd.s64 b, b, 2;\n" \
    "@e tcgen05.mma.cta_group::" G ".kind::f16 [%0], a, b, %3, q;\n}\n"
__device__ __forceinline__ void umma_ss_k4(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(GGB_K4("1") ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(kUmmaDescHi) : "memory");
}
// A from tensor memory: row = lane, a 32-bit column holds two neighbours of K
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p, e;\n.reg .b64 b;\n" GGB_ELECT "setp.ne.b32 p, %4, 0;\nmov.b64 b, {%2, %5};\n"
                 "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, p;\n}\n" ::"r"(tmem_d),
                 "r"(tmem_a), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(kUmmaDescHi)
                 : "memory");
}
__device__ __forceinline__ void umma_arrive(uint32_t bar) { // arrives when all MMAs issued so far are done
    asm volatile("{\n.reg .pred e;\n" GGB_ELECT "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar) : "memory");
}

// Two CTAs of a cluster on one tile (cta_group::2): M = 256, the rows of A and of the accumulators half in each CTA, the rows of B (columns of
// the tile) half in each CTA's shared memory at the same offsets.  The CTA of rank 0 issues; a commit arrives on both CTAs' barriers.
__device__ __forceinline__ void umma_ss_pair(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p, e;\n.reg .b64 a, b;\n" GGB_ELECT "setp.ne.b32 p, %4, 0;\nmov.b64 a, {%1, %5};\nmov.b64 b, {%2, %5};\n"
                 "@e tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n}\n" ::"r"(tmem_d),
                 "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(kUmmaDescHi)
                 : "memory");
}
__device__ __forceinline__ void umma_ss_pair_k4(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(GGB_K4("2") ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(kUmmaDescHi) : "memory");
}
#undef GGB_K4
__device__ __forceinline__ void umma_arrive_pair(uint32_t bar) {
    asm volatile("{\n.reg .pred e;\n" GGB_ELECT "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}\n" ::"r"(bar),
                 "h"((uint16_t)3)
                 : "memory");
}
#undef GGB_ELECT
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t smem, uint32_t rank) { // the same offset in another CTA's shared memory
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem), "r"(rank));
    return r;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ double ld_cluster_f64(uint32_t addr) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
    return v;
}
// The lanes of a warp together again: behind waits that each lane leaves by its own answer, and behind an `if (lane == 0)`, they may be apart for as long as nothing
// joins them (a barrier of the warp does not, a vote does).  Ahead of every barrier of a CTA or cluster that such a warp comes to: one that is executed by parts of a warp
// counts it twice, and then lets CTAs go on, or leave, ahead of others that still reach them.
__device__ __forceinline__ void warp_meet() { asm volatile("{\n.reg .pred p, q;\nsetp.eq.u32 p, 0, 0;\nvote.sync.all.pred q, p, 0xffffffff;\n}" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() {
    warp_meet();
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
    cluster_arrive();
    cluster_wait();
}
// An arrival on another CTA's barrier.  What it announces lies in this CTA's own shared or tensor memory and is read there by the tensor
// cores, behind this CTA's proxy fence and barrier: no release at cluster scope, which would flush for a microsecond.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void tmem_alloc512_pair(uint32_t slot) { // one warp of each CTA
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(slot) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free512_pair(uint32_t base) {
    warp_meet();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(base) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

#define GGB_R8(v, o) "=r"(v[o]), "=r"(v[o + 1]), "=r"(v[o + 2]), "=r"(v[o + 3]), "=r"(v[o + 4]), "=r"(v[o + 5]), "=r"(v[o + 6]), "=r"(v[o + 7])
#define GGB_S8(v, o) "r"(v[o]), "r"(v[o + 1]), "r"(v[o + 2]), "r"(v[o + 3]), "r"(v[o + 4]), "r"(v[o + 5]), "r"(v[o + 6]), "r"(v[o + 7])
// 32 lanes x 16 (32, 8) columns.  A load and the wait for it are one statement: no use of a register can move in front of it
__device__ __forceinline__ void tmem_load16(uint32_t taddr, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 "tcgen05.wait::ld.sync.aligned;"
                 : GGB_R8(v, 0), GGB_R8(v, 8)
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_load32(uint32_t taddr, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, "
                 "%24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
                 "tcgen05.wait::ld.sync.aligned;"
                 : GGB_R8(v, 0), GGB_R8(v, 8), GGB_R8(v, 16), GGB_R8(v, 24)
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_store16(uint32_t taddr, const uint32_t *v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr), GGB_S8(v, 0),
                 GGB_S8(v, 8)
                 : "memory");
}
__device__ __forceinline__ void tmem_store8(uint32_t taddr, const uint32_t *v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), GGB_S8(v, 0) : "memory");
}
#undef GGB_R8
#undef GGB_S8
// all 512 columns (one CTA a SM), by one warp
__device__ __forceinline__ void tmem_alloc512(uint32_t slot) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(slot) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free512(uint32_t base) { // by the warp that issued MMAs, often, whose lanes may be apart
    warp_meet();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(base) : "memory");
}

// TMA: a box of a 2-dimensional tensor map, x (a multiple of 16 bytes) and y of its first element, to shared memory; out-of-range elements
// arrive as zeros.  One thread.
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}

// the same from a CTA of a pair, whose bytes count on the barrier of the CTA of rank 0 (a cluster address)
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void *map, int x, int y, uint32_t cluster_bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y),
                 "r"(cluster_bar)
                 : "memory");
}
// untiled: bytes (a multiple of 16) between 16-byte boundaries.  One thread.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// two fp32 numbers in one register pair: one instruction for both where the issue of instructions is what bounds a loop
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float ex2_approx(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Attention with soft-max counts its scores in powers of two: the queries are multiplied by log2 e, so that a weight is 2^(s - m) by the unit that
// computes it, as exact as expf of the difference and without its product (which, rounded and left at that, moves a weight by up to
// |s - m| 2^-24 of itself).
constexpr double kLog2E = 1.4426950408889634074; // 1 / ln 2
constexpr float kLog2e = (float)kLog2E, kLog2eRest = (float)(kLog2E - (double)kLog2e), kLn2 = 0.69314718055994530942f;
// 2^m over e^nat: for sums that are relative to m, counted in powers of two, where others are relative to nat.  What nat's rounding left of m is kept
// (a multiply-add is exact where its terms nearly cancel).
__device__ __forceinline__ float over_e(float m, float nat) { return m == -INFINITY ? 0.f : exp2f(fmaf(-nat, kLog2eRest, fmaf(-nat, kLog2e, m))); }

// Two fp32 numbers as three pairs of bf16 numbers whose sums they are: 3 x 8 significant bits hold the 24 of an fp32 number, each
// remainder is exact (and taken two at a time).  An fp32 x bf16 product is then three bf16 x bf16 products of the tensor cores, each exact before it is added.
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&p);
}
__device__ __forceinline__ void split3(f32x2 v, uint32_t &h, uint32_t &m, uint32_t &l) {
    const f32x2 minus = pack2(-1.f, -1.f);
    float2 x = unpack2(v);
    h = pack_bf16x2(x.x, x.y);
    v = fma2(pack2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u)), minus, v);
    x = unpack2(v);
    m = pack_bf16x2(x.x, x.y);
    v = fma2(pack2(__uint_as_float(m << 16), __uint_as_float(m & 0xffff0000u)), minus, v);
    x = unpack2(v);
    l = pack_bf16x2(x.x, x.y);
}
#endif
