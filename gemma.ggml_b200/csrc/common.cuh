// common.cuh — shared device helpers and the library context for libggb_cuda.so (sm_100a).
// Compiled with -fmad=false: every fp32 expression rounds once per operator unless it
// spells fmaf()/__fmaf_rn() explicitly, so the kernels' arithmetic matches the oracle's.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/ggml_b200.h"

#define GGB_QK 32

// ---- error plumbing -------------------------------------------------------
void ggb_set_error(const char *fmt, ...);
bool ggb_is_init();
cudaStream_t ggb_cuda_stream();
void ggb_count_launch(int n = 1);
// What is kept from call to call belongs to the context (ggb_shutdown gives it back; a later ggb_init, of another device perhaps, starts
// without it): device memory that only grows, its content not kept, its address good for as long as a graph may hold it, and how much dynamic
// shared memory a kernel may take
enum ggb_workspace_id { GGB_WS_GEMM_SPLITS, GGB_WS_MOE_GATHER, GGB_WS_ARGMAX, GGB_WS_RECURRENCE, GGB_WS_COUNT };
int ggb_workspace(ggb_workspace_id id, size_t bytes, void **p);
bool ggb_workspace_fits(ggb_workspace_id id, size_t bytes); // it is that large, or may grow: no graph is being captured
int ggb_allow_smem_of(const void *kernel, size_t bytes);
// how many clusters of `ctas` CTAs (along z) the device runs at once: a cluster lies in one GPC, whose SMs are no multiple of it
int ggb_clusters_at_once_of(const void *kernel, int ctas, int threads, size_t smem, int *n);
template <typename... P> int ggb_allow_smem(void (*kernel)(P...), size_t bytes) { return ggb_allow_smem_of(reinterpret_cast<const void *>(kernel), bytes); }

#define GGB_CUDA(...)                                                                           \
    do {                                                                                        \
        cudaError_t err__ = (__VA_ARGS__);                                                      \
        if (err__ != cudaSuccess) {                                                             \
            ggb_set_error("%s:%d: %s -> %s", __FILE__, __LINE__, #__VA_ARGS__, cudaGetErrorString(err__)); \
            return GGB_ERR_CUDA;                                                                \
        }                                                                                       \
    } while (0)

#define GGB_REQUIRE_INIT()                                  \
    do {                                                    \
        if (!ggb_is_init()) {                               \
            ggb_set_error("ggb_init has not succeeded");    \
            return GGB_ERR_NOT_INIT;                        \
        }                                                   \
    } while (0)

#define GGB_CHECK_ARG(cond, ...)        \
    do {                                \
        if (!(cond)) {                  \
            ggb_set_error(__VA_ARGS__); \
            return GGB_ERR_ARG;         \
        }                               \
    } while (0)

#define GGB_LAUNCH_CHECK()                                                                       \
    do {                                                                                         \
        cudaError_t err__ = cudaGetLastError();                                                  \
        if (err__ != cudaSuccess) {                                                              \
            ggb_set_error("%s:%d: kernel launch -> %s", __FILE__, __LINE__, cudaGetErrorString(err__)); \
            return GGB_ERR_CUDA;                                                                 \
        }                                                                                        \
        ggb_count_launch();                                                                      \
    } while (0)

// ---- device weight layout -------------------------------------------------
// SoA repack of ggml AoS blocks: payload plane [rows][nb][16|32 B], scale plane [rows][nb] fp16.
struct ggb_weight {
    int type;
    int64_t rows, cols, nb; // nb = cols / 32
    uint8_t *qs;            // payload plane
    __half *d;              // scale plane
    void *base;             // owning allocation (null for slices)
    size_t bytes;
};

static inline int ggb_payload_bytes(int type) { return type == GGB_TYPE_Q4_0 ? 16 : 32; }
static inline int ggb_block_bytes(int type) { return type == GGB_TYPE_Q4_0 ? 18 : 34; }

// The mat-vecs of a host program's call (matvec.cu): T rows of nb Q8_0 blocks in host memory; each result goes to `out` [T][rows] in page-locked host memory as
// one word, the call in its upper half
bool ggb_matvec_host_rows_fits(const ggb_weight *w, int64_t T);
int ggb_matvec_host_rows(const ggb_weight *w, const char *blocks, int64_t T, int64_t row_size, uint64_t *out, uint32_t call);

// ---- device helpers -------------------------------------------------------
#ifdef __CUDACC__

__device__ __forceinline__ float warp_sum_f32(float v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}
__device__ __forceinline__ double warp_sum_f64(double v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}
__device__ __forceinline__ float warp_max_f32(float v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}

// 128-bit streaming loads (read once per token: do not allocate in L1): of weights, through the path that takes it for granted that nobody writes
// them while the kernel runs; and of anything
__device__ __forceinline__ uint4 ldg_stream_u4(const void *p) {
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p));
    return r;
}
__device__ __forceinline__ uint4 ld_stream_u4(const void *p) {
    uint4 r;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
    return r;
}

// Holds until the kernels before this one are done and their writes are seen: ahead of every access to memory in a kernel that
// ggb_launch_step launches, run by every thread.  No pointer parameter of such a kernel is __restrict__: what that promises (a const one is
// not written while the kernel runs, none is reached by another way) does not hold until here, and a compiler that believes it may read
// through the read-only cache or ahead of this statement.  For the same reason only weights are read by __ldg and ldg_stream_u4 there.
__device__ __forceinline__ void step_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The same in a kernel that ggb_launch_early launches.  Ahead of it such a kernel sets itself up - barriers, tensor memory, numbers of its arguments - and
// reads weights at most, which stand longer; threads that do not come by here touch memory only behind one that does.
__device__ __forceinline__ void early_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Behind the wait: once every block has said so, blocks of the next kernel may take what room there is and run up to their own wait.  What
// they read ahead of it was written before the kernels that came before this one ended.  A kernel with tensor memory says so when it has it:
// a block of the next kernel that took it first would hold it until this kernel ends.
__device__ __forceinline__ void step_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ float half_bits_to_float(uint16_t h) { return __half2float(__ushort_as_half(h)); }
__device__ __forceinline__ uint16_t float_to_half_bits(float f) { return __half_as_ushort(__float2half_rn(f)); }

// quantize_row_q8_0 for one block spread over a warp: lane i holds element i.
// returns the int8 value; d_out (all lanes) is the fp32 scale before fp16 rounding.
__device__ __forceinline__ int quantize_q8_lane(float x, float &d_out) {
    const float amax = warp_max_f32(fabsf(x));
    const float d = __fdiv_rn(amax, 127.0f);
    const float id = d != 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
    d_out = d;
    return (int)roundf(__fmul_rn(x, id));
}

// counter-based synthetic weights; identical to oracle/ggml_oracle.c orc_synth_value
__host__ __device__ __forceinline__ uint64_t ggb_splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
__host__ __device__ __forceinline__ uint64_t ggb_synth_key(uint64_t seed, uint64_t tensor_id) {
    return ggb_splitmix64(seed + tensor_id * 0xD1B54A32D192ED03ull);
}
__device__ __forceinline__ float ggb_synth_value(uint64_t key, uint64_t index, float unit) {
    const uint64_t r = ggb_splitmix64(key + index);
    const int sum = (int)(r & 0xffff) + (int)((r >> 16) & 0xffff) + (int)((r >> 32) & 0xffff) +
                    (int)((r >> 48) & 0xffff) - 131070;
    return __fmul_rn((float)sum, unit);
}

#endif // __CUDACC__

// host: sigma * (1/37837.2274f) with the same two roundings the oracle performs
static inline float ggb_synth_unit(float sigma) {
    volatile float inv = 1.0f / 37837.2274f;
    volatile float u = sigma * inv;
    return u;
}

#ifdef __CUDACC__
// A kernel of a step of few tokens: a chain of short kernels on a nearly empty GPU, bound by the time from the end of one to the first
// instruction of the next.  The attribute lets the next one be set up while the one before ends; step_wait() orders its reads and writes.
// A layer of 10 such kernels (2048 wide, 16 heads, 8192 in the feed-forward, one token, replayed as a graph): 60.1 us plainly launched,
// 56.8 like this.  Letting the next one start at once (griddepcontrol.launch_dependents) gives no more: 57.3 behind the wait, 63.5 ahead of
// it.  Nor does bringing a mat-vec's matrix into L2 before the wait: 63 to 70, the lines are asked for twice.
template <typename... P, typename... A>
cudaError_t ggb_launch_ahead(void (*k)(P...), dim3 cluster, dim3 grid, dim3 block, size_t smem, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = ggb_cuda_stream();
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster.x, at[1].val.clusterDim.y = cluster.y, at[1].val.clusterDim.z = cluster.z;
    cfg.attrs = at, cfg.numAttrs = cluster.x * cluster.y * cluster.z > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}
struct ggb_cluster { // CTAs that share their shared memory
    unsigned x, y, z;
};
template <typename... P, typename... A> cudaError_t ggb_launch_step(void (*k)(P...), dim3 grid, dim3 block, size_t smem, A... args) {
    return ggb_launch_ahead(k, dim3(1), grid, block, smem, args...);
}
template <typename... P, typename... A> cudaError_t ggb_launch_step(void (*k)(P...), ggb_cluster c, dim3 grid, dim3 block, size_t smem, A... args) {
    return ggb_launch_ahead(k, dim3(c.x, c.y, c.z), grid, block, smem, args...);
}
// The same for kernels that set themselves up ahead of their wait (early_wait)
template <typename... P, typename... A> cudaError_t ggb_launch_early(void (*k)(P...), ggb_cluster c, dim3 grid, dim3 block, size_t smem, A... args) {
    return ggb_launch_ahead(k, dim3(c.x, c.y, c.z), grid, block, smem, args...);
}
#endif

// tables shared by several translation units (runtime.cu owns them)
const uint16_t *ggb_exp_table_dev();  // 64 Ki fp16: exp(f16)
const uint16_t *ggb_gelu_table_dev(); // 64 Ki fp16: gelu(f16)
size_t ggb_tables_bytes();            // both tables are one allocation starting at ggb_exp_table_dev()
const float *ggb_rope_cos_dev();      // [n_ctx][n_dims/2]
const float *ggb_rope_sin_dev();
int ggb_rope_n_ctx();
int ggb_rope_n_dims();
