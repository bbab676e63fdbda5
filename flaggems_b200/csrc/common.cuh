// Shared host/device helpers for the C-ABI library (sm_100a only).
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/flaggems_b200.h"

// Thread-local text of the last error returned by an entry point.
void fg_set_error(const char* fmt, ...);

#define FG_REQUIRE(cond, code, ...)        \
    do {                                   \
        if (!(cond)) {                     \
            fg_set_error(__VA_ARGS__);     \
            return (code);                 \
        }                                  \
    } while (0)

#define FG_CUDA(call)                                                              \
    do {                                                                           \
        cudaError_t e__ = (call);                                                  \
        if (e__ != cudaSuccess) {                                                  \
            fg_set_error("%s failed: %s", #call, cudaGetErrorString(e__));         \
            return FG_ERR_CUDA;                                                    \
        }                                                                          \
    } while (0)

#define FG_LAUNCH_CHECK()                                                          \
    do {                                                                           \
        cudaError_t e__ = cudaGetLastError();                                      \
        if (e__ != cudaSuccess) {                                                  \
            fg_set_error("kernel launch failed: %s", cudaGetErrorString(e__));     \
            return FG_ERR_CUDA;                                                    \
        }                                                                          \
    } while (0)

// Device-side status word (0 = healthy).  Kernels with bounded waits record the
// first failure here; fg_device_status() reads and clears it.
unsigned int* fg_status_word_device_ptr();

static inline int64_t fg_cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

int fg_num_sms();

// Index of the current device clamped to [0, 63]: the key of every per-device cache in the library.
int fg_device_index();

// Grouped expert GEMM with every option of the C-ABI forms, for the pipelines of this library.
// gather_div > 0: a (row stride ld_a elements) and a_scale hold one row per token and route slot s
// reads row s / gather_div through sorted_ids; 0: rows are in sorted order.
struct FgGroupedGemm {
    void* c;
    const void *a, *w;
    const float *a_scale, *w_scale;
    const void* topk_w;
    int topk_w_dtype;
    int64_t topk_w_stride;
    const int32_t *sorted_ids, *expert_ids, *num_post_pad;
    int64_t a_rows;    // rows of a
    int64_t max_rows;  // sorted rows
    int64_t numel;
    int gather_div;
    int a_contiguous;  // with gather_div = 1: the slots of a block are consecutive rows of a
    int num_experts;
    int64_t N, K, ld_a, ld_as, ld_c;  // ld_as: block scales only
    int operand;  // 0 e4m3, 1 int8, 2 bf16, 3 fp16
    int block_rows, scale_mode, a_scale_per_row, fuse_silu, scatter, mul_weight, out_dtype;
    int cta_pairs;  // block_rows = 256: every block is one tile row of a CTA pair
    const float* bias;  // fp32, added before the cast; bias_stride elements between the rows of consecutive experts
    int64_t bias_stride;
    const int32_t* dest;
    int64_t dest_stride;
    void* const* peer_out;
    int n_peers;
    int64_t peer_rows;
};
int fg_grouped_gemm(const FgGroupedGemm& g, cudaStream_t stream);

// sorted_ids / expert_ids / num_post_pad of rows grouped by the ends `offs`, padded to `block` per group.
int fg_group_tiles(const int32_t* offs, int num_groups, int64_t rows, int block, int32_t* sorted_ids, int64_t max_pad,
                   int32_t* expert_ids, int64_t n_blocks, int32_t* num_post_pad, cudaStream_t stream);

// fg_moe_align_block_size_regions; fill_tail = false leaves the entries past the last block unwritten.
int fg_moe_align(const void* topk_ids, int ids_are_i64, int64_t numel, int num_experts, int block_size, const int32_t* expert_map,
                 int expert_map_len, int32_t* sorted_ids, int64_t max_pad, int32_t* expert_ids, int64_t n_blocks,
                 int32_t* num_post_pad, int64_t ids_stride, int id_div, int32_t* expert_counts, const int32_t* numel_dev,
                 int64_t region_rows, const int32_t* region_counts, int64_t region_stride, bool fill_tail, cudaStream_t stream);

// x[0:n] = 1
int fg_fill_ones(float* x, int64_t n, cudaStream_t stream);

// Contiguous rows [*, K] -> quantised rows [rows, K] and scales, optionally through row_index (output row
// r takes row row_index[r] / index_div; index_div = 0: row r itself) and with the row count on the
// device.  Output rows whose index is outside [0, index_limit) are padding and become zeros.
// FG_QUANT_TENSOR: tensor_scale is the given scale, or with scale_out != NULL the
// amax it is derived from.
enum { FG_QUANT_GROUP128 = 0, FG_QUANT_TOKEN = 1, FG_QUANT_INT8 = 2, FG_QUANT_TENSOR = 3 };
int fg_quant_rows(int kind, const void* x, int x_dtype, void* q, float* s, const float* tensor_scale, float* scale_out, int64_t rows,
                  int64_t K, const int32_t* row_index, int32_t index_div, int32_t index_limit, const int32_t* n_rows_dev,
                  cudaStream_t st);

// fg_abs_max over the rows row_index names (entries outside [0, index_limit) are skipped); NULL: rows 0 .. M - 1.
int fg_abs_max_rows(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ld_x, const int32_t* n_rows_dev,
                    const int32_t* row_index, int32_t index_limit, float* amax, cudaStream_t st);

// Adds n to the process-wide count of kernels launched by this library.
void fg_count_launch(int n);

#ifdef __CUDACC__
// Programmatic dependent launch: the kernels of this library are launched so that they may start while the
// kernel before them in the stream is still running.  Each of them calls fg_pdl_wait() before it touches
// global memory (it returns once every earlier kernel has finished and its writes are visible) and
// fg_pdl_trigger() when the kernel after it may be scheduled.  What overlaps is launch latency and
// prologues: ~2 us per kernel, which is a fifth of a decode-sized product.
// Everything that an earlier kernel may have written, so any operand of a public entry point, is read with ordinary
// loads.  The read-only path (__ldg, const __restrict__) is defined for memory that nobody writes while the kernel
// lives, and that now includes the end of its predecessor; the compiler may also move such loads above the wait.
__device__ __forceinline__ void fg_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void fg_pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launches `kernel` that way (or, without `early`, after everything before it), with clusters of `cluster` CTAs
// when cluster > 1.
template <typename... Params, typename... Args>
cudaError_t fg_launch_when(bool early, void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                           unsigned cluster, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(block, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    if (early) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = cluster;
        attr[cfg.numAttrs].val.clusterDim.y = 1;
        attr[cfg.numAttrs++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
    if (e == cudaSuccess) fg_count_launch(1);
    return e;
}

template <typename... Params, typename... Args>
cudaError_t fg_launch(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, unsigned cluster,
                      Args&&... args) {
    // Not where the grid fills more than half of the chip's thread slots: its CTAs would sit in them, waiting, while
    // another stream (a layer's shared expert) has work for the SMs.  A layer of 8192 tokens takes 6018 us with every
    // kernel launched early, 5827 with this rule and that of the products, and took 5772 before there were early launches.
    const bool early = (int64_t)grid * block <= 1024 * (int64_t)fg_num_sms();
    return fg_launch_when(early, kernel, grid, block, smem, st, cluster, args...);
}

template <typename T> struct FgVec8;  // eight elements of T as raw words

__device__ __forceinline__ float fg_to_float(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float fg_to_float(__half v) { return __half2float(v); }
__device__ __forceinline__ float fg_to_float(float v) { return v; }

template <typename T> __device__ __forceinline__ T fg_from_float(float v);
template <> __device__ __forceinline__ __nv_bfloat16 fg_from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half fg_from_float<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ float fg_from_float<float>(float v) { return v; }

// Load eight consecutive elements as floats; p must be 16-byte aligned for
// 16-bit types and 32-byte aligned for fp32.
template <typename T>
__device__ __forceinline__ void fg_load8(const T* p, float (&f)[8]) {
    if constexpr (sizeof(T) == 2) {
        uint4 raw = *reinterpret_cast<const uint4*>(p);
        const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = fg_to_float(e[i]);
    } else {
        float4 a = reinterpret_cast<const float4*>(p)[0];
        float4 b = reinterpret_cast<const float4*>(p)[1];
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
        f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }
}

// Eight 16-bit elements already in registers (one 16-byte load) as floats.
template <typename T>
__device__ __forceinline__ void fg_unpack8(const uint4& raw, float (&f)[8]) {
    static_assert(sizeof(T) == 2, "16-bit element types only");
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = fg_to_float(e[i]);
}

template <typename T>
__device__ __forceinline__ void fg_store8(T* p, const float (&f)[8]) {
    if constexpr (sizeof(T) == 2) {
        uint4 raw;
        T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = fg_from_float<T>(f[i]);
        *reinterpret_cast<uint4*>(p) = raw;
    } else {
        reinterpret_cast<float4*>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
        reinterpret_cast<float4*>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
    }
}

// Eight floats -> eight e4m3 bytes (round to nearest even, saturate to +-448).
__device__ __forceinline__ uint2 fg_pack_e4m3x8(const float (&q)[8]) {
    uint32_t w[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(q[4 * h + 0], q[4 * h + 1]), __NV_SATFINITE, __NV_E4M3);
        uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(q[4 * h + 2], q[4 * h + 3]), __NV_SATFINITE, __NV_E4M3);
        w[h] = lo | (hi << 16);
    }
    return make_uint2(w[0], w[1]);
}
#endif
