// Shared declarations for the sm_100a TurboQuant kernels: context layout, dtype
// helpers, error plumbing.  Internal to the library; the public surface is
// include/tq_b200.h.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/tq_b200.h"

#define TQ_D 128
#define TQ_MAX_DEVICES 64  // devices one process may hold contexts on

// Device-resident codec tables.  Matrices are [128][128] fp32, row-major.
struct tq_ctx {
    int device;
    int bits;      // total bits
    int key_bits;  // bits-1 with QJL, else bits
    int use_qjl;
    int sm_count;
    float *rot_k;    // R_k[j][d]
    float *rot_k_t;  // R_k^T[d][j]
    float *rot_v;    // R_v[j][d]
    float *rot_v_t;
    float *qjl;      // S[i][d]
    float *qjl_t;    // S^T[d][i]
    float *centers_k;  // [16] (padded)
    float *bounds_k;   // [16] (padded with +inf)
    float *centers_v;
    float *bounds_v;
    // Shared-memory images of the tcgen05 kernels' B operands (64 KB each, see tq_build_operand_image): R_k, R_v and S
    // in two f16 terms, times a power of two.  A kernel reads one as it lies (vec R^T, vec S^T) or transposed (vec R, vec S).
    struct Image {
        uint16_t *data;
        float unscale;  // what undoes the power of two
    };
    Image img_rot_k, img_rot_v, img_qjl;
    struct Grid {  // cell of z: round(clamp(z * scale + shift, 0, 1) * last); last == 0: no grid separates the boundaries
        float scale, shift, last;
    };
    Grid grid_k, grid_v;
    float cen_k_scale, cen_v_scale;  // powers of two that bring the largest centre just below 2^14
    float res_scale;    // power of two <= 1 that keeps a unit vector's scaled residual inside f16 whatever the centres
    void *base;       // one allocation holding everything above
    size_t base_bytes;
    struct tq_prof *prof;  // measurement hooks, see tq_profile_enable
    int *error_flag;       // device word, set by a kernel whose bounded wait ran out
    int wait_limit_ms;     // how long tq_gather_wait polls for a peer before it gives up (tq_set_wait_limit_ms)
    int64_t splits_cache_key;  // last (rows, length bucket) asked of tq_decode_suggest_splits
    int splits_cache_val;
};

// Measurement hooks: bracket the main decode kernel with events, count launches.
void tq_prof_begin(tq_ctx *ctx, cudaStream_t stream);
void tq_prof_end(tq_ctx *ctx, cudaStream_t stream);
void tq_prof_count(tq_ctx *ctx, int n_launches);

void tq_set_cuda_error(cudaError_t e, const char *where);

// Named NVTX range around the host side of an entry point (header-only NVTX: a no-op unless a
// profiler is attached), so that a timeline shows pack / append / decode / gather calls by name.
#include <nvtx3/nvToolsExt.h>
struct TqRange {
    explicit TqRange(const char *name) { nvtxRangePushA(name); }
    ~TqRange() { nvtxRangePop(); }
    TqRange(const TqRange &) = delete;
    TqRange &operator=(const TqRange &) = delete;
};

#define TQ_CUDA_CHECK(expr)                         \
    do {                                            \
        cudaError_t _e = (expr);                    \
        if (_e != cudaSuccess) {                    \
            tq_set_cuda_error(_e, #expr);           \
            return TQ_ERR_CUDA;                     \
        }                                           \
    } while (0)

// Kernel launch with the optional "programmatic stream serialization" attribute: the kernel may
// start while the preceding kernel of the stream is still running and must call
// griddepcontrol.wait before it touches anything that kernel writes.  `cluster` > 1: CTAs per cluster (along x).
template <typename... KArgs, typename... Args>
cudaError_t tq_launch_cluster(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              bool programmatic, int cluster, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    if (programmatic) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = cluster;
        attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1, ++cfg.numAttrs;
    }
    cfg.attrs = attr;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
template <typename... KArgs, typename... Args>
cudaError_t tq_launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                             bool programmatic, Args... args) {
    return tq_launch_cluster(kernel, grid, block, smem, stream, programmatic, 1, args...);
}

// Lets a kernel use `smem` bytes of dynamic shared memory (an attribute of the kernel on one device: set once).
template <auto KERNEL> cudaError_t tq_allow_shared(int device, int smem) {
    static bool configured[TQ_MAX_DEVICES] = {};
    if (device < 0 || device >= TQ_MAX_DEVICES) return cudaErrorInvalidDevice;
    if (configured[device]) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    configured[device] = e == cudaSuccess;
    return e;
}

template <typename T> __device__ __forceinline__ float tq_to_float(T x);
template <> __device__ __forceinline__ float tq_to_float<float>(float x) { return x; }
template <> __device__ __forceinline__ float tq_to_float<__half>(__half x) { return __half2float(x); }
template <> __device__ __forceinline__ float tq_to_float<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T> __device__ __forceinline__ T tq_from_float(float x);
template <> __device__ __forceinline__ float tq_from_float<float>(float x) { return x; }
template <> __device__ __forceinline__ __half tq_from_float<__half>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ __nv_bfloat16 tq_from_float<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

// Round a float through storage type T and back (the reference's `.to(dtype).float()`).
template <typename T> __device__ __forceinline__ float tq_round_through(float x) {
    return tq_to_float<T>(tq_from_float<T>(x));
}

__device__ __forceinline__ float tq_half_bits_to_float(uint16_t h) {
    return __half2float(__ushort_as_half(h));
}
__device__ __forceinline__ uint16_t tq_float_to_half_bits(float x) {
    return __half_as_ushort(__float2half_rn(x));
}

__device__ __forceinline__ float tq_warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float tq_warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Argument validators shared by every entry point that takes the descriptor (nothing is
// launched before they pass): all stream pointers present and 16-byte aligned, strides
// multiples of 8 tokens that do not overlap rows; every peer pointer and the counter present.
int tq_check_cache(const tq_ctx *ctx, const tq_cache_desc *c);
int tq_check_gather(const tq_gather_desc *g);

// Entry points implemented in the other translation units.
int32_t tq_launch_pack(tq_ctx *ctx, const tq_dense_desc *k, const tq_dense_desc *v, int32_t n_tokens,
                       const tq_cache_desc *cache, int32_t pos0, cudaStream_t stream);
int32_t tq_launch_decode_exact(tq_ctx *ctx, const void *q, int32_t q_dtype, int32_t q_heads,
                               const tq_cache_desc *cache, int32_t seq_len, const tq_dense_desc *tail_k,
                               const tq_dense_desc *tail_v, int32_t n_tail, int32_t n_splits,
                               void *workspace, void *out, cudaStream_t stream);
// What a whole-step entry point adds to a plain decode launch (all optional).
struct TqStepExtras {
    const struct TqPackArgs *append;  // encode and append the step's new token in the query-preparation launch
    const int *len_ptr;               // the sequence length lives in device memory
    const tq_gather_desc *gather;     // KV-head shard: write the outputs into every rank's gathered buffer
    float *out_f32;                   // write the result unrounded (fp32) here instead of `out`
    int parts;                        // sequence split: ranks per KV-head group (0: off), see tq_decode_attn_parts
};
int tq_mma4_tokens_per_cta_step();
int32_t tq_launch_decode_mma4(tq_ctx *ctx, const void *q, int32_t q_dtype, int32_t q_heads,
                              const tq_cache_desc *cache, int32_t seq_len, const tq_dense_desc *tail_k,
                              const tq_dense_desc *tail_v, int32_t n_tail, int32_t n_splits,
                              void *workspace, void *out, const TqStepExtras *extras, cudaStream_t stream);
float tq_fit_power(float largest);  // the power of two that brings `largest` into [2^13, 2^14)
bool tq_fit_grid(const float *bounds, int n, tq_ctx::Grid *g);
float tq_build_operand_image(const float *m, uint16_t *image);
// `k` null: values only.  TQ_ERR_UNSUPPORTED when a tensor's alignment rules the kernel out.
int32_t tq_launch_pack_tc(tq_ctx *ctx, const tq_dense_desc *k, const tq_dense_desc *v, int32_t n_tokens,
                          const tq_cache_desc *cache, int32_t pos0, cudaStream_t stream);
// TQ_ERR_UNSUPPORTED when the output's alignment rules the kernel out.
int32_t tq_launch_dequant_tc(tq_ctx *ctx, const tq_cache_desc *cache, int32_t which, int32_t pos0, int32_t n_tokens,
                             const tq_dense_desc *out, cudaStream_t stream);
int32_t tq_launch_dequant(tq_ctx *ctx, const tq_cache_desc *cache, int32_t which, int32_t pos0,
                          int32_t n_tokens, const tq_dense_desc *out, cudaStream_t stream);
