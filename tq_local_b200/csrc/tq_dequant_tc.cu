// Dequantisation on the 5th-generation tensor cores, 128 vectors at a time:
//
//   out = round_T(|x| * centres[codes] R)  [ + round_T(|r| * sqrt(pi/2)/128 * signs S), rounded again ]
//
// with the matrices in two f16 terms (tq_umma.cuh), the centres in two and the signs (+-1) in one.  The
// structure is the prefill encoder's: one persistent CTA per SM, two groups of sixteen warps that each walk
// their own tiles, four threads to a vector, A written to TMEM, the matrices resident in shared memory; the two
// contractions of a key go one after the other through the group's one accumulator, the first result waiting as
// packed T.  16-bit rows leave through shared memory, sixteen lanes to a row.
// Bound, like the encoder, by the CUDA-core work between the contractions.  8 x 32768 bf16, keys with the sketch and values: 93.5 us with the
// issuing thread chosen by its index and a bulk copy per row, issued lane by lane by the warps that all others then waited
// for; 78.5 with an elected issuer whose operands stay in uniform registers and the groups' contractions one after the
// other (80.0 without that order); 72.4 with rows that all warps copy out, 16 bytes a lane (HBM floor 26; 1694 us with fp32
// multiply-adds and the matrix read from L2 per vector).
#include <math.h>

#include <type_traits>

#include "tq_common.cuh"
#include "tq_umma.cuh"

namespace {

constexpr int kGroups = 2;
constexpr int kGroupThreads = 512;
constexpr int kThreads = kGroups * kGroupThreads;
constexpr int kParts = kGroupThreads / kUmmaRows;  // threads per vector
constexpr int kCoords = TQ_D / kParts;             // coordinates per thread

struct DequantTcArgs {
    const uint8_t *codes;
    const uint16_t *norms;
    const uint8_t *signs;
    const uint16_t *rnorms;
    int64_t cache_sb, cache_sh;
    VectorIndex vec;
    int pos0, n_tiles;
    void *out;
    int64_t ob, oh, ot;
    const uint16_t *image, *image2;  // R, S
    float unscale, unscale2;         // undo the scales of R and the centres (a power of two), and of S
    const float *centers;            // 16 floats
    float cen_scale;
    int *error_flag;
};

template <typename T> __device__ __forceinline__ uint32_t pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2<__half>(float a, float b) { return half2_bits(a, b); }
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
template <typename T> __device__ __forceinline__ float2 unpack2(uint32_t w);
template <> __device__ __forceinline__ float2 unpack2<__half>(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2 *>(&w)); }
template <> __device__ __forceinline__ float2 unpack2<__nv_bfloat16>(uint32_t w) {
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

template <typename T, int BITS, bool QJL>
__global__ void __launch_bounds__(kThreads, 1) tq_dequant_tc_kernel(const __grid_constant__ DequantTcArgs a) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint32_t s_cen[16];  // f16 hi term | lo term << 16 of a scaled centre
    __shared__ uint64_t s_bar_image[2], s_bar_mma[kGroups];
    __shared__ uint32_t s_tmem, s_turn;  // (see turn_take)
    const uint32_t images = (smem_u32(smem_raw) + 1023u) & ~1023u;  // swizzle atoms need 1024-byte alignment
    const int tid = threadIdx.x, warp = tid >> 5, group = tid / kGroupThreads;
    if (tid < 16) {
        const float c = a.centers[tid] * a.cen_scale;
        const __half hi = __float2half_rn(c), lo = __float2half_rn(c - __half2float(hi));
        s_cen[tid] = (uint32_t)__half_as_ushort(hi) | (uint32_t)__half_as_ushort(lo) << 16;
    }
    if (warp == 0) {  // all of TMEM: one CTA per SM
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (tid == 0) {
        s_turn = 0;
        for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&s_bar_image[i]), 1), mbar_init(smem_u32(&s_bar_mma[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        umma_load_image(images, a.image, smem_u32(&s_bar_image[0]));  // (every CTA has at least one tile)
        if (QJL) umma_load_image(images + kUmmaImageBytes, a.image2, smem_u32(&s_bar_image[1]));
    }
    umma_fence_before();
    __syncthreads();
    umma_fence_after();

    const int vrow = tid & (kUmmaRows - 1), part = (tid / kUmmaRows) % kParts;
    const uint32_t acc = __shfl_sync(0xffffffffu, s_tmem + group * 256, 0), a_hi = acc + 128, a_lo = acc + 192;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t my_acc = acc + lanes + kCoords * part, my_hi = a_hi + lanes + kCoords / 2 * part, my_lo = my_hi + 64;
    const uint32_t bar_mma = smem_u32(&s_bar_mma[group]);
    const bool issuer = __shfl_sync(0xffffffffu, tid & (kGroupThreads - 1), 0) == 0;  // a group's first warp
    // `landed`: the issuer's images seen in shared memory, bits 0 and 1; bit 2: a wait of this thread ran out.  (One word for both: 64 registers
    // are all there are, and keys of two bits were short of one - 8 x 32768 bf16 keys and values of 3 bits 75.7 us, 72.5 like this.)
    uint32_t mma_phase = 0, landed = 0;
    constexpr uint32_t kTimedOut = 4;
    constexpr bool kStaged = sizeof(T) == 2;
    // The lock of turn_take: 16-bit rows 4 % faster with it; fp32 rows slower, a CTA with one tile most, whose three batches of MMAs
    // each pass it for nothing (8 x 1000 keys and values of 3 bits 19.5 us with it, 18.25 without; 8 x 32768 152.5 and 150.8).
    constexpr bool kInTurn = sizeof(T) == 2;
    const uint32_t my_stage = images + (QJL ? 2 : 1) * kUmmaImageBytes + group * kStageBytes + vrow * kStagePitch;
    auto group_sync = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + group), "r"(kGroupThreads) : "memory"); };
    // The tensor core rounds its running sum towards zero at every step.  A row with one large element, whose products all have
    // one sign, loses 4e-7 of it; the fp32 results' sums of centres come in two pieces of four steps each, which leaves 2e-7, and
    // half of that is given back by scaling one piece by kUmmaRestore.  Relative to 64 bits, 2-norm over 262144 rows, 3-bit
    // values: rows with one large element 3.5e-7 in one piece, 1.5e-7 in two (fp32 multiply-adds one after the other: 2.0e-7), Gaussian
    // rows 1.3e-7 and 1.1e-7 (2.0e-7).  The signs' sums stay below 1.1e-7 in one.
    constexpr int kPieces = sizeof(T) == 4 ? 2 : 1;
    const std::integral_constant<int, 0> first_piece;
    const std::integral_constant<int, 1> second_piece;
    // Everybody has stored its part of A and read the accumulators of the stage or piece before: two products when A
    // has one term (the signs), three when it has two.
    auto gemm = [&](auto terms, auto piece) {  // stage 0: the centres, two terms; stage 1: the signs, one
        constexpr int kTerms = decltype(terms)::value, stage = 2 - kTerms;
        tmem_st_wait();
        umma_fence_before();
        group_sync();
        if (issuer && elect_one()) {
            umma_fence_after();
            if (!(landed >> stage & 1)) {
                if (!mbar_wait(smem_u32(&s_bar_image[stage]), 0)) landed |= kTimedOut;
                landed |= 1u << stage;
            }
            if (kInTurn && !turn_take(&s_turn)) landed |= kTimedOut;
            umma_issue<kTerms, true, decltype(piece)::value, kTerms == 2 ? kPieces : 1>(acc, a_hi, a_lo, images + stage * kUmmaImageBytes);
            umma_commit(bar_mma);
            if (kInTurn) turn_give(&s_turn);
        }
    };
    auto gemm_wait = [&]() {
        if (!mbar_wait(bar_mma, mma_phase)) landed |= kTimedOut;
        mma_phase ^= 1;
        __syncwarp();
        umma_fence_after();
    };

    // this thread's 32 codes
    uint32_t words[BITS + 1];
    uint32_t sw = 0;
    uint16_t nh = 0, rh = 0;
    T *dst = nullptr;
    words[BITS] = 0;
    auto fetch = [&](int tile) {
        const int64_t vid = (int64_t)tile * kUmmaRows + vrow;
        const int64_t v = vid < a.vec.n ? vid : 0;
        int t, h, b;
        vector_at(a.vec, v, b, h, t);
        const int64_t row = b * a.cache_sb + h * a.cache_sh + a.pos0 + t;
        const uint32_t *src = reinterpret_cast<const uint32_t *>(a.codes + row * (16 * BITS)) + BITS * part;
        if constexpr (BITS == 4) {
            const uint4 c = __ldg(reinterpret_cast<const uint4 *>(src));
            words[0] = c.x, words[1] = c.y, words[2] = c.z, words[3] = c.w;
        } else {
#pragma unroll
            for (int w = 0; w < BITS; ++w) words[w] = __ldg(src + w);
        }
        nh = a.norms[row];
        if (QJL) sw = __ldg(reinterpret_cast<const uint32_t *>(a.signs + row * 16) + part), rh = a.rnorms[row];
        dst = vid < a.vec.n ? reinterpret_cast<T *>(a.out) + b * a.ob + h * a.oh + (int64_t)t * a.ot : nullptr;
    };
    const int first = (int)blockIdx.x + (int)gridDim.x * group, stride = (int)gridDim.x * kGroups;
    if (first < a.n_tiles) fetch(first);
    for (int tile = first; tile < a.n_tiles; tile += stride) {
        // ---------------- A = centres[codes]
        __syncwarp();  // (tcgen05.st is warp-collective)
#pragma unroll
        for (int c = 0; c < kCoords / 16; ++c) {
            uint32_t hi[8], lo[8];
            auto centre = [&](int e) {
                const int bit = e * BITS, w = bit >> 5, sh = bit & 31;
                const uint32_t v = sh + BITS > 32 ? __funnelshift_r(words[w], words[w + 1], sh) : words[w] >> sh;
                return s_cen[v & ((1u << BITS) - 1u)];
            };
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t t0 = centre(16 * c + 2 * i), t1 = centre(16 * c + 2 * i + 1);
                hi[i] = __byte_perm(t0, t1, 0x5410), lo[i] = __byte_perm(t0, t1, 0x7632);
            }
            tmem_st8(my_hi + 8 * c, hi), tmem_st8(my_lo + 8 * c, lo);
        }
        gemm(std::integral_constant<int, 2>(), first_piece);
        const float nf = tq_half_bits_to_float(nh) * (sizeof(T) == 4 ? a.unscale : a.unscale * kUmmaRestore);
        const float rf = tq_half_bits_to_float(rh);
        const uint32_t signs = sw;
        T *const to = dst;
        if (tile + stride < a.n_tiles) fetch(tile + stride);
        gemm_wait();
        constexpr int kOutWords = kCoords * (int)sizeof(T) / 4;
        uint32_t o[kOutWords];  // this thread's 32 outputs
        const uint64_t nf2 = f32x2(nf, nf);
        // fp32 results: o = combine(the accumulators, o), two at a time
        auto accumulators = [&](auto combine) {
            if constexpr (sizeof(T) == 4) {
#pragma unroll
                for (int q = 0; q < kCoords / 16; ++q) {
                    uint32_t y[16];
                    tmem_ld16(my_acc + 16 * q, y);
#pragma unroll
                    for (int e = 0; e < 16; e += 2) {
                        uint32_t *p = o + 16 * q + e;
                        float y0, y1;
                        f32x2_split(combine(f32x2(__uint_as_float(y[e]), __uint_as_float(y[e + 1])), f32x2(__uint_as_float(p[0]), __uint_as_float(p[1]))), y0, y1);
                        p[0] = __float_as_uint(y0), p[1] = __float_as_uint(y1);
                    }
                }
            }
        };
#pragma unroll
        for (int q = 0; q < kCoords / 16; ++q) {
            uint32_t y[16];
            tmem_ld16(my_acc + 16 * q, y);
#pragma unroll
            for (int e = 0; e < 16; e += 2) {
                if constexpr (sizeof(T) == 4) {
                    o[16 * q + e] = y[e], o[16 * q + e + 1] = y[e + 1];
                } else {
                    float y0, y1;
                    f32x2_split(f32x2_mul(f32x2(__uint_as_float(y[e]), __uint_as_float(y[e + 1])), nf2), y0, y1);
                    o[8 * q + e / 2] = pack2<T>(y0, y1);
                }
            }
        }
        if constexpr (kPieces == 2) {
            gemm(std::integral_constant<int, 2>(), second_piece);
            gemm_wait();
            const uint64_t restore2 = f32x2(kUmmaRestore, kUmmaRestore);
            accumulators([&](uint64_t y, uint64_t first) { return f32x2_mul(f32x2_fma(first, restore2, y), nf2); });
        }
        if constexpr (QJL) {
            // ---------------- A = signs: f16 1.0 with the complement of the sign bit on top
#pragma unroll
            for (int c = 0; c < kCoords / 16; ++c) {
                const uint32_t w = ~signs >> (16 * c);
                uint32_t s[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) s[i] = 0x3C003C00u | ((w << (15 - 2 * i)) & 0x8000u) | ((w << (30 - 2 * i)) & 0x80000000u);
                tmem_st8(my_hi + 8 * c, s);
            }
            gemm(std::integral_constant<int, 1>(), first_piece);
            gemm_wait();
            const float scale = 1.2533141373155003f / (float)TQ_D;  // sqrt(pi/2)/D
            if constexpr (sizeof(T) == 4) {
                const uint64_t rs2 = f32x2(a.unscale2 * rf * scale, a.unscale2 * rf * scale);
                accumulators([&](uint64_t y, uint64_t rec) { return f32x2_fma(y, rs2, rec); });
            } else {
#pragma unroll
                for (int q = 0; q < kCoords / 16; ++q) {
                    uint32_t y[16];
                    tmem_ld16(my_acc + 16 * q, y);
#pragma unroll
                    for (int e = 0; e < 16; e += 2) {
                        const float y0 = __uint_as_float(y[e]) * a.unscale2 * rf * scale, y1 = __uint_as_float(y[e + 1]) * a.unscale2 * rf * scale;
                        const float2 r = unpack2<T>(o[8 * q + e / 2]), c = unpack2<T>(pack2<T>(y0, y1));
                        o[8 * q + e / 2] = pack2<T>(r.x + c.x, r.y + c.y);
                    }
                }
            }
        }
        if constexpr (kStaged) {
            // (every warp has read its rows of the tile before: it did so ahead of this tile's first barrier)
#pragma unroll
            for (int i = 0; i < kOutWords; i += 4) sts128(my_stage + 2 * kCoords * part + 4 * i, o[i], o[i + 1], o[i + 2], o[i + 3]);
            group_sync();
            const int lane = tid & 31;
#pragma unroll
            for (int i = 0; i < 8; i += 2) {  // eight of the warp's 32 rows (the other parts' warps take the others), sixteen lanes to a row
                const int from = 8 * part + i + (lane >> 4);
                T *const row = reinterpret_cast<T *>(__shfl_sync(0xffffffffu, reinterpret_cast<uint64_t>(to), from));
                const uint4 v = lds128(my_stage + (from - lane) * kStagePitch + 16 * (lane & 15));
                if (row) reinterpret_cast<uint4 *>(row)[lane & 15] = v;
            }
        } else if (to) {
#pragma unroll
            for (int i = 0; i < kOutWords; i += 4)
                *reinterpret_cast<uint4 *>(reinterpret_cast<uint32_t *>(to) + kOutWords * part + i) = make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]);
        }
    }
    if (landed & kTimedOut) atomicExch(a.error_flag, 3);
    umma_fence_before();
    __syncthreads();
    if (warp == 0) {
        umma_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(s_tmem), "r"(512));
    }
}

template <typename T, int BITS, bool QJL> cudaError_t launch(const DequantTcArgs &a, int grid, int device, cudaStream_t stream) {
    constexpr int smem = (QJL ? 2 : 1) * kUmmaImageBytes + (sizeof(T) == 2 ? kGroups * kStageBytes : 0) + 1024;
    // the attribute belongs to the (kernel, device) pair: one flag per device of this instantiation
    static bool configured[TQ_MAX_DEVICES] = {};
    if (device < 0 || device >= TQ_MAX_DEVICES) return cudaErrorInvalidDevice;
    if (!configured[device]) {
        cudaError_t e = cudaFuncSetAttribute(tq_dequant_tc_kernel<T, BITS, QJL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        configured[device] = true;
    }
    tq_dequant_tc_kernel<T, BITS, QJL><<<grid, kThreads, smem, stream>>>(a);
    return cudaGetLastError();
}
template <typename T> cudaError_t launch(const DequantTcArgs &a, int bits, bool qjl, int grid, int device, cudaStream_t stream) {
    switch (bits) {
        case 1: return qjl ? launch<T, 1, true>(a, grid, device, stream) : cudaErrorInvalidValue;
        case 2: return qjl ? launch<T, 2, true>(a, grid, device, stream) : launch<T, 2, false>(a, grid, device, stream);
        case 3: return qjl ? launch<T, 3, true>(a, grid, device, stream) : launch<T, 3, false>(a, grid, device, stream);
        case 4: return qjl ? cudaErrorInvalidValue : launch<T, 4, false>(a, grid, device, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

int32_t tq_launch_dequant_tc(tq_ctx *ctx, const tq_cache_desc *cache, int32_t which, int32_t pos0, int32_t n_tokens,
                             const tq_dense_desc *out, cudaStream_t stream) {
    const int64_t esize = out->dtype == TQ_DTYPE_F32 ? 4 : 2;
    if (((uintptr_t)out->data | (uintptr_t)((out->stride_b | out->stride_h | out->stride_t) * esize)) & 15) return TQ_ERR_UNSUPPORTED;
    const bool key = which == 0, qjl = key && ctx->use_qjl;
    DequantTcArgs a;
    a.codes = key ? cache->k_codes : cache->v_codes, a.norms = key ? cache->k_norms : cache->v_norms;
    a.signs = cache->k_signs, a.rnorms = cache->k_rnorms;
    a.cache_sb = cache->stride_b, a.cache_sh = cache->stride_h;
    a.vec = vector_index(cache->batch, cache->kv_heads, n_tokens), a.pos0 = pos0;
    a.n_tiles = (int)((a.vec.n + kUmmaRows - 1) / kUmmaRows);
    a.out = const_cast<void *>(out->data), a.ob = out->stride_b, a.oh = out->stride_h, a.ot = out->stride_t;
    const tq_ctx::Image &image = key ? ctx->img_rot_k : ctx->img_rot_v;
    a.image = image.data, a.image2 = ctx->img_qjl.data;
    a.cen_scale = key ? ctx->cen_k_scale : ctx->cen_v_scale;
    a.unscale = image.unscale / a.cen_scale, a.unscale2 = kUmmaRestore * ctx->img_qjl.unscale;
    a.centers = key ? ctx->centers_k : ctx->centers_v;
    a.error_flag = ctx->error_flag;
    const int grid = a.n_tiles < ctx->sm_count ? a.n_tiles : ctx->sm_count;
    const int bits = key ? ctx->key_bits : ctx->bits;
    cudaError_t e;
    if (out->dtype == TQ_DTYPE_F32) e = launch<float>(a, bits, qjl, grid, ctx->device, stream);
    else if (out->dtype == TQ_DTYPE_F16) e = launch<__half>(a, bits, qjl, grid, ctx->device, stream);
    else e = launch<__nv_bfloat16>(a, bits, qjl, grid, ctx->device, stream);
    TQ_CUDA_CHECK(e);
    return TQ_OK;
}
