// Prefill encoder on the 5th-generation tensor cores: rotate 128 vectors at a time with
// tcgen05.mma, quantise and bit-pack in the epilogue.
//
//   values, and keys without the sketch (one contraction):   z = x R^T / |x|  -> codes, |x|
//   keys with the sketch (three, chained):
//     1. z     = x R_k^T / |x|                  -> codes, |x|
//     2. y     = round_T(fp16(|x|) * centres[codes] R_k);   r = x - y, |r|
//     3. p     = r S^T                          -> sign bits, |r|
//
// Operands are f16 in two terms (see tq_umma.cuh); a 16-bit vector needs one: f16 rows are used as they
// are, bf16 rows times the power of two that brings |x| to [2^12, 2^13), which is exact down to 2^-37 |x|.
// Nothing is normalised before a contraction; the accumulators are multiplied by 1 / |x| instead.
//
// One CTA of 16 warps per SM: two groups of eight warps, each walking tiles of 128 vectors on its own, so
// that one group's CUDA-core work runs beside the other group's MMAs.  Two threads share a vector (64
// coordinates each).  The A operand is written to TMEM (tcgen05.st, no swizzle, no bank conflicts), so
// shared memory is left for the matrices: the three of the sketch path (192 KB) stay resident and nothing
// is reloaded between the stages.  A group owns 256 TMEM columns: 128 of accumulator, 64 for each term of A.
// The first CTAs of a launch encode keys and the others values, in the proportion of their costs.
// Every mbarrier wait is bounded and reports through the device status word.
#include <math.h>
#include <string.h>

#include <type_traits>

#include "tq_common.cuh"
#include "tq_umma.cuh"

namespace {

constexpr int kGroups = 2;
constexpr int kGroupThreads = 256;
constexpr int kThreads = kGroups * kGroupThreads;
constexpr int kHalf = TQ_D / 2;  // coordinates per thread

struct PackTcRole {
    const void *x;
    int64_t sb, sh, st;
    uint8_t *codes;
    uint16_t *norms;
    const uint16_t *image;  // the rotation
    float unscale;
    const float *bounds;    // 16 floats, padded with +inf
};
struct PackTcArgs {
    PackTcRole role[2];  // keys, values
    int key_ctas;        // CTAs [0, key_ctas) encode keys, the others values
    int B, H, S, pos0;
    int64_t cache_sb, cache_sh;
    int n_tiles;
    int *error_flag;
    // the sketch
    const uint16_t *image2, *image3;  // R_k^T (reconstruction), S (projection)
    float unscale2;                   // undoes the scales of R_k^T and of the centres
    float cen_scale, res_scale;
    const float *centers;  // 16 floats
    uint8_t *signs;
    uint16_t *rnorms;
};

template <typename T> struct Raw;  // how many 32-bit words 64 coordinates take, and pairs of them as floats
template <> struct Raw<float> {
    static constexpr int kWords = kHalf;
    static __device__ __forceinline__ uint64_t pair(const uint32_t (&w)[kWords], int i) {
        return f32x2(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1]));
    }
};
template <> struct Raw<__nv_bfloat16> {
    static constexpr int kWords = kHalf / 2;
    static __device__ __forceinline__ uint64_t pair(const uint32_t (&w)[kWords], int i) {
        return f32x2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
    }
};
template <> struct Raw<__half> {
    static constexpr int kWords = kHalf / 2;
    static __device__ __forceinline__ uint64_t pair(const uint32_t (&w)[kWords], int i) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
        return f32x2(f.x, f.y);
    }
};

// Two values rounded through the cache dtype and back (the reference's `.to(dtype).float()`).
template <typename T> __device__ __forceinline__ uint64_t round_through2(uint64_t v);
template <> __device__ __forceinline__ uint64_t round_through2<float>(uint64_t v) { return v; }
template <> __device__ __forceinline__ uint64_t round_through2<__nv_bfloat16>(uint64_t v) {
    float a, b;
    f32x2_split(v, a, b);
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    const uint32_t u = *reinterpret_cast<const uint32_t *>(&h);
    return f32x2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
template <> __device__ __forceinline__ uint64_t round_through2<__half>(uint64_t v) {
    float a, b;
    f32x2_split(v, a, b);
    const float2 f = __half22float2(__floats2half2_rn(a, b));
    return f32x2(f.x, f.y);
}

// The power of two that brings a positive number's magnitude into [2^12, 2^13): exact products.  (Numbers
// below 2^-115 get 2^127; infinity and NaN get 2^-116.)
__device__ __forceinline__ float fit_power(float v) {
    const int e = (int)(__float_as_uint(v) >> 23);
    return __uint_as_float((uint32_t)min(254, 266 - e) << 23);
}

// 4 * (number of boundaries strictly below z), a byte offset into the tables of 16 floats.  The first two
// levels of the search compare with registers, the others with shared memory (one bank per entry).
template <int BITS> struct Search {
    float top, lo, hi;
    const float *table;
    __device__ __forceinline__ explicit Search(const float *bounds) : table(bounds) {
        top = bounds[(1 << (BITS - 1)) - 1];
        lo = BITS > 1 ? bounds[(1 << BITS) / 4 - 1] : 0.f;
        hi = BITS > 1 ? bounds[3 * (1 << BITS) / 4 - 1] : 0.f;
    }
    __device__ __forceinline__ uint32_t operator()(float z) const {
        const bool up = top < z;
        uint32_t o = up ? 2u << BITS : 0u;
        if (BITS > 1 && (up ? hi : lo) < z) o += 1u << BITS;
#pragma unroll
        for (int step = (1 << BITS) / 8; step > 0; step >>= 1)
            if (*reinterpret_cast<const float *>(reinterpret_cast<const char *>(table + step - 1) + o) < z) o += 4 * step;
        return o;
    }
};

// ORs code c (given as 4 * c) into place i of a bitstream of BITS-bit codes
template <int BITS, int N> __device__ __forceinline__ void put_code(uint32_t (&words)[N], int i, uint32_t c4) {
    const int bit = i * BITS, w = bit >> 5, sh = bit & 31;
    words[w] |= sh >= 2 ? c4 << (sh - 2) : c4 >> (2 - sh);
    if (sh + BITS > 32) words[w + 1] |= c4 >> (34 - sh);
}

struct PackTcShared {
    float bounds[16];
    uint32_t centers[16];  // f16 hi term | lo term << 16 of a scaled key centre
    float sq[kGroups][2][2][kUmmaRows];  // squared norms: [group][tile parity][half of the coordinates][vector]
    float big[kGroups][2][2][kUmmaRows];  // largest magnitudes of halves whose squared norm is zero
    float rs[kGroups][2][kUmmaRows];     // squared residual norms
    uint64_t bar_image[3], bar_mma[kGroups];
    uint32_t tmem;
};

template <typename T, int BITS, bool QJL>
__device__ __forceinline__ void encode(const PackTcArgs &a, const PackTcRole &r, PackTcShared &sm, uint32_t images, int cta, int n_ctas) {
    using R = Raw<T>;
    constexpr int kTermsX = sizeof(T) == 4 ? 2 : 1;
    const int tid = threadIdx.x, group = tid / kGroupThreads, warp = tid >> 5;
    const int vrow = tid & (kUmmaRows - 1);            // this thread's vector within the tile (= its TMEM lane)
    const int half = (tid >> 7) & 1;                   // which half of the coordinates it works on
    const uint32_t acc = sm.tmem + group * 256, a_hi = acc + 128, a_lo = acc + 192;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t my_acc = acc + lanes + kHalf * half, my_hi = a_hi + lanes + kHalf / 2 * half, my_lo = a_lo + lanes + kHalf / 2 * half;
    const uint32_t bar_mma = smem_u32(&sm.bar_mma[group]);
    const bool issuer = (tid & (kGroupThreads - 1)) == 0;
    bool timed_out = false;
    uint32_t mma_phase = 0;
    uint32_t landed = 0;  // issuer: the images seen in shared memory

    auto group_sync = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + group), "r"(kGroupThreads) : "memory"); };
    // Everybody has stored its part of A (and read the accumulators of the stage before): issue the MMAs.
    auto gemm_issue = [&](int stage, int terms) {
        tmem_st_wait();
        umma_fence_before();
        group_sync();
        if (issuer) {
            umma_fence_after();
            if (!(landed >> stage & 1)) {
                if (!mbar_wait(smem_u32(&sm.bar_image[stage]), 0)) timed_out = true;
                landed |= 1u << stage;
            }
            umma_issue(acc, a_hi, a_lo, images + stage * kUmmaImageBytes, terms);
            umma_commit(bar_mma);
        }
    };
    auto gemm_wait = [&]() {
        if (!mbar_wait(bar_mma, mma_phase)) timed_out = true;
        mma_phase ^= 1;
        __syncwarp();  // the issuer took its own path; tcgen05.ld is warp-collective
        umma_fence_after();
    };

    const int64_t n_vec = (int64_t)a.B * a.H * a.S;
    struct RowRef {
        const T *src;
        int64_t row;
        bool valid;
    };
    auto locate = [&](int tile) {  // this thread's vector of a tile: where it comes from, where it goes
        const int64_t vid = (int64_t)tile * kUmmaRows + vrow;
        RowRef ref;
        ref.valid = vid < n_vec;
        const int64_t v = ref.valid ? vid : 0;
        int t, h, b;
        if (n_vec <= 0x7fffffff) {  // (32-bit divisions are several times cheaper)
            const uint32_t q = (uint32_t)v / (uint32_t)a.S;
            t = (int)((uint32_t)v - q * a.S), b = (int)(q / (uint32_t)a.H), h = (int)(q - (uint32_t)b * a.H);
        } else {
            t = (int)(v % a.S), h = (int)((v / a.S) % a.H), b = (int)(v / ((int64_t)a.S * a.H));
        }
        ref.src = reinterpret_cast<const T *>(r.x) + b * r.sb + h * r.sh + (int64_t)t * r.st + kHalf * half;
        ref.row = b * a.cache_sb + h * a.cache_sh + a.pos0 + t;
        return ref;
    };
    uint32_t raw[R::kWords];  // this thread's half of the vector, as stored
    auto fetch = [&](const RowRef &ref) {
#pragma unroll
        for (int i = 0; i < R::kWords / 4; ++i) {
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(ref.src) + i);
            raw[4 * i] = v.x, raw[4 * i + 1] = v.y, raw[4 * i + 2] = v.z, raw[4 * i + 3] = v.w;
        }
    };
    // (keeps the compiler from holding the 64 converted values in registers from one use to the next)
    auto forget_conversions = [&]() {
        if (sizeof(T) == 2) {
#pragma unroll
            for (int i = 0; i < R::kWords; ++i) asm volatile("" : "+r"(raw[i]));
        }
    };
    const Search<BITS> search(sm.bounds);
    const int first = cta + n_ctas * group, stride = n_ctas * kGroups;
    RowRef cur = locate(first);
    if (first < a.n_tiles) fetch(cur);
    int parity = 0;
    for (int tile = first; tile < a.n_tiles; tile += stride, parity ^= 1) {
        // ---------------- stage 1: A = x (scaled).  The rows were requested while the last tile's MMAs ran.
        const bool more = tile + stride < a.n_tiles;
        RowRef nxt = cur;
        float ss;
        {
            uint64_t s0 = 0, s1 = 0;
#pragma unroll
            for (int i = 0; i < kHalf / 2; i += 2) {
                const uint64_t p0 = R::pair(raw, i), p1 = R::pair(raw, i + 1);
                s0 = f32x2_fma(p0, p0, s0), s1 = f32x2_fma(p1, p1, s1);
            }
            float s[4];
            f32x2_split(s0, s[0], s[1]), f32x2_split(s1, s[2], s[3]);
            ss = (s[0] + s[1]) + (s[2] + s[3]);
        }
        float (*sq)[kUmmaRows] = sm.sq[group][parity], (*big)[kUmmaRows] = sm.big[group][parity];
        sq[half][vrow] = ss;
        float nrm, inv;  // |x|; z = accumulator * inv
        if constexpr (!std::is_same<T, __half>::value) {
            if (ss == 0.f) {
                float m = 0.f;
#pragma unroll
                for (int i = 0; i < kHalf / 2; ++i) {
                    float u, v;
                    f32x2_split(R::pair(raw, i), u, v);
                    m = fmaxf(m, fmaxf(fabsf(u), fabsf(v)));
                }
                big[half][vrow] = m;
            }
            group_sync();
            forget_conversions();
            nrm = sqrtf(sq[0][vrow] + sq[1][vrow]);
            float scale = fit_power(nrm);
            if (nrm != 0.f) {  // (scale * nrm is exact and lies in [2^12, 2^13))
                inv = r.unscale / (scale * nrm);
            } else {  // a zero vector, or one whose squares underflow: taken as it is (norm 1)
                scale = fit_power(fmaxf(big[0][vrow], big[1][vrow]));
                inv = r.unscale / scale;
            }
            const uint64_t scale2 = f32x2(scale, scale);
            __syncwarp();  // (tcgen05.st is warp-collective)
#pragma unroll
            for (int c = 0; c < kHalf / 16; ++c) {
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint64_t u = f32x2_mul(R::pair(raw, 8 * c + i), scale2);
                    if (kTermsX == 2) {
                        split_half2(u, hi[i], lo[i]);
                    } else {
                        float u0, u1;
                        f32x2_split(u, u0, u1);
                        hi[i] = half2_bits(u0, u1);
                    }
                }
                tmem_st8(my_hi + 8 * c, hi);
                if (kTermsX == 2) tmem_st8(my_lo + 8 * c, lo);
            }
            gemm_issue(0, kTermsX);
        } else {
            __syncwarp();
#pragma unroll
            for (int c = 0; c < kHalf / 16; ++c) {
                uint32_t hi[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) hi[i] = raw[8 * c + i];
                tmem_st8(my_hi + 8 * c, hi);
            }
            gemm_issue(0, 1);
            nrm = sqrtf(sq[0][vrow] + sq[1][vrow]);
            inv = nrm > 0.f ? r.unscale / nrm : r.unscale;
        }
        const float safe = nrm > 0.f ? nrm : 1.f;
        forget_conversions();
        if (!QJL && more) {  // the rows are stored: fetch the next tile's under the MMAs
            nxt = locate(tile + stride);
            fetch(nxt);
        }
        gemm_wait();

        // ---------------- epilogue 1: this thread's accumulators -> codes (and, for the sketch, A = centres[codes])
        constexpr int kWords = 2 * BITS;
        uint32_t words[kWords + 1];
#pragma unroll
        for (int w = 0; w <= kWords; ++w) words[w] = 0;
        const uint64_t inv2 = f32x2(inv, inv);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            uint32_t z[32];
            tmem_ld32(my_acc + 32 * q, z);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int e = 16 * c + 2 * i;
                    float z0, z1;
                    f32x2_split(f32x2_mul(f32x2(__uint_as_float(z[e]), __uint_as_float(z[e + 1])), inv2), z0, z1);
                    const uint32_t c0 = search(z0), c1 = search(z1);
                    put_code<BITS>(words, 32 * q + e, c0), put_code<BITS>(words, 32 * q + e + 1, c1);
                    if (QJL) {
                        const uint32_t t0 = *reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(sm.centers) + c0);
                        const uint32_t t1 = *reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(sm.centers) + c1);
                        hi[i] = __byte_perm(t0, t1, 0x5410), lo[i] = __byte_perm(t0, t1, 0x7632);
                    }
                }
                if (QJL) tmem_st8(my_hi + 16 * q + 8 * c, hi), tmem_st8(my_lo + 16 * q + 8 * c, lo);
            }
        }
        const uint16_t nh = tq_float_to_half_bits(safe);
        if (QJL) gemm_issue(1, 2);
        if (cur.valid) {
            uint32_t *dst = reinterpret_cast<uint32_t *>(r.codes + cur.row * (int64_t)(16 * BITS) + half * (8 * BITS));
            if constexpr (kWords % 4 == 0) {
#pragma unroll
                for (int w = 0; w < kWords; w += 4)
                    *reinterpret_cast<uint4 *>(dst + w) = make_uint4(words[w], words[w + 1], words[w + 2], words[w + 3]);
            } else {
#pragma unroll
                for (int w = 0; w < kWords; w += 2) *reinterpret_cast<uint2 *>(dst + w) = make_uint2(words[w], words[w + 1]);
            }
            if (half == 0) r.norms[cur.row] = nh;
        }
        if constexpr (QJL) {
            gemm_wait();
            // ---------------- epilogue 2: the residual against the dtype-rounded reconstruction
            const float nf = tq_half_bits_to_float(nh) * a.unscale2, scale = fit_power(safe) * a.res_scale;
            const uint64_t nf2 = f32x2(nf, nf), scale2 = f32x2(scale, scale);
            uint64_t rs2 = 0;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                uint32_t y[32];
                tmem_ld32(my_acc + 32 * q, y);
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t hi[8], lo[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int e = 16 * c + 2 * i;
                        const uint64_t rec = round_through2<T>(f32x2_mul(f32x2(__uint_as_float(y[e]), __uint_as_float(y[e + 1])), nf2));
                        const uint64_t res = f32x2_sub(R::pair(raw, 16 * q + 8 * c + i), rec);
                        rs2 = f32x2_fma(res, res, rs2);
                        split_half2(f32x2_mul(res, scale2), hi[i], lo[i]);
                    }
                    tmem_st8(my_hi + 16 * q + 8 * c, hi), tmem_st8(my_lo + 16 * q + 8 * c, lo);
                }
            }
            float rs, rs_hi;
            f32x2_split(rs2, rs, rs_hi);
            sm.rs[group][half][vrow] = rs + rs_hi;
            // ---------------- stage 3: projection, sign bits
            gemm_issue(2, 2);
            const float rn = sqrtf(sm.rs[group][0][vrow] + sm.rs[group][1][vrow]);
            if (more) {  // the residual is stored: fetch the next tile's rows under the MMAs
                nxt = locate(tile + stride);
                fetch(nxt);
            }
            gemm_wait();
            uint32_t sg[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                uint32_t p[32];
                tmem_ld32(my_acc + 32 * q, p);
                uint32_t neg = 0;  // sign bits, shifted in from element 31 down to 0; -0 counts as +0
#pragma unroll
                for (int i = 30; i >= 0; i -= 2) {
                    float p0, p1;
                    f32x2_split(f32x2_fma(f32x2(__uint_as_float(p[i]), __uint_as_float(p[i + 1])), f32x2(1.f, 1.f), 0ull), p0, p1);
                    neg = __funnelshift_l(__float_as_uint(p1), neg, 1);
                    neg = __funnelshift_l(__float_as_uint(p0), neg, 1);
                }
                sg[q] = rn < INFINITY ? ~neg : 0u;  // (an infinite or undefined residual makes every projection undefined)
            }
            if (cur.valid) {
                *reinterpret_cast<uint2 *>(a.signs + cur.row * 16 + 8 * half) = make_uint2(sg[0], sg[1]);
                if (half == 0) a.rnorms[cur.row] = tq_float_to_half_bits(rn > 0.f ? rn : 1.f);
            }
        }
        cur = nxt;
    }
    if (timed_out) atomicExch(a.error_flag, 3);
}

template <typename T, int BITS, bool QJL>
__global__ void __launch_bounds__(kThreads, 1) tq_pack_tc_kernel(const __grid_constant__ PackTcArgs a) {
    constexpr int KEY_BITS = QJL ? BITS - 1 : BITS;
    extern __shared__ uint8_t smem_raw[];
    __shared__ PackTcShared sm;
    const uint32_t images = (smem_u32(smem_raw) + 1023u) & ~1023u;  // swizzle atoms need 1024-byte alignment
    const int tid = threadIdx.x, warp = tid >> 5;
    const bool keys = (int)blockIdx.x < a.key_ctas;
    const PackTcRole &r = a.role[keys ? 0 : 1];
    if (tid < 16) {
        sm.bounds[tid] = r.bounds[tid];
        if (QJL) {
            const float c = a.centers[tid] * a.cen_scale;
            const __half hi = __float2half_rn(c), lo = __float2half_rn(c - __half2float(hi));
            sm.centers[tid] = (uint32_t)__half_as_ushort(hi) | (uint32_t)__half_as_ushort(lo) << 16;
        }
    }
    if (warp == 0) {  // all of TMEM: one CTA per SM
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sm.tmem)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (tid == 0) {
        for (int i = 0; i < 3; ++i) mbar_init(smem_u32(&sm.bar_image[i]), 1);
        for (int i = 0; i < kGroups; ++i) mbar_init(smem_u32(&sm.bar_mma[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        umma_load_image(images, r.image, smem_u32(&sm.bar_image[0]));  // (every CTA has at least one tile)
        if (QJL && keys) {
            umma_load_image(images + kUmmaImageBytes, a.image2, smem_u32(&sm.bar_image[1]));
            umma_load_image(images + 2 * kUmmaImageBytes, a.image3, smem_u32(&sm.bar_image[2]));
        }
    }
    umma_fence_before();
    __syncthreads();
    umma_fence_after();
    if (keys) encode<T, KEY_BITS, QJL>(a, r, sm, images, blockIdx.x, a.key_ctas);
    else encode<T, BITS, false>(a, r, sm, images, blockIdx.x - a.key_ctas, gridDim.x - a.key_ctas);
    umma_fence_before();
    __syncthreads();
    if (warp == 0) {
        umma_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(sm.tmem), "r"(512));
    }
}

}  // namespace

float tq_fit_power(float largest) {
    if (!(largest > 0.f) || !isfinite(largest)) return 1.f;
    int e;
    frexpf(largest, &e);  // largest < 2^e
    return ldexpf(1.f, e < -100 ? 114 : e > 100 ? -86 : 14 - e);
}

// Host: the 64 KB shared-memory image of a [128 x 128] K-major operand `m[row][k]`, times a power of two, in
// two f16 terms of two 64-wide slabs each, with the 128-byte swizzle.  Returns what undoes the power of two.
float tq_build_operand_image(const float *m, uint16_t *image) {
    float largest = 0.f;
    for (int i = 0; i < TQ_D * TQ_D; ++i) largest = fmaxf(largest, fabsf(m[i]));
    const float scale = tq_fit_power(largest);
    for (int row = 0; row < TQ_D; ++row)
        for (int k = 0; k < TQ_D; ++k) {
            const float v = m[(size_t)row * TQ_D + k] * scale;
            const __half hi = __float2half_rn(v), lo = __float2half_rn(v - __half2float(hi));
            const int off = umma_operand_offset(row, k) / 2;
            memcpy(image + off, &hi, 2);
            memcpy(image + kUmmaTermBytes / 2 + off, &lo, 2);
        }
    return 1.f / scale;
}

template <typename T, int BITS, bool QJL>
static cudaError_t launch_tc(const PackTcArgs &a, int grid, int device, cudaStream_t stream) {
    const int smem = (QJL && a.key_ctas ? 3 : 1) * kUmmaImageBytes + 1024;
    // the attribute belongs to the (kernel, device) pair: one flag per device of this instantiation
    static bool configured[TQ_MAX_DEVICES] = {};
    if (device < 0 || device >= TQ_MAX_DEVICES) return cudaErrorInvalidDevice;
    if (!configured[device]) {
        cudaError_t e = cudaFuncSetAttribute(tq_pack_tc_kernel<T, BITS, QJL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (QJL ? 3 : 1) * kUmmaImageBytes + 1024);
        if (e != cudaSuccess) return e;
        configured[device] = true;
    }
    tq_pack_tc_kernel<T, BITS, QJL><<<grid, kThreads, smem, stream>>>(a);
    return cudaGetLastError();
}

int32_t tq_launch_pack_tc(tq_ctx *ctx, const tq_dense_desc *k, const tq_dense_desc *v, int32_t n_tokens,
                          const tq_cache_desc *cache, int32_t pos0, cudaStream_t stream) {
    const int esize = v->dtype == TQ_DTYPE_F32 ? 4 : 2;
    PackTcArgs a = {};
    for (int i = 0; i < 2; ++i) {
        const tq_dense_desc *x = i == 0 ? k : v;
        if (!x) continue;
        if (((uintptr_t)x->data & 15) || ((x->stride_b * esize) & 15) || ((x->stride_h * esize) & 15) || ((x->stride_t * esize) & 15))
            return TQ_ERR_UNSUPPORTED;
        PackTcRole &r = a.role[i];
        const tq_ctx::Image &image = i == 0 ? ctx->img_rot_k : ctx->img_rot_v;
        r.x = x->data, r.sb = x->stride_b, r.sh = x->stride_h, r.st = x->stride_t;
        r.codes = i == 0 ? cache->k_codes : cache->v_codes, r.norms = i == 0 ? cache->k_norms : cache->v_norms;
        r.image = image.data, r.unscale = image.unscale;
        r.bounds = i == 0 ? ctx->bounds_k : ctx->bounds_v;
    }
    const bool qjl = ctx->use_qjl && k;
    a.B = cache->batch, a.H = cache->kv_heads, a.S = n_tokens, a.pos0 = pos0;
    a.cache_sb = cache->stride_b, a.cache_sh = cache->stride_h;
    a.error_flag = ctx->error_flag;
    a.image2 = ctx->img_rot_kt.data, a.image3 = ctx->img_qjl.data;
    a.unscale2 = ctx->img_rot_kt.unscale / ctx->cen_k_scale;
    a.cen_scale = ctx->cen_k_scale, a.res_scale = ctx->res_scale;
    a.centers = ctx->centers_k;
    a.signs = cache->k_signs, a.rnorms = cache->k_rnorms;
    const int64_t n_vec = (int64_t)a.B * a.H * a.S;
    a.n_tiles = (int)((n_vec + kUmmaRows - 1) / kUmmaRows);
    // One CTA per SM.  With tiles enough for all of them, keys with the sketch get the share of the SMs that
    // their cost asks for; with few tiles each side gets a CTA per tile.
    const int sms = ctx->sm_count;
    int key_ctas = !k ? 0 : qjl ? sms * 7 / 10 : sms / 2, val_ctas = sms - key_ctas;
    if (k && a.n_tiles <= sms / 2) key_ctas = val_ctas = a.n_tiles;
    key_ctas = key_ctas < a.n_tiles ? key_ctas : a.n_tiles, val_ctas = val_ctas < a.n_tiles ? val_ctas : a.n_tiles;
    a.key_ctas = key_ctas;
    const int grid = key_ctas + val_ctas;
    cudaError_t e = cudaErrorInvalidValue;
#define TQ_TC_CASE(T)                                                                                                     \
    switch (ctx->bits) {                                                                                                  \
        case 2: e = qjl ? launch_tc<T, 2, true>(a, grid, ctx->device, stream) : launch_tc<T, 2, false>(a, grid, ctx->device, stream); break; \
        case 3: e = qjl ? launch_tc<T, 3, true>(a, grid, ctx->device, stream) : launch_tc<T, 3, false>(a, grid, ctx->device, stream); break; \
        case 4: e = qjl ? launch_tc<T, 4, true>(a, grid, ctx->device, stream) : launch_tc<T, 4, false>(a, grid, ctx->device, stream); break; \
        default: return TQ_ERR_UNSUPPORTED;                                                                               \
    }
    if (v->dtype == TQ_DTYPE_F32) {
        TQ_TC_CASE(float)
    } else if (v->dtype == TQ_DTYPE_F16) {
        TQ_TC_CASE(__half)
    } else {
        TQ_TC_CASE(__nv_bfloat16)
    }
#undef TQ_TC_CASE
    tq_prof_count(ctx, 1);
    TQ_CUDA_CHECK(e);
    return TQ_OK;
}
