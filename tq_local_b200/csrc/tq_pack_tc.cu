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
// One CTA of 32 warps per SM: two groups of sixteen warps, each walking tiles of 128 vectors on its own, so
// that one group's CUDA-core work runs beside the other group's MMAs.  Four threads share a vector (32
// coordinates each).  The A operand is written to TMEM (tcgen05.st, no swizzle, no bank conflicts), so
// shared memory is left for the matrices: R_k (stage 1; stage 2 reads the same image transposed) and S stay
// resident and nothing is reloaded between the stages.  Rows of 16-bit vectors come through shared memory, copied
// by all warps, 16 bytes a lane and sixteen lanes to a row: read by the threads that own them they took 2048 of the 4500
// L1 wavefronts of a value tile, which bounded it, and as a bulk copy per row they are issued lane by lane by the warps that are
// waited for (2 x 8 x 32768 bf16 vectors a tensor 220 us instead of 209).  A group owns 256 TMEM columns: 128 of accumulator, 64 for each term of A.
// The first CTAs of a launch encode keys and the others values, in the proportion of their costs.
// What bounds it is the CUDA-core work between the contractions: time stamps in one CTA show both groups in step, so that their
// instructions share the schedulers, then their MMAs follow one another (1150 cycles for sixteen, 1660 for 24, alone or beside
// shared-memory and TMEM traffic).  The issuing thread is elected in a converged warp and the accumulator's address is
// uniform, which leaves an instruction or two per MMA: with a thread chosen by its index the operands went through vector
// registers, and sixteen MMAs took 2000 - 2400 cycles to issue between the other warps' instructions.
// 2 x 8 x 32768 keys and values, 4 bits with the sketch: bf16 242 -> 203 us, f16 252 -> 194; 3 bits 259 -> 215, 269 -> 200; 4 bits
// without 142 -> 128, 124 -> 114 (before: look-ups one by one, bulk copies, issue by index).  All sixteen warps of a
// group on one tile at a time with dedicated loading and issuing warps, two tiles in flight: 262 us and more, too few warps to hide the
// latencies of a phase.
// Every mbarrier wait is bounded and reports through the device status word.
#include <math.h>
#include <string.h>

#include <type_traits>

#include "tq_common.cuh"
#include "tq_umma.cuh"

namespace {

constexpr int kGroups = 2;
constexpr int kGroupThreads = 512;
constexpr int kThreads = kGroups * kGroupThreads;
constexpr int kMaxCells = 64;
constexpr int kCellCopies = 16;  // of the search table: lane l reads copy l % 16, so an 8-byte look-up has no bank conflicts
constexpr int kParts = kGroupThreads / kUmmaRows;  // threads per vector
constexpr int kCoords = TQ_D / kParts;             // coordinates per thread

struct PackTcRole {
    const void *x;
    int64_t sb, sh, st;
    uint8_t *codes;
    uint16_t *norms;
    const uint16_t *image;  // the rotation
    float unscale;
    const float *bounds;    // 16 floats, padded with +inf
    tq_ctx::Grid grid;      // the search grid of these boundaries
};
struct PackTcArgs {
    PackTcRole role[2];  // keys, values
    int key_ctas;        // CTAs [0, key_ctas) encode keys, the others values
    VectorIndex vec;
    int pos0;
    int64_t cache_sb, cache_sh;
    int n_tiles;
    int *error_flag;
    // the sketch
    const uint16_t *image_s;          // S (projection)
    float unscale2;                   // undoes the scales of R_k and of the centres
    float cen_scale, res_scale;
    const float *centers;  // 16 floats
    uint8_t *signs;
    uint16_t *rnorms;
};

template <typename T> struct Raw;  // how many 32-bit words a thread's coordinates take, and pairs of them as floats
template <> struct Raw<float> {
    static constexpr int kWords = kCoords;
    static __device__ __forceinline__ uint64_t pair(const uint32_t (&w)[kWords], int i) {
        return f32x2(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1]));
    }
};
template <> struct Raw<__nv_bfloat16> {
    static constexpr int kWords = kCoords / 2;
    static __device__ __forceinline__ uint64_t pair(const uint32_t (&w)[kWords], int i) {
        return f32x2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
    }
};
template <> struct Raw<__half> {
    static constexpr int kWords = kCoords / 2;
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

// MUL * (number of boundaries strictly below z).  One or two bits: binary search in registers.  More: z's cell
// in a uniform grid gives the number of boundaries in the cells before it and the one boundary that may lie
// in its own (tq_fit_grid makes sure that there is no second one); the cell is a monotone function of z and
// the boundaries' cells are formed by the same instructions, so the answer is that of comparing with all of them.
// Against a binary search in shared memory this saves five instructions a coordinate at four bits.  Codebooks that no grid
// separates take that search (GRID false: four dependent loads, whose sixteen words lie in sixteen banks): 4 x 8 x 32768
// bf16 keys and values, 4 bits with the sketch, 668 us against 480 (12 ms in the CUDA-core encoder).
__device__ __forceinline__ uint32_t grid_cell(float z, const tq_ctx::Grid &g) {  // + 0x4B000000
    float t;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;\n" : "=f"(t) : "f"(z), "f"(g.scale), "f"(g.shift));  // (NaN: 0)
    return __float_as_uint(fmaf(t, g.last, 8388608.f));
}
template <int BITS, int MUL, bool GRID> struct Search {
    float b0, b1, b2;
    tq_ctx::Grid grid;
    uint32_t table;  // of cells, or the boundaries
    __device__ __forceinline__ Search(const float *bounds, const uint2 *cells, const tq_ctx::Grid &g) : grid(g) {
        b0 = bounds[0], b1 = bounds[1], b2 = bounds[2];
        table = GRID ? smem_u32(cells) + 8 * (threadIdx.x % kCellCopies) - (0x4B000000u << 7) : smem_u32(bounds);
    }
    __device__ __forceinline__ bool below(uint32_t offset, float z) const {  // the boundary at that byte offset
        float b;
        asm("ld.shared.f32 %0, [%1];\n" : "=f"(b) : "r"(table + offset));
        return b < z;
    }
    // Eight coordinates at a time: eight look-ups under way and no more registers.  (Written one by one, the look-ups of 32 coordinates
    // were all moved ahead of the comparisons, whose outcomes were then packed into registers and spilled: twice 8 x 32768 bf16 keys
    // and values 234 us instead of 203, eight at a time with the comparison as a predicated instruction 236.)
    __device__ __forceinline__ void operator()(const float (&z)[8], uint32_t *code) const {
        if (BITS == 1) {
#pragma unroll
            for (int e = 0; e < 8; ++e) code[e] = b0 < z[e] ? MUL : 0u;
        } else if (BITS == 2) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const bool up = b1 < z[e];
                code[e] = (up ? 2u * MUL : 0u) + ((up ? b2 : b0) < z[e] ? MUL : 0u);
            }
        } else if (!GRID) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                uint32_t c = 0;  // (four times the boundaries known to be below)
                if (BITS == 4) c = below(4 * 7, z[e]) ? 32u : 0u;
                c += below(c + 4 * 3, z[e]) ? 16u : 0u;
                c += below(c + 4 * 1, z[e]) ? 8u : 0u;
                c += below(c, z[e]) ? 4u : 0u;
                code[e] = c / 4 * MUL;
            }
        } else {
            uint32_t bound[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
                asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];\n" : "=r"(bound[e]), "=r"(code[e]) : "r"(grid_cell(z[e], grid) * (8u * kCellCopies) + table));
#pragma unroll
            for (int e = 0; e < 8; ++e)
                code[e] += __uint_as_float(bound[e]) < z[e] ? MUL : 0u;
        }
    }
};
// Fills the grid's table (all threads of the CTA; barriers around it are the caller's).
__device__ __forceinline__ void build_cells(uint2 *cells, const float *bounds, int n_bounds, const tq_ctx::Grid &g, uint32_t mul) {
    for (int i = threadIdx.x; i < kCellCopies * ((int)g.last + 1); i += kThreads) {
        const int c = i / kCellCopies;
        uint32_t below = 0;
        float mine = INFINITY;
        for (int e = 0; e < n_bounds; ++e) {
            const int at = (int)(grid_cell(bounds[e], g) - 0x4B000000u);
            below += at < c ? mul : 0u;
            if (at == c) mine = bounds[e];
        }
        cells[i] = make_uint2(__float_as_uint(mine), below);
    }
}

// 32 codes of BITS bits (times MUL, a power of two) as a bitstream, LSB first, sixteen codes at a time.
template <int BITS, int MUL> __device__ __forceinline__ void put_codes(uint32_t (&words)[BITS], int q, const uint32_t (&c)[16]) {
    constexpr int kPer = BITS == 3 ? 8 : BITS == 4 ? 8 : 16;  // codes that fit one register
    uint32_t piece[16 / kPer];
#pragma unroll
    for (int p = 0; p < 16 / kPer; ++p) {
        uint32_t v = c[kPer * p + kPer - 1];
        if (MUL > 1 && BITS != 3) v /= MUL;
#pragma unroll
        for (int i = kPer - 2; i >= 0; --i) v = v * (1u << BITS) + (MUL > 1 && BITS != 3 ? c[kPer * p + i] / MUL : c[kPer * p + i]);
        piece[p] = MUL > 1 && BITS == 3 ? v / MUL : v;
    }
    if (BITS == 1) {
        if (q == 0) words[0] = piece[0];
        else words[0] |= piece[0] << 16;
    } else if (BITS == 2) {
        words[q % BITS] = piece[0];
    } else if (BITS == 4) {
        words[(2 * q) % BITS] = piece[0], words[(2 * q + 1) % BITS] = piece[1 % (16 / kPer)];
    } else {  // 24-bit pieces
        const uint32_t p0 = piece[0], p1 = piece[1 % (16 / kPer)];
        if (q == 0) {
            words[0] = p0 | p1 << 24, words[1 % BITS] = p1 >> 8;
        } else {
            words[1 % BITS] |= p0 << 16, words[2 % BITS] = p0 >> 16 | p1 << 8;
        }
    }
}

struct PackTcShared {
    uint2 cells[kMaxCells * kCellCopies];  // {boundary, codes below}, see Search
    float bounds[16];
    uint32_t centers[16];  // f16 hi term | lo term << 16 of a scaled key centre
    float sq[kGroups][2][kParts][kUmmaRows];   // squared norms: [group][tile parity][part of the coordinates][vector]
    float big[kGroups][2][kParts][kUmmaRows];  // largest magnitudes of parts whose squared norm is zero
    float rs[kGroups][kParts][kUmmaRows];         // squared residual norms
    uint64_t bar_image[2], bar_mma[kGroups], bar_rows[kGroups][4];
    uint32_t tmem;
};

template <typename T, int BITS, bool QJL, bool GRID>
__device__ __forceinline__ void encode(const PackTcArgs &a, const PackTcRole &r, PackTcShared &sm, uint32_t images, uint32_t staged, int cta, int n_ctas) {
    using R = Raw<T>;
    constexpr int kTermsX = sizeof(T) == 4 ? 2 : 1;
    const int tid = threadIdx.x, group = tid / kGroupThreads, warp = tid >> 5;
    const int vrow = tid & (kUmmaRows - 1);            // this thread's vector within the tile (= its TMEM lane)
    const int part = (tid / kUmmaRows) % kParts;       // which part of the coordinates it works on
    const uint32_t acc = __shfl_sync(0xffffffffu, sm.tmem + group * 256, 0), a_hi = acc + 128, a_lo = acc + 192;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t my_acc = acc + lanes + kCoords * part, my_hi = a_hi + lanes + kCoords / 2 * part, my_lo = my_hi + 64;
    const uint32_t bar_mma = smem_u32(&sm.bar_mma[group]);
    const bool issuer = __shfl_sync(0xffffffffu, tid & (kGroupThreads - 1), 0) == 0;  // a group's first warp
    uint32_t mma_phase = 0;
    uint32_t landed = 0;  // issuer: the images seen in shared memory

    auto group_sync = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + group), "r"(kGroupThreads) : "memory"); };
    // Everybody has stored its part of A (and read the accumulators of the stage before): issue the MMAs.
    auto gemm_issue = [&](int image, auto terms, auto transposed) {
        tmem_st_wait();
        umma_fence_before();
        group_sync();
        if (issuer && elect_one()) {  // (always the same thread of the warp: `landed`, and what a commit covers, are its own)
            umma_fence_after();
            if (!(landed >> image & 1)) {
                if (!mbar_wait(smem_u32(&sm.bar_image[image]), 0)) atomicExch(a.error_flag, 3);
                landed |= 1u << image;
            }
            umma_issue<decltype(terms)::value, decltype(transposed)::value>(acc, a_hi, a_lo, images + image * kUmmaImageBytes);
            umma_commit(bar_mma);
        }
    };
    auto gemm_wait = [&]() {
        if (!mbar_wait(bar_mma, mma_phase)) atomicExch(a.error_flag, 3);
        mma_phase ^= 1;
        __syncwarp();  // the issuer took its own path; tcgen05.ld is warp-collective
        umma_fence_after();
    };
    const std::integral_constant<int, 1> one_term;
    const std::integral_constant<int, 2> two_terms;

    // Rows of 16-bit vectors are staged in shared memory (each warp requests eight of its quadrant's); fp32
    // rows, for which there is no room, come straight from global memory.
    constexpr bool kStaged = sizeof(T) == 2;
    const uint32_t my_stage = staged + group * kStageBytes + vrow * kStagePitch, bar_rows = smem_u32(&sm.bar_rows[group][warp & 3]);
    uint32_t raw[R::kWords];  // this thread's part of the vector, as stored
    int64_t row = 0;          // the vector's cache row (< 0: no vector)
    uint32_t rows_phase = 0;
    auto request = [&](int tile) {  // (the group is done with the rows before)
        const int64_t vid = (int64_t)tile * kUmmaRows + vrow;
        const bool valid = vid < a.vec.n;
        int t, h, b;
        vector_at(a.vec, valid ? vid : 0, b, h, t);
        const T *src = reinterpret_cast<const T *>(r.x) + b * r.sb + h * r.sh + (int64_t)t * r.st;
        row = valid ? b * a.cache_sb + h * a.cache_sh + a.pos0 + t : -1;
        if constexpr (kStaged) {
            const int lane = tid & 31;
#pragma unroll
            for (int i = 0; i < 8; i += 2) {  // eight of the warp's 32 rows (the other parts' warps take the others), sixteen lanes to a row
                const int from = 8 * part + i + (lane >> 4);
                const uint64_t at = __shfl_sync(0xffffffffu, reinterpret_cast<uint64_t>(src), from);
                async_copy16(my_stage + (from - lane) * kStagePitch + 16 * (lane & 15), reinterpret_cast<const void *>(at + 16 * (lane & 15)));
            }
            async_arrive(bar_rows);
        } else {
#pragma unroll
            for (int i = 0; i < R::kWords / 4; ++i) {
                const uint4 v = __ldg(reinterpret_cast<const uint4 *>(src + kCoords * part) + i);
                raw[4 * i] = v.x, raw[4 * i + 1] = v.y, raw[4 * i + 2] = v.z, raw[4 * i + 3] = v.w;
            }
        }
    };
    auto read_rows = [&]() {
        if constexpr (kStaged) {
#pragma unroll
            for (int i = 0; i < R::kWords / 4; ++i) {
                const uint4 v = lds128(my_stage + 2 * kCoords * part + 16 * i);
                raw[4 * i] = v.x, raw[4 * i + 1] = v.y, raw[4 * i + 2] = v.z, raw[4 * i + 3] = v.w;
            }
        }
    };
    auto rows_wait = [&]() {
        if constexpr (kStaged) {
            if (!mbar_wait(bar_rows, rows_phase)) atomicExch(a.error_flag, 3);
            rows_phase ^= 1;
        }
    };
    // (keeps the compiler from holding the converted values in registers from one use to the next)
    auto forget_conversions = [&]() {
        if (sizeof(T) == 2) {
#pragma unroll
            for (int i = 0; i < R::kWords; ++i) asm volatile("" : "+r"(raw[i]));
        }
    };
    const Search<BITS, QJL ? 4 : 1, GRID> search(sm.bounds, sm.cells, r.grid);
    const int first = cta + n_ctas * group, stride = n_ctas * kGroups;
    if (first < a.n_tiles) request(first);
    int parity = 0;
    for (int tile = first; tile < a.n_tiles; tile += stride, parity ^= 1) {
        // ---------------- stage 1: A = x (scaled).  The rows were requested while the last tile's MMAs ran.
        const bool more = tile + stride < a.n_tiles;
        const int64_t my_row = row;
        rows_wait();
        read_rows();
        float ss;
        {
            uint64_t s0 = 0, s1 = 0;
#pragma unroll
            for (int i = 0; i < kCoords / 2; i += 2) {
                const uint64_t p0 = R::pair(raw, i), p1 = R::pair(raw, i + 1);
                s0 = f32x2_fma(p0, p0, s0), s1 = f32x2_fma(p1, p1, s1);
            }
            float s[4];
            f32x2_split(s0, s[0], s[1]), f32x2_split(s1, s[2], s[3]);
            ss = (s[0] + s[1]) + (s[2] + s[3]);
        }
        float (*sq)[kUmmaRows] = sm.sq[group][parity], (*big)[kUmmaRows] = sm.big[group][parity];
        sq[part][vrow] = ss;
        float nrm, inv;  // |x|; z = accumulator * inv
        auto norm = [&]() { return sqrtf((sq[0][vrow] + sq[1][vrow]) + (sq[2][vrow] + sq[3][vrow])); };
        if constexpr (!std::is_same<T, __half>::value) {
            if (ss == 0.f) {
                float m = 0.f;
#pragma unroll
                for (int i = 0; i < kCoords / 2; ++i) {
                    float u, v;
                    f32x2_split(R::pair(raw, i), u, v);
                    m = fmaxf(m, fmaxf(fabsf(u), fabsf(v)));
                }
                big[part][vrow] = m;
            }
            group_sync();
            forget_conversions();
            nrm = norm();
            float scale = fit_power(nrm);
            if (nrm != 0.f) {  // (scale * nrm is exact and lies in [2^12, 2^13))
                inv = r.unscale / (scale * nrm);
            } else {  // a zero vector, or one whose squares underflow: taken as it is (norm 1)
                scale = fit_power(fmaxf(fmaxf(big[0][vrow], big[1][vrow]), fmaxf(big[2][vrow], big[3][vrow])));
                inv = r.unscale / scale;
            }
            const uint64_t scale2 = f32x2(scale, scale);
            __syncwarp();  // (tcgen05.st is warp-collective)
#pragma unroll
            for (int c = 0; c < kCoords / 16; ++c) {
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
            gemm_issue(0, std::integral_constant<int, kTermsX>(), std::false_type());
        } else {
            __syncwarp();
#pragma unroll
            for (int c = 0; c < kCoords / 16; ++c) {
                uint32_t hi[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) hi[i] = raw[8 * c + i];
                tmem_st8(my_hi + 8 * c, hi);
            }
            gemm_issue(0, one_term, std::false_type());
            nrm = norm();
            inv = nrm > 0.f ? r.unscale / nrm : r.unscale;
        }
        const float safe = nrm > 0.f ? nrm : 1.f;
        forget_conversions();
        if (!QJL && more) request(tile + stride);  // everybody has read its rows: request the next tile's under the MMAs
        gemm_wait();

        // ---------------- epilogue 1: this thread's accumulators -> codes (and, for the sketch, A = centres[codes])
        uint32_t words[BITS];
        const uint64_t inv2 = f32x2(inv, inv);
#pragma unroll
        for (int q = 0; q < kCoords / 16; ++q) {
            uint32_t z[16], code[16];
            tmem_ld16(my_acc + 16 * q, z);
#pragma unroll
            for (int h = 0; h < 16; h += 8) {
                float x[8];
#pragma unroll
                for (int e = 0; e < 8; e += 2)
                    f32x2_split(f32x2_mul(f32x2(__uint_as_float(z[h + e]), __uint_as_float(z[h + e + 1])), inv2), x[e], x[e + 1]);
                search(x, code + h);
            }
            put_codes<BITS, QJL ? 4 : 1>(words, q, code);
            if (QJL) {
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint32_t t0 = *reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(sm.centers) + code[2 * i]);
                    const uint32_t t1 = *reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(sm.centers) + code[2 * i + 1]);
                    hi[i] = __byte_perm(t0, t1, 0x5410), lo[i] = __byte_perm(t0, t1, 0x7632);
                }
                tmem_st8(my_hi + 8 * q, hi), tmem_st8(my_lo + 8 * q, lo);
            }
        }
        const uint16_t nh = tq_float_to_half_bits(safe);
        if (QJL) gemm_issue(0, two_terms, std::true_type());
        if (my_row >= 0) {
            uint32_t *dst = reinterpret_cast<uint32_t *>(r.codes + my_row * (16 * BITS)) + BITS * part;
            if constexpr (BITS == 4) *reinterpret_cast<uint4 *>(dst) = make_uint4(words[0], words[1], words[2], words[3]);
            else if constexpr (BITS == 2) *reinterpret_cast<uint2 *>(dst) = make_uint2(words[0], words[1]);
            else {
#pragma unroll
                for (int w = 0; w < BITS; ++w) dst[w] = words[w];
            }
            if (part == 0) r.norms[my_row] = nh;
        }
        if constexpr (QJL) {
            read_rows();  // (again: cheaper than holding them through epilogue 1)
            gemm_wait();
            // ---------------- epilogue 2: the residual against the dtype-rounded reconstruction
            const float nf = tq_half_bits_to_float(nh) * a.unscale2, scale = fit_power(safe) * a.res_scale;
            const uint64_t nf2 = f32x2(nf, nf), scale2 = f32x2(scale, scale);
            uint64_t rs2 = 0;
#pragma unroll
            for (int q = 0; q < kCoords / 16; ++q) {
                uint32_t y[16], hi[8], lo[8];
                tmem_ld16(my_acc + 16 * q, y);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint64_t rec = round_through2<T>(f32x2_mul(f32x2(__uint_as_float(y[2 * i]), __uint_as_float(y[2 * i + 1])), nf2));
                    const uint64_t res = f32x2_sub(R::pair(raw, 8 * q + i), rec);
                    rs2 = f32x2_fma(res, res, rs2);
                    split_half2(f32x2_mul(res, scale2), hi[i], lo[i]);
                }
                tmem_st8(my_hi + 8 * q, hi), tmem_st8(my_lo + 8 * q, lo);
            }
            float rs, rs_hi;
            f32x2_split(rs2, rs, rs_hi);
            sm.rs[group][part][vrow] = rs + rs_hi;
            // ---------------- stage 3: projection, sign bits
            gemm_issue(1, two_terms, std::false_type());
            float (*rsq)[kUmmaRows] = sm.rs[group];
            const float rn = sqrtf((rsq[0][vrow] + rsq[1][vrow]) + (rsq[2][vrow] + rsq[3][vrow]));
            if (more) request(tile + stride);  // everybody has formed its residual: request the next tile's rows under the MMAs
            gemm_wait();
            uint32_t neg = 0;  // sign bits, shifted in from coordinate 31 down to 0; -0 counts as +0
#pragma unroll
            for (int q = kCoords / 16 - 1; q >= 0; --q) {
                uint32_t p[16];
                tmem_ld16(my_acc + 16 * q, p);
#pragma unroll
                for (int i = 14; i >= 0; i -= 2) {
                    float p0, p1;
                    f32x2_split(f32x2_fma(f32x2(__uint_as_float(p[i]), __uint_as_float(p[i + 1])), f32x2(1.f, 1.f), 0ull), p0, p1);
                    neg = __funnelshift_l(__float_as_uint(p1), neg, 1);
                    neg = __funnelshift_l(__float_as_uint(p0), neg, 1);
                }
            }
            if (my_row >= 0) {  // (an infinite or undefined residual makes every projection undefined: no bit is set)
                reinterpret_cast<uint32_t *>(a.signs + my_row * 16)[part] = rn < INFINITY ? ~neg : 0u;
                if (part == 0) a.rnorms[my_row] = tq_float_to_half_bits(rn > 0.f ? rn : 1.f);
            }
        }
    }
}

template <typename T, int BITS, bool QJL, bool GRID>
__global__ void __launch_bounds__(kThreads, 1) tq_pack_tc_kernel(const __grid_constant__ PackTcArgs a) {
    constexpr int KEY_BITS = QJL ? BITS - 1 : BITS;
    extern __shared__ uint8_t smem_raw[];
    __shared__ PackTcShared sm;
    const uint32_t images = (smem_u32(smem_raw) + 1023u) & ~1023u;  // swizzle atoms need 1024-byte alignment
    const uint32_t staged = images + (QJL ? 2 : 1) * kUmmaImageBytes;
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
        for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&sm.bar_image[i]), 1);
        for (int i = 0; i < kGroups; ++i) {
            mbar_init(smem_u32(&sm.bar_mma[i]), 1);
            for (int q = 0; q < 4; ++q) mbar_init(smem_u32(&sm.bar_rows[i][q]), kUmmaRows);  // (32 threads of four warps)
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        umma_load_image(images, r.image, smem_u32(&sm.bar_image[0]));  // (every CTA has at least one tile)
        if (QJL && keys) umma_load_image(images + kUmmaImageBytes, a.image_s, smem_u32(&sm.bar_image[1]));
    }
    umma_fence_before();
    __syncthreads();
    umma_fence_after();
    {
        const int bits = keys ? KEY_BITS : BITS;
        if (GRID && bits > 2) {
            build_cells(sm.cells, sm.bounds, (1 << bits) - 1, r.grid, QJL && keys ? 4 : 1);
            __syncthreads();
        }
    }
    if (keys) encode<T, KEY_BITS, QJL, GRID>(a, r, sm, images, staged, blockIdx.x, a.key_ctas);
    else encode<T, BITS, false, GRID>(a, r, sm, images, staged, blockIdx.x - a.key_ctas, gridDim.x - a.key_ctas);
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

// A uniform grid over n boundaries with at most one of them in any cell: see Search.  Its cells are formed by the
// operations the kernel uses (fma rounds once on both sides), the clamp to [0, 1] included.
bool tq_fit_grid(const float *bounds, int n, tq_ctx::Grid *g) {
    for (int i = 0; i < n; ++i)
        if (!isfinite(bounds[i]) || (i && !(bounds[i - 1] < bounds[i]))) return false;
    for (int cells = 32; cells <= kMaxCells; cells *= 2) {
        const float width = bounds[n - 1] - bounds[0];
        g->last = (float)(cells - 1);
        g->scale = width > 0.f ? (1.f - 2.f / cells) / width : 1.f;
        g->shift = 1.f / cells - bounds[0] * g->scale;
        if (!isfinite(g->scale) || !isfinite(g->shift)) return false;
        bool single = true;
        float before = -1.f;
        for (int i = 0; i < n && single; ++i) {
            const float t = fminf(fmaxf(fmaf(bounds[i], g->scale, g->shift), 0.f), 1.f), at = fmaf(t, g->last, 8388608.f);
            single = at != before;
            before = at;
        }
        if (single) return true;
    }
    return false;
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

template <typename T, int BITS, bool QJL, bool GRID>
static cudaError_t launch_tc_search(const PackTcArgs &a, int grid, int device, cudaStream_t stream) {
    constexpr int smem = (QJL ? 2 : 1) * kUmmaImageBytes + (sizeof(T) == 2 ? kGroups * kStageBytes : 0) + 1024;
    // the attribute belongs to the (kernel, device) pair: one flag per device of this instantiation
    static bool configured[TQ_MAX_DEVICES] = {};
    if (device < 0 || device >= TQ_MAX_DEVICES) return cudaErrorInvalidDevice;
    if (!configured[device]) {
        cudaError_t e = cudaFuncSetAttribute(tq_pack_tc_kernel<T, BITS, QJL, GRID>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        configured[device] = true;
    }
    tq_pack_tc_kernel<T, BITS, QJL, GRID><<<grid, kThreads, smem, stream>>>(a);
    return cudaGetLastError();
}

template <typename T, int BITS, bool QJL>
static cudaError_t launch_tc(const PackTcArgs &a, int grid, int device, cudaStream_t stream, bool cells) {
    if constexpr (BITS > 2) {
        if (!cells) return launch_tc_search<T, BITS, QJL, false>(a, grid, device, stream);
    }
    return launch_tc_search<T, BITS, QJL, true>(a, grid, device, stream);  // (up to two bits: no search in shared memory at all)
}

int32_t tq_launch_pack_tc(tq_ctx *ctx, const tq_dense_desc *k, const tq_dense_desc *v, int32_t n_tokens,
                          const tq_cache_desc *cache, int32_t pos0, cudaStream_t stream) {
    const int esize = v->dtype == TQ_DTYPE_F32 ? 4 : 2;
    PackTcArgs a = {};
    bool cells = true;  // a grid separates the boundaries
    for (int i = 0; i < 2; ++i) {
        const tq_dense_desc *x = i == 0 ? k : v;
        if (!x) continue;
        if (((uintptr_t)x->data & 15) || ((x->stride_b * esize) & 15) || ((x->stride_h * esize) & 15) || ((x->stride_t * esize) & 15))
            return TQ_ERR_UNSUPPORTED;
        PackTcRole &r = a.role[i];
        const tq_ctx::Image &image = i == 0 ? ctx->img_rot_k : ctx->img_rot_v;
        r.x = x->data, r.sb = x->stride_b, r.sh = x->stride_h, r.st = x->stride_t;
        r.codes = i == 0 ? cache->k_codes : cache->v_codes, r.norms = i == 0 ? cache->k_norms : cache->v_norms;
        r.image = image.data, r.unscale = kUmmaRestore * image.unscale;
        r.bounds = i == 0 ? ctx->bounds_k : ctx->bounds_v;
        r.grid = i == 0 ? ctx->grid_k : ctx->grid_v;
        if ((i == 0 ? ctx->key_bits : ctx->bits) > 2 && r.grid.last == 0.f) cells = false;
    }
    const bool qjl = ctx->use_qjl && k;
    a.vec = vector_index(cache->batch, cache->kv_heads, n_tokens), a.pos0 = pos0;
    a.cache_sb = cache->stride_b, a.cache_sh = cache->stride_h;
    a.error_flag = ctx->error_flag;
    a.image_s = ctx->img_qjl.data;
    a.unscale2 = kUmmaRestore * ctx->img_rot_k.unscale / ctx->cen_k_scale;
    a.cen_scale = ctx->cen_k_scale, a.res_scale = ctx->res_scale;
    a.centers = ctx->centers_k;
    a.signs = cache->k_signs, a.rnorms = cache->k_rnorms;
    a.n_tiles = (int)((a.vec.n + kUmmaRows - 1) / kUmmaRows);
    // One CTA per SM.  With tiles enough for all of them, keys with the sketch get the share of the SMs that
    // their cost asks for, which depends on the type (fp32 rows go straight to registers, which tells most on values) and on
    // what the bits leave to search.  2 x 8 x 32768 vectors a tensor, us at 92, 94, 98 and 103 of 148 SMs: bf16 4 bits 236, 229, 221, 210,
    // 3 bits 230, 223, 215, 229, 2 bits 206, 199, 193, 214; f16 3 bits 225, 219, 209, 200 (4 and 2 bits alike); fp32 4 bits
    // 399, 389, 403, 446, 3 bits 365, 375, 405, 447, 2 bits 330, 340, 364, 401.  The same places are best from 8 x 11000 to
    // 40 x 20011 vectors.  With few tiles each side gets a CTA per tile, and no SM two (8 x 1000 vectors a tensor:
    // 16 us, 31 us in two launches).
    const int sms = ctx->sm_count;
    const int share = v->dtype == TQ_DTYPE_F32 ? (ctx->bits == 4 ? 640 : 625) : v->dtype == TQ_DTYPE_BF16 && ctx->bits < 4 ? 665 : 700;  // of 1000
    int key_ctas = !k ? 0 : qjl ? sms * share / 1000 : sms / 2, val_ctas = sms - key_ctas;
    if (k && a.n_tiles <= sms / 2) key_ctas = val_ctas = a.n_tiles;
    key_ctas = key_ctas < a.n_tiles ? key_ctas : a.n_tiles, val_ctas = val_ctas < a.n_tiles ? val_ctas : a.n_tiles;
    a.key_ctas = key_ctas;
    const int grid = key_ctas + val_ctas;
    cudaError_t e = cudaErrorInvalidValue;
#define TQ_TC_CASE(T)                                                                                                     \
    switch (ctx->bits) {                                                                                                  \
        case 2: e = qjl ? launch_tc<T, 2, true>(a, grid, ctx->device, stream, cells) : launch_tc<T, 2, false>(a, grid, ctx->device, stream, cells); break; \
        case 3: e = qjl ? launch_tc<T, 3, true>(a, grid, ctx->device, stream, cells) : launch_tc<T, 3, false>(a, grid, ctx->device, stream, cells); break; \
        case 4: e = qjl ? launch_tc<T, 4, true>(a, grid, ctx->device, stream, cells) : launch_tc<T, 4, false>(a, grid, ctx->device, stream, cells); break; \
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
