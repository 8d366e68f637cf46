// Helpers of the tcgen05 kernels (prefill encoder, dequantisation): matrix descriptors, TMEM loads and stores, and the f16 operand images of the 128 x 128 matrices.
//
// Every contraction here is [128 vectors x 128] * M with fp32 accuracy on f16 tensor cores: an fp32
// operand, scaled by a power of two so that its largest element is below 2^15, is split in two f16
// terms hi + lo (22 bits, and an absolute floor of 2^-25), and the products hi*lo, lo*hi and hi*hi are
// accumulated in fp32 in that order, so that the accumulator is small until the last eight steps.
// The A operand (the vectors) lives in TMEM, the B operand (the matrix) in shared memory.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

#include "tq_bulk.cuh"
#include "tq_common.cuh"

constexpr int kUmmaRows = 128;                         // vectors per tile: the rows of A and of the accumulator
constexpr int kUmmaSlabBytes = 128 * 128;              // 128 rows x 64 f16 (one 128-byte swizzle row each): 16 KB
constexpr int kUmmaTermBytes = 2 * kUmmaSlabBytes;     // one f16 term of a 128 x 128 matrix: 32 KB
constexpr int kUmmaImageBytes = 2 * kUmmaTermBytes;    // hi and lo terms: 64 KB

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Rows of 16-bit vectors staged in shared memory lie 272 bytes apart: 16-byte accesses of a warp to one
// column of 32 rows touch every bank the same number of times.
constexpr int kStagePitch = 2 * TQ_D + 16;
constexpr int kStageBytes = kUmmaRows * kStagePitch;

// 16 bytes to shared memory without a register in between; `async_arrive` counts on `bar` when this thread's copies are there.
__device__ __forceinline__ void async_copy16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void async_arrive(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];\n" ::"r"(bar) : "memory");
}

// One matrix image to shared memory (one thread; `bar` counts one arrival and the bytes).
__device__ __forceinline__ void umma_load_image(uint32_t dst, const uint16_t *image, uint32_t bar) {
    mbar_expect_tx(bar, kUmmaImageBytes);
#pragma unroll 1
    for (int i = 0; i < 4; ++i)
        tma_load_1d(dst + i * kUmmaSlabBytes, reinterpret_cast<const uint8_t *>(image) + i * kUmmaSlabBytes, kUmmaSlabBytes, bar);
}

// Shared-memory descriptor of an image read as it lies (operand row n = image row, contraction along it: K-major)
// or transposed (contraction over the image rows: N-major): 128-byte swizzle, 8-row groups 1024 bytes apart, and for
// the transposed form the two slabs along N.
template <bool TRANSPOSED> __device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)(TRANSPOSED ? kUmmaSlabBytes >> 4 : 1) << 16) |
           ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor: D = f32, A = B = f16, A K-major, N = 128, M = 128.
template <bool TRANSPOSED> __host__ __device__ constexpr uint32_t umma_instr() {
    return (1u << 4) | (TRANSPOSED ? 1u << 16 : 0u) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
}

// One thread of a converged warp, in a form that lets the compiler keep what the branch needs in uniform registers.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}

// D[128 x 128] (+)= A[128 x 16] (TMEM, two f16 per column) * B (shared memory)
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t instr, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(instr), "r"(accumulate)
        : "memory");
}
// The MMAs of one contraction (one thread): A in `TERMS` f16 terms at a_hi, a_lo, the matrix image at b_addr,
// out[n] = sum_k vec[k] * image[n][k], or image[k][n] when TRANSPOSED.  Of PIECES that are summed up outside the
// tensor core, the first holds the products with a lo term.
template <int TERMS, bool TRANSPOSED, int PIECE = 0, int PIECES = 1>
__device__ __forceinline__ void umma_issue(uint32_t d, uint32_t a_hi, uint32_t a_lo, uint32_t b_addr) {
    const uint64_t desc = umma_desc<TRANSPOSED>(b_addr);
    auto pass = [&](uint32_t a, uint32_t b_offset, uint32_t first, uint32_t from, uint32_t to) {
#pragma unroll
        for (uint32_t s = from; s < to; ++s) {  // (the address field counts 16-byte units and does not overflow)
            const uint32_t step = TRANSPOSED ? s * 16 * 128 : (s >> 2) * kUmmaSlabBytes + (s & 3) * 32;
            umma_f16(d, a + 8 * s, desc + ((b_offset + step) >> 4), umma_instr<TRANSPOSED>(), first | (s > from));
        }
    };
    if (PIECE == 0) {
        pass(a_hi, kUmmaTermBytes, 0, 0, 8);
        if (TERMS == 2) pass(a_lo, 0, 1, 0, 8);
    }
    pass(a_hi, 0, PIECE == 0, 8 * PIECE / PIECES, 8 * (PIECE + 1) / PIECES);
}
// The tensor core's accumulator drops what lies below its last place (rounds towards zero), which leaves a
// result of eight full-size steps 1.5e-7 to 1.7e-7 too small on average (the slope of result against 64 bits,
// 16.8 M results of each codebook; individual errors 1.1e-7 around it).  Results are scaled up by one fp32 ulp.
constexpr float kUmmaRestore = 1.f + 1.1920929e-7f;

__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void umma_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void umma_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// The contractions of a CTA's two groups one after the other (a lock in shared memory, held while a batch is issued): left to
// themselves the MMAs of both alternate, and the group that was first waits for the other's as well.
__device__ __forceinline__ bool turn_take(uint32_t *turn) {
    for (uint32_t i = 0; i < kSpinLimit; ++i)
        if (atomicCAS(turn, 0u, 1u) == 0u) return true;
    return false;
}
__device__ __forceinline__ void turn_give(uint32_t *turn) { atomicExch(turn, 0u); }

// Byte offset of element (row, k) inside one f16 term of an image (two 64-wide slabs, 128-byte swizzle).
__host__ __device__ inline int umma_operand_offset(int row, int k) {
    const int slab = k >> 6, kk = k & 63;
    return slab * kUmmaSlabBytes + (row >> 3) * 1024 + (row & 7) * 128 + (((kk >> 3) ^ (row & 7)) << 4) + (kk & 7) * 2;
}

// 16 consecutive accumulator columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}
// Eight columns (16 f16 of an A operand row) of this thread's TMEM lane; tmem_st_wait before anybody reads them.
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

// Division of numbers below 2^31 by a divisor known to the host: a multiplication, an addition and a shift (Granlund and
// Montgomery, Division by invariant integers using multiplication, 1994).
struct FastDiv {
    uint32_t d, m, s;
};
inline FastDiv fast_div(uint32_t d) {
    FastDiv f = {d, 0, 0};
    while (((uint64_t)1 << f.s) < d) ++f.s;
    f.m = (uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << f.s) - d)) / d + 1);
    return f;
}
__device__ __forceinline__ uint32_t fast_div(uint32_t n, const FastDiv &f) { return (__umulhi(n, f.m) + n) >> f.s; }

// The vectors of a [B][H][S] tensor in that order.
struct VectorIndex {
    int64_t n;  // B * H * S
    int H, S;
    FastDiv by_h, by_s;
};
inline VectorIndex vector_index(int B, int H, int S) { return {(int64_t)B * H * S, H, S, fast_div(H), fast_div(S)}; }
__device__ __forceinline__ void vector_at(const VectorIndex &x, int64_t v, int &b, int &h, int &t) {
    if (x.n <= 0x7fffffff) {
        const uint32_t q = fast_div((uint32_t)v, x.by_s);
        t = (int)((uint32_t)v - q * (uint32_t)x.S), b = (int)fast_div(q, x.by_h), h = (int)(q - (uint32_t)b * (uint32_t)x.H);
    } else {
        t = (int)(v % x.S), h = (int)((v / x.S) % x.H), b = (int)(v / ((int64_t)x.S * x.H));
    }
}

// Two floats at a time (one instruction for both on this architecture).
__device__ __forceinline__ uint64_t f32x2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f32x2_split(uint64_t v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t f32x2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f32x2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t f32x2_sub(uint64_t a, uint64_t b) {  // a - b
    return f32x2_fma(b, f32x2(-1.f, -1.f), a);
}

// Two values as packed f16: rounded (hi) and what is left of them (lo).
__device__ __forceinline__ uint32_t half2_bits(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
// (v is given as a packed pair)
__device__ __forceinline__ void split_half2(uint64_t v, uint32_t &hi, uint32_t &lo) {
    float a, b;
    f32x2_split(v, a, b);
    hi = half2_bits(a, b);
    const float2 h = __half22float2(*reinterpret_cast<const __half2 *>(&hi));
    float ra, rb;
    f32x2_split(f32x2_sub(v, f32x2(h.x, h.y)), ra, rb);
    lo = half2_bits(ra, rb);
}
