// Decode attention over the packed cache, fp32-exact CUDA-core variant, plus the
// pieces every variant shares: query preparation (rotate / project) and the
// split combine (+ dense tail merge + un-rotation).
//
//   logit[n] = (1/sqrt(D)) * ( |k_n| * <q R_k^T, c_k[idx_n]> + sqrt(pi/2)/D * |r_n| * <q S^T, sign_n> )
//   out      = ( sum_n softmax(logit)_n * |v_n| * c_v[idx_n] ) @ R_v
#include <cooperative_groups.h>
#include <math.h>

#include "tq_common.cuh"
#include "tq_decode_shared.cuh"

namespace {

constexpr int kExactWarps = 16;

struct ExactArgs {
    const uint8_t *k_codes;
    const uint16_t *k_norms;
    const uint8_t *k_signs;
    const uint16_t *k_rnorms;
    const uint8_t *v_codes;
    const uint16_t *v_norms;
    int64_t cache_sb, cache_sh;
    int Hkv, G, N, n_splits;
    const int *seq_start;  // per batch entry: first token attended (null: 0)
    const float *qrot;   // [B*Hq][128]
    const float *qproj;  // [B*Hq][128]
    float *part_m, *part_l, *part_acc;
    const float *centers_k, *centers_v;
};

template <int BITS> __device__ __forceinline__ uint32_t code_at(const uint32_t *w, int j) {
    const int o = j * BITS, wi = o >> 5, s = o & 31;
    uint32_t v = w[wi] >> s;
    if (s + BITS > 32) v |= w[wi + 1] << (32 - s);
    return v & ((1u << BITS) - 1u);
}

// One warp attends 32 tokens at a time: first with a token per lane (all logits of its NG heads: a
// centre look-up and NG multiply-adds per coordinate, the queries read as 16-byte broadcasts), then,
// after the softmax, with four value coordinates per lane.  What bounds it is the chain of about 2000
// instructions a warp runs per 32 tokens, so the work of a (split, KV row) is spread over 16 warps -
// a whole 512-token split at once - and the value codes are requested before the logits are formed.
// 1 x 8 x 4096 tokens, 4 heads each: 13 us; 53 us with four warps and value codes fetched token by token.
template <int VB, int NG> struct ExactShared {
    float q[NG][TQ_D];
    float qp[NG][TQ_D];
    float ck[16], cv[16];
    float m[kExactWarps][NG], l[kExactWarps][NG];
    float p[kExactWarps][32][NG];
    union {
        uint4 v[kExactWarps][32 * VB];  // the 32 tokens' value codes
        float acc[kExactWarps][TQ_D];   // merge of the warps, one head at a time
    };
};

template <int KB, int VB, bool QJL, int NG>
__global__ void __launch_bounds__(kExactWarps * 32) tq_decode_exact_kernel(ExactArgs a) {
    extern __shared__ __align__(16) uint8_t s_raw[];
    ExactShared<VB, NG> &sm = *reinterpret_cast<ExactShared<VB, NG> *>(s_raw);
    const int split = blockIdx.x;
    const int bh = blockIdx.y;  // b * Hkv + h
    const int b = bh / a.Hkv, h = bh % a.Hkv;
    const int G = a.G;  // (> NG / 2 or NG == 4; heads >= G of the block attend a zero query)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t q_row0 = ((int64_t)b * a.Hkv + h) * G;  // first query head of this KV head
    if (threadIdx.x < 16) {
        sm.ck[threadIdx.x] = a.centers_k[threadIdx.x];
        sm.cv[threadIdx.x] = a.centers_v[threadIdx.x];
    }
    tq_grid_dependency_wait();
    tq_launch_dependents();
    for (int i = threadIdx.x; i < NG * TQ_D; i += blockDim.x) {
        const bool live = i < G * TQ_D;
        (&sm.q[0][0])[i] = live ? a.qrot[q_row0 * TQ_D + i] : 0.f;
        if (QJL) (&sm.qp[0][0])[i] = live ? a.qproj[q_row0 * TQ_D + i] : 0.f;
    }
    __syncthreads();

    const int chunks = (a.N + 31) / 32;
    const int chunks_per_split = (chunks + a.n_splits - 1) / a.n_splits;
    const int c_begin = split * chunks_per_split;
    const int c_end = min(chunks, c_begin + chunks_per_split);
    const int64_t row0 = (int64_t)b * a.cache_sb + (int64_t)h * a.cache_sh;
    const int t_lo = a.seq_start ? a.seq_start[b] : 0;        // tokens before it are masked (left padding)
    const float hs = 0.08838834764831845f;                    // 1/sqrt(128)
    const float qjl_scale = 1.2533141373155003f / (float)TQ_D;  // sqrt(pi/2)/D

    float m[NG], l[NG], acc[NG][4];
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        m[g] = -INFINITY;
        l[g] = 0.f;
        acc[g][0] = acc[g][1] = acc[g][2] = acc[g][3] = 0.f;
    }

    for (int c = c_begin + warp; c < c_end; c += kExactWarps) {
        const int base = c * 32;
        const int tok = base + lane;
        const bool valid = tok < a.N && tok >= t_lo;
        const int64_t row = row0 + (tok < a.N ? tok : base);
        const int n_here = min(32, a.N - base);
        // ---- phase A: one token per lane, all logits
        uint32_t kw[4 * KB + 1];
        {
            const uint4 *src = (const uint4 *)(a.k_codes + row * (16 * KB));
#pragma unroll
            for (int i = 0; i < KB; ++i) {
                const uint4 t = __ldg(src + i);
                kw[4 * i] = t.x, kw[4 * i + 1] = t.y, kw[4 * i + 2] = t.z, kw[4 * i + 3] = t.w;
            }
            kw[4 * KB] = 0;
        }
        uint4 sw4 = make_uint4(0, 0, 0, 0);
        float rn = 0.f;
        if (QJL) sw4 = __ldg((const uint4 *)(a.k_signs + row * 16)), rn = tq_half_bits_to_float(a.k_rnorms[row]);
        const float kn = tq_half_bits_to_float(a.k_norms[row]), vn = tq_half_bits_to_float(a.v_norms[row]);
        uint4 vw[VB];  // the chunk's value codes are one contiguous piece of the row
#pragma unroll
        for (int i = 0; i < VB; ++i) {
            vw[i] = make_uint4(0, 0, 0, 0);
            if (32 * i + lane < n_here * VB) vw[i] = __ldg((const uint4 *)(a.v_codes + (row0 + base) * (16 * VB)) + 32 * i + lane);
        }
        float dot[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) dot[g] = 0.f;
#pragma unroll
        for (int j = 0; j < TQ_D; j += 4) {
            float cv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) cv[i] = sm.ck[code_at<KB>(kw, j + i)];
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                const float4 q4 = *reinterpret_cast<const float4 *>(&sm.q[g][j]);
                dot[g] = fmaf(cv[0], q4.x, dot[g]), dot[g] = fmaf(cv[1], q4.y, dot[g]);
                dot[g] = fmaf(cv[2], q4.z, dot[g]), dot[g] = fmaf(cv[3], q4.w, dot[g]);
            }
        }
        float logit[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) logit[g] = dot[g] * kn * hs;
        if (QJL) {
            const uint32_t sw[4] = {sw4.x, sw4.y, sw4.z, sw4.w};
            float dq[NG];
#pragma unroll
            for (int g = 0; g < NG; ++g) dq[g] = 0.f;
#pragma unroll
            for (int j = 0; j < TQ_D; j += 4) {
                float sg[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) sg[i] = ((sw[j >> 5] >> ((j + i) & 31)) & 1u) ? 1.0f : -1.0f;
#pragma unroll
                for (int g = 0; g < NG; ++g) {
                    const float4 q4 = *reinterpret_cast<const float4 *>(&sm.qp[g][j]);
                    dq[g] = fmaf(sg[0], q4.x, dq[g]), dq[g] = fmaf(sg[1], q4.y, dq[g]);
                    dq[g] = fmaf(sg[2], q4.z, dq[g]), dq[g] = fmaf(sg[3], q4.w, dq[g]);
                }
            }
#pragma unroll
            for (int g = 0; g < NG; ++g) logit[g] += qjl_scale * rn * dq[g] * hs;
        }
        // ---- phase B: online softmax over the 32 tokens of the chunk
        __syncwarp();
#pragma unroll
        for (int i = 0; i < VB; ++i) sm.v[warp][32 * i + lane] = vw[i];
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const float lg = valid ? logit[g] : -INFINITY;
            const float nm = fmaxf(m[g], tq_warp_max(lg));
            const float corr = (m[g] == -INFINITY) ? 0.f : expf(m[g] - nm);
            const float p = valid ? expf(lg - nm) : 0.f;
            l[g] = l[g] * corr + tq_warp_sum(p);
            acc[g][0] *= corr, acc[g][1] *= corr, acc[g][2] *= corr, acc[g][3] *= corr;
            m[g] = nm;
            sm.p[warp][lane][g] = valid ? p * vn : 0.f;  // (a masked token's norm may be stale and not finite)
        }
        __syncwarp();
        // ---- phase C: lane owns value dims 4*lane..4*lane+3
#pragma unroll 4
        for (int t = 0; t < n_here; ++t) {
            const uint8_t *vr = reinterpret_cast<const uint8_t *>(&sm.v[warp][0]) + t * (16 * VB);
            uint32_t v;
            if (VB == 2) {
                v = vr[lane];
            } else if (VB == 4) {
                v = ((const uint16_t *)vr)[lane];
            } else {  // 3 bits: 12 bits starting at bit 12*lane
                const int by = (3 * lane) >> 1;
                v = ((uint32_t)vr[by] | ((uint32_t)vr[by + 1] << 8)) >> ((lane & 1) * 4);
            }
            float cv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) cv[i] = sm.cv[(v >> (VB * i)) & ((1u << VB) - 1u)];
#pragma unroll
            for (int g = 0; g < NG; g += 4) {
                const float4 w = *reinterpret_cast<const float4 *>(&sm.p[warp][t][g]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    acc[g][i] = fmaf(w.x, cv[i], acc[g][i]), acc[g + 1][i] = fmaf(w.y, cv[i], acc[g + 1][i]);
                    acc[g + 2][i] = fmaf(w.z, cv[i], acc[g + 2][i]), acc[g + 3][i] = fmaf(w.w, cv[i], acc[g + 3][i]);
                }
            }
        }
        __syncwarp();
    }

    // ---- merge the warps of this CTA, one head at a time, and write the split partial
#pragma unroll
    for (int g = 0; g < NG; ++g)
        if (lane == 0) sm.m[warp][g] = m[g], sm.l[warp][g] = l[g];
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        if (g >= G) break;
        __syncthreads();  // (the value codes, then the previous head's accumulators, are done with)
        *reinterpret_cast<float4 *>(&sm.acc[warp][4 * lane]) = make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
        __syncthreads();
        const int d = threadIdx.x;
        if (d < TQ_D) {
            float M = -INFINITY;
            for (int w = 0; w < kExactWarps; ++w) M = fmaxf(M, sm.m[w][g]);
            float L = 0.f, A = 0.f;
            for (int w = 0; w < kExactWarps; ++w) {
                const float sc = (sm.m[w][g] == -INFINITY) ? 0.f : expf(sm.m[w][g] - M);
                L += sm.l[w][g] * sc;
                A += sm.acc[w][d] * sc;
            }
            const int64_t prow = (q_row0 + g) * a.n_splits + split;
            a.part_acc[prow * TQ_D + d] = A;
            if (d == 0) a.part_m[prow] = M, a.part_l[prow] = L;
        }
    }
}

template <int KB, int VB, bool QJL, int NG>
cudaError_t launch_exact_variant(const ExactArgs &a, int device, dim3 grid, cudaStream_t stream) {
    const size_t smem = sizeof(ExactShared<VB, NG>);
    // the attribute belongs to the (kernel, device) pair: one flag per device of this instantiation
    static bool configured[TQ_MAX_DEVICES] = {};
    if (device < 0 || device >= TQ_MAX_DEVICES) return cudaErrorInvalidDevice;
    if (!configured[device]) {
        cudaError_t e = cudaFuncSetAttribute(tq_decode_exact_kernel<KB, VB, QJL, NG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        configured[device] = true;
    }
    return tq_launch_kernel(tq_decode_exact_kernel<KB, VB, QJL, NG>, grid, dim3(kExactWarps * 32), smem, stream, true, a);
}
template <int KB, int VB, bool QJL> cudaError_t launch_exact(const ExactArgs &a, int device, dim3 grid, cudaStream_t stream) {
    return a.G > 4 ? launch_exact_variant<KB, VB, QJL, 8>(a, device, grid, stream)
                   : launch_exact_variant<KB, VB, QJL, 4>(a, device, grid, stream);
}

}  // namespace

// ---------------------------------------------------------------------------
// Shared pieces: query preparation and split combine
// ---------------------------------------------------------------------------

// Rotated (first half of the grid) and projected (second half, with a QJL sketch) queries as plain
// rows, four rows per block: a thread's 32 matrix elements come in one batch of loads.  One row per
// block and a chain of loads over the 128 matrix rows took 4.8 us for 32 rows, this takes 2.4.
template <typename T>
__global__ void __launch_bounds__(4 * TQ_D, 2) tq_qprep_kernel(const T *q, const float *rot_k_t, const float *qjl_t,
                                                              float *qrot, float *qproj, int64_t rows) {
    __shared__ float s_q[4][TQ_D], s_part[4][4][TQ_D];
    const int64_t groups = (rows + 3) / 4;
    const bool proj = blockIdx.x >= groups;
    const int64_t row0 = 4 * (proj ? blockIdx.x - groups : blockIdx.x);
    const int tid = threadIdx.x, j = tid & (TQ_D - 1), dq = tid >> 7;
    float m[32];
    tq_load_column(m, proj ? qjl_t : rot_k_t, dq, j);  // (codec constants: fetched before the wait)
    tq_grid_dependency_wait();
    tq_launch_dependents();
    s_q[dq][j] = row0 + dq < rows ? tq_to_float<T>(q[(row0 + dq) * TQ_D + j]) : 0.f;
    __syncthreads();
    float r[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 32; ++i)
#pragma unroll
        for (int g = 0; g < 4; ++g) r[g] = fmaf(s_q[g][32 * dq + i], m[i], r[g]);
#pragma unroll
    for (int g = 0; g < 4; ++g) s_part[dq][g][j] = r[g];
    __syncthreads();
    if (row0 + dq < rows)
        (proj ? qproj : qrot)[(row0 + dq) * TQ_D + j] =
            (s_part[0][dq][j] + s_part[1][dq][j]) + (s_part[2][dq][j] + s_part[3][dq][j]);
}

// Query preparation for the tensor-core kernel (see tq_qprep_block): kv_rows * ceil(G / 4) blocks
// rotate, another kv_rows blocks project when the keys carry a QJL sketch.  Launched as a
// programmatic dependent of whatever precedes it in the stream: a block fetches its matrix
// column, waits for that kernel, then lets the decode kernel begin its own set-up.
template <typename T>
__global__ void __launch_bounds__(4 * TQ_D, 2) tq_qprep_frag_kernel(TqQprepArgs a) {
    tq_qprep_block<T>(a, blockIdx.x);
}

// The whole latency-bound front of a decode step in one launch: query preparation blocks
// first, then one block per new key and value vector to append (tq_pack_small_block).
template <typename T, bool QJL, bool STAGED>
__global__ void __launch_bounds__(4 * TQ_D, STAGED ? 1 : 2) tq_step_prologue_kernel(TqQprepArgs qa, TqPackArgs pa, int n_qprep) {
    if ((int)blockIdx.x < n_qprep)
        tq_qprep_block<T>(qa, blockIdx.x);
    else
        tq_pack_small_block<T, QJL, STAGED, true>(pa, (int64_t)blockIdx.x - n_qprep);
}

// Publishing rows to the peers and waiting for theirs (system scope, PTX memory model):
// a block's threads store their rows with plain stores, the block barrier orders those stores
// before thread 0, which adds the block's row count to the flag word with a RELEASE reduction at
// system scope (cumulative over what the barrier ordered before it); the waiting side polls the
// word with ACQUIRE loads at system scope, and its own block barrier orders the data reads of
// the other threads behind the observation.  No separate fence on either side: on a B200 pair
// the two full system fences this replaces cost 3.3 us of a 92 us step.
__device__ __forceinline__ void tq_release_add_sys(unsigned *word, unsigned value) {
    asm volatile("red.release.sys.global.add.u32 [%0], %1;\n" ::"l"(word), "r"(value) : "memory");
}
__device__ __forceinline__ unsigned tq_acquire_load_sys(const unsigned *word) {
    unsigned v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];\n" : "=r"(v) : "l"(word) : "memory");
    return v;
}

// Eight consecutive elements as floats: one (16-bit types) or two (fp32) 16-byte loads when the
// tensor is 16-byte aligned (`vec`, uniform over the launch), else element by element.
template <typename T> __device__ __forceinline__ void tq_load8(const T *p, bool vec, float (&v)[8]) {
    if (vec) {
        uint4 raw[sizeof(T) / 2];
#pragma unroll
        for (int i = 0; i < (int)sizeof(T) / 2; ++i) raw[i] = __ldg(reinterpret_cast<const uint4 *>(p) + i);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = tq_to_float<T>(reinterpret_cast<const T *>(raw)[i]);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = tq_to_float<T>(p[i]);
    }
}

// Attention of up to four heads of one KV row over the row's un-quantised tail tokens, by the 512
// threads of a combine block, 256 tokens at a time with an online softmax.  Logits: eight lanes
// share a token, so a warp reads four whole rows per load and sums each over three shuffles;
// values: sixteen threads cover a row with 16-byte loads and 32 rows are read side by side.
// Returns this thread's element (head threadIdx.x / 128, column threadIdx.x % 128) of the
// unnormalised sum; the maximum and the sum of every head are left in s_tm / s_tl.
// What bounds it is the latency of two dependent trips to memory per 256 tokens; where SMs are free for it, the
// row's tail is shared out over the CTAs of a cluster (tq_merge_tails, tq_set_combine_tail).
constexpr int kTailChunk = 256;
constexpr int kTailCtas = 4;         // CTAs of a cluster, at most
constexpr int kRowTailTokens = 256;  // tail tokens that tq_combine_row_kernel takes, at most
struct TailShared {
    float p[4][kTailChunk];
    float corr[4], m[4], l[4];
    float acc[16][4][TQ_D];
};
template <typename T>
__device__ __forceinline__ float tq_attend_tail(const CombineArgs &a, TailShared &sm, int64_t R, int h0, int n_heads, int t_begin, int t_end) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t row0 = R * a.G + h0;
    const int b = (int)(row0 / a.Hq), hkv = (int)(row0 % a.Hq) / a.G;
    const T *tk = (const T *)a.tail_k + b * a.tk_sb + hkv * a.tk_sh;
    const T *tv = (const T *)a.tail_v + b * a.tv_sb + hkv * a.tv_sh;
    const float hs = 0.08838834764831845f;
    const int sub = lane & 7, tg = tid >> 4, dc = 8 * (tid & 15);
    float acc[4][8];
#pragma unroll
    for (int g = 0; g < 4; ++g)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[g][i] = 0.f;
    float q[4][16];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        const T *qr = (const T *)a.q + (row0 + (g < n_heads ? g : 0)) * TQ_D + 16 * sub;  // (q is 16-byte aligned)
        float lo[8], hi[8];
        tq_load8<T>(qr, true, lo), tq_load8<T>(qr + 8, true, hi);
#pragma unroll
        for (int i = 0; i < 8; ++i) q[g][i] = lo[i], q[g][8 + i] = hi[i];
    }
    float m_run = -INFINITY, l_run = 0.f;  // warp g < 4: head g
    for (int c0 = t_begin; c0 < t_end; c0 += kTailChunk) {
        const int n = min(kTailChunk, t_end - c0);
#pragma unroll
        for (int it = 0; it < kTailChunk / 64; ++it) {
            const int t = 64 * it + 4 * warp + (lane >> 3);
            float d[4] = {0.f, 0.f, 0.f, 0.f};
            if (t < n) {
                const T *kr = tk + (int64_t)(c0 + t) * a.tk_st + 16 * sub;
                float lo[8], hi[8];
                tq_load8<T>(kr, a.tail_vec, lo), tq_load8<T>(kr + 8, a.tail_vec, hi);
#pragma unroll
                for (int g = 0; g < 4; ++g)
#pragma unroll
                    for (int i = 0; i < 8; ++i) d[g] = fmaf(q[g][i], lo[i], d[g]), d[g] = fmaf(q[g][8 + i], hi[i], d[g]);
            }
#pragma unroll
            for (int g = 0; g < 4; ++g) {
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) d[g] += __shfl_xor_sync(0xffffffffu, d[g], o);
                if (sub == 0) sm.p[g][t] = t < n ? d[g] * hs : -INFINITY;
            }
        }
        __syncthreads();
        if (warp < 4) {
            float x[kTailChunk / 32], mx = -INFINITY, sum = 0.f;
#pragma unroll
            for (int i = 0; i < kTailChunk / 32; ++i) x[i] = sm.p[warp][32 * i + lane], mx = fmaxf(mx, x[i]);
            const float nm = fmaxf(m_run, tq_warp_max(mx));
            const float base = nm == -INFINITY ? 0.f : nm;  // (every logit so far is -inf: weights of 0, not undefined ones)
            const float corr = expf(m_run - base);
#pragma unroll
            for (int i = 0; i < kTailChunk / 32; ++i) {
                const float p = expf(x[i] - base);
                sm.p[warp][32 * i + lane] = p, sum += p;
            }
            l_run = l_run * corr + tq_warp_sum(sum), m_run = nm;
            if (lane == 0) sm.corr[warp] = corr;
        }
        __syncthreads();
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const float corr = sm.corr[g];
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[g][i] *= corr;
        }
#pragma unroll 4
        for (int t = tg; t < n; t += 32) {
            float v[8];
            tq_load8<T>(tv + (int64_t)(c0 + t) * a.tv_st + dc, a.tail_vec, v);
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const float p = sm.p[g][t];
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[g][i] = fmaf(p, v[i], acc[g][i]);
            }
        }
        __syncthreads();  // the weights are free for the next chunk
    }
#pragma unroll
    for (int g = 0; g < 4; ++g)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[g][i] += __shfl_xor_sync(0xffffffffu, acc[g][i], 16);
    if (lane < 16) {
#pragma unroll
        for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int i = 0; i < 8; i += 4)
                *reinterpret_cast<float4 *>(&sm.acc[warp][g][dc + i]) = make_float4(acc[g][i], acc[g][i + 1], acc[g][i + 2], acc[g][i + 3]);
    }
    if (warp < 4 && lane == 0) sm.m[warp] = m_run, sm.l[warp] = l_run;
    __syncthreads();
    float o = 0.f;
#pragma unroll
    for (int w = 0; w < 16; ++w) o += sm.acc[w][tid >> 7][tid & (TQ_D - 1)];
    return o;
}

// The tails of a cluster's CTAs (each attended its share of the row's tail tokens) merged in its first CTA;
// returns false in the others, which have nothing left to do.  `o` is the caller's element of its own share.
__device__ __forceinline__ bool tq_merge_tails(TailShared &sm, float &o, float &m, float &l) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, g = tid >> 7, n = (int)cluster.num_blocks();
    m = sm.m[g], l = sm.l[g];
    if (n == 1) return true;
    (&sm.acc[0][0][0])[tid] = o;  // (a thread reads the sum of its own element alone, so nobody else's is overwritten early)
    cluster.sync();
    if (cluster.block_rank() == 0) {
        for (int r = 1; r < n; ++r) {
            const TailShared &peer = *cluster.map_shared_rank(&sm, r);
            const float pm = peer.m[g], pl = peer.l[g], po = (&peer.acc[0][0][0])[tid];
            const float M = fmaxf(m, pm), w = m == -INFINITY ? 0.f : expf(m - M), pw = pm == -INFINITY ? 0.f : expf(pm - M);
            o = o * w + po * pw, l = l * w + pl * pw, m = M;
        }
    }
    cluster.sync();
    return cluster.block_rank() == 0;
}

// Split combine for up to four heads of one (batch, KV head) row per block: the un-rotation
// matrix is read once for the G heads.  An un-quantised tail of the row, if there is one (TAIL), is
// attended by a cluster of CTAs before the splits are waited for: the decode kernel
// releases this one as soon as the query and the tail are known to be there, so the tail is attended on
// SMs that the decode kernel leaves free.  12001 packed + 300 dense tokens, 8 KV rows, launches recorded: 17.0 us
// from query preparation to output; 28.2 us with one block per four heads that began after the decode kernel.
template <typename T, bool TAIL>
__global__ void __launch_bounds__(4 * TQ_D) tq_combine_group_kernel(CombineArgs a) {
    __shared__ __align__(16) float s_o[4][TQ_D];
    __shared__ float s_part[4][4][TQ_D];  // [quarter of d][head][column]
    __shared__ float s_L[4], s_M[4];
    const int groups = (a.G + 3) >> 2;           // a block (TAIL: a cluster) serves up to four heads of a KV row
    const unsigned blk = TAIL ? blockIdx.x / (unsigned)a.tail_ctas : blockIdx.x;
    const int64_t R = blk / groups;
    const int h0 = 4 * (blk % groups);
    const int n_heads = a.G - h0 < 4 ? a.G - h0 : 4;
    const int tid = threadIdx.x, e = tid & (TQ_D - 1), dq = tid >> 7, lane = tid & 31;
    float tail_o = 0.f, tail_m = -INFINITY, tail_l = 0.f;  // of head dq, column e
    if (TAIL) {
        extern __shared__ __align__(16) uint8_t s_dyn[];
        TailShared &ts = *reinterpret_cast<TailShared *>(s_dyn);
        // (no wait here: the kernel before this one releases it after its own dependency wait, when everything
        // ordered before the query preparation - the query and the tail among it - has completed)
        const int rank = (int)(blockIdx.x % (unsigned)a.tail_ctas), t0 = rank * a.tail_per_cta;
        tail_o = tq_attend_tail<T>(a, ts, R, h0, n_heads, t0, min(a.n_tail, t0 + a.tail_per_cta));
        if (!tq_merge_tails(ts, tail_o, tail_m, tail_l)) return;
    }
    float rv[32];  // this thread's un-rotation elements, fetched while the decode kernel drains
    tq_load_column(rv, a.rot_v, dq, e);
    // (the length was there before the query preparation began, and the decode kernel has planned with it)
    int n_valid = a.n_splits;
    TqPlan plan = {a.seg_npad, a.seg_chunk};
    if (a.len_ptr) plan = tq_make_plan(min(*a.len_ptr + a.len_add, a.capacity), a.plan_rows, a.plan_ctas, a.n_splits, a.plan_step);
    if (plan.chunk > 0) {
        const int64_t lo = R * (int64_t)plan.n_pad, hi = lo + plan.n_pad - 1;
        n_valid = 1 + (hi <= 0x7fffffff ? (int)((unsigned)hi / (unsigned)plan.chunk - (unsigned)lo / (unsigned)plan.chunk)
                                        : (int)(hi / plan.chunk - lo / plan.chunk));
        if (!TAIL && a.next_blocks && tq_leaves_idle(plan, a.plan_rows, a.sm_count, a.next_blocks)) tq_launch_dependents();
    }
    tq_grid_dependency_wait();
    {   // thread (e, dq) merges the splits of head dq.  Up to four, the usual number with many rows: everything is
        // requested in one batch and merged in registers (sixty pairs of runs each: 0.65 +- 0.08 us less than the other way for
        // 8 x 8 x 32768 tokens, 0.45 to 0.6 +- 0.02 for six smaller caches, 1.5 for 64 x 8 x 500 of one head).  More: 32 at a
        // time, lane s of each warp holds split s's maximum and weight, and all accumulator columns are requested before
        // the first is used: one trip to L2, where eight at a time took one for every eight (eight layer steps of nine splits
        // 98.5 -> 96.6 us, 32768 tokens of seven heads in 33 splits 17.45 -> 17.2, of four heads 19.1 -> 18.9).  (With one
        // thread walking all splits twice the kernel took twice as long, with maxima, sums and columns of eight splits in every
        // thread 1.1 us more.)
        const int g = dq;
        float o = 0.f, L = 0.f, Mx = -INFINITY;
        if (g < n_heads) {
            const int64_t slot0 = (R * a.G + h0 + g) * a.n_splits;
            if (n_valid <= 4) {
                float pm[4], pl[4], pa[4];
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const bool on = s < n_valid;
                    pm[s] = on ? a.part_m[slot0 + s] : -INFINITY, pl[s] = on ? a.part_l[slot0 + s] : 0.f;
                    pa[s] = on ? a.part_acc[(slot0 + s) * TQ_D + e] : 0.f;
                }
                Mx = fmaxf(fmaxf(pm[0], pm[1]), fmaxf(pm[2], pm[3]));
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const float w = pm[s] == -INFINITY ? 0.f : expf(pm[s] - Mx);
                    L += pl[s] * w, o += pa[s] * w;
                }
            } else for (int s0 = 0; s0 < n_valid; s0 += 32) {
                const int n = min(32, n_valid - s0);
                const float *acc = a.part_acc + (slot0 + s0) * TQ_D + e;
                float pa[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) pa[i] = i < n ? acc[i * TQ_D] : 0.f;
                const float pm = lane < n ? a.part_m[slot0 + s0 + lane] : -INFINITY;
                const float pl = lane < n ? a.part_l[slot0 + s0 + lane] : 0.f;
                const float M = fmaxf(Mx, tq_warp_max(pm));
                const float corr = Mx == -INFINITY ? 0.f : expf(Mx - M);
                const float w = pm == -INFINITY ? 0.f : expf(pm - M);
                L = L * corr + tq_warp_sum(pl * w), o *= corr, Mx = M;
#pragma unroll
                for (int i0 = 0; i0 < 32; i0 += 8) {
                    if (i0 < n) {
#pragma unroll
                        for (int i = i0; i < i0 + 8; ++i) o = fmaf(pa[i], __shfl_sync(0xffffffffu, w, i), o);
                    }
                }
            }
        }
        s_o[g][e] = o;
        if (e == 0) s_L[g] = L, s_M[g] = Mx;
        if (a.parts > 0 && g < n_heads) {
            // Sequence split: this rank holds only a part of the row's tokens.  Its merged partial goes,
            // unfinished, into slot `part` of every rank's exchange buffer [row][parts] (laid out like a
            // decode workspace: all maxima, then all sums, then the accumulators); whoever has waited for
            // all parts finishes the rows with this same kernel (n_splits = parts).
            const int64_t row0 = R * a.G + h0;
            const int64_t bi = row0 / a.Hq, hl = row0 % a.Hq;
            const int64_t grow = bi * a.gather_heads_total + (int64_t)a.head_group * a.Hq + hl + g;  // row of the whole model
            const unsigned seq = a.gather_seq;
            for (int p = 0; p < a.gather_world; ++p) {
                float *base = reinterpret_cast<float *>(static_cast<char *>(a.gather_out[p]) + ((seq & 1u) ? a.gather_out_stride : 0));
                const int64_t n_rows = a.exch_rows;
                float *xm = base, *xl = base + n_rows * a.parts, *xacc = base + 2 * n_rows * a.parts;
                const int64_t slot = grow * a.parts + a.part;
                xacc[slot * TQ_D + e] = o;
                if (e == 0) xm[slot] = Mx, xl[slot] = L;
            }
        }
    }
    if (a.parts > 0) {  // report the rows (see the gather below) and leave: nothing is finished here
        __syncthreads();
        // (lane p of the first warp reports to rank p: one instruction, so one wait for the stores)
        if (tid < a.gather_world) tq_release_add_sys(a.gather_flags[tid] + a.gather_rank, (unsigned)n_heads);
        return;
    }
    __syncthreads();
    {   // thread (e, dq) un-rotates rows d in [32 dq, 32 dq + 32) for all heads
        float out[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const float4 o = *reinterpret_cast<const float4 *>(&s_o[g][32 * dq + i]);
                out[g] = fmaf(o.x, rv[i], out[g]), out[g] = fmaf(o.y, rv[i + 1], out[g]);
                out[g] = fmaf(o.z, rv[i + 2], out[g]), out[g] = fmaf(o.w, rv[i + 3], out[g]);
            }
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) s_part[dq][g][e] = out[g];
    }
    __syncthreads();
    if (dq < n_heads) {
        const int g = dq;
        float v = (s_part[0][g][e] + s_part[1][g][e]) + (s_part[2][g][e] + s_part[3][g][e]);
        float L = s_L[g];
        if (TAIL) {  // (when packed tokens and tail both have logits of -inf alone, the result is undefined, as a softmax is)
            const float M = fmaxf(s_M[g], tail_m), wt = expf(tail_m - M);
            const float wp = s_M[g] == -INFINITY ? 0.f : expf(s_M[g] - M);
            v = v * wp + tail_o * wt, L = L * wp + tail_l * wt;
        }
        const T res = tq_from_float<T>(v / fmaxf(L, 1e-8f));
        const int64_t row = R * a.G + h0 + g;  // = batch index * local query heads + local head
        if (a.gather_world > 0) {
            reinterpret_cast<T *>(&s_o[0][0])[g * TQ_D + e] = res;  // staged: the peers get 16-byte stores below
        } else if (a.out_f32) {
            a.out_f32[row * TQ_D + e] = v / fmaxf(L, 1e-8f);
        } else {
            ((T *)a.out)[row * TQ_D + e] = res;
        }
    }
    if (a.gather_world > 0) {
        static_assert(sizeof(T) == 2 || sizeof(T) == 4, "");
        __syncthreads();
        // The block's heads are consecutive rows of one batch entry: one contiguous piece of every
        // rank's gathered buffer.  Thread (p, i) stores 16-byte piece i of it into rank p's buffer.
        const unsigned seq = a.gather_seq_ptr ? *a.gather_seq_ptr + 1u : a.gather_seq;
        const long long buf = (seq & 1u) ? a.gather_out_stride : 0;
        const int64_t row0 = R * a.G + h0;  // = batch index * local query heads + local head
        const int64_t bi = row0 / a.Hq, hl = row0 % a.Hq;
        const int64_t dst0 = (bi * a.gather_heads_total + (int64_t)a.gather_rank * a.Hq + hl) * TQ_D;  // elements
        const int pieces = n_heads * TQ_D * (int)sizeof(T) / 16;
        for (int w = tid; w < a.gather_world * pieces; w += blockDim.x) {
            const int p = w / pieces, i = w % pieces;
            uint4 *dst = reinterpret_cast<uint4 *>(static_cast<char *>(a.gather_out[p]) + buf + dst0 * sizeof(T));
            dst[i] = reinterpret_cast<const uint4 *>(&s_o[0][0])[i];
        }
        // Every block reports its own rows: after a system-scope fence (cumulative over the block's
        // stores, which the barrier ordered before it) it adds its row count to this rank's word in
        // every peer's flag block.  A peer has all of this rank's rows of step s once that word has
        // reached s * (rows per step); no block waits for another, no counter round trip.
        __syncthreads();
        // (lane p of the first warp reports to rank p: the release reductions of all peers are one
        // instruction and wait for the block's stores once; one after the other they cost one such
        // wait per peer)
        if (tid < a.gather_world) tq_release_add_sys(a.gather_flags[tid] + a.gather_rank, (unsigned)n_heads);
    }
}

// The combine of one query row per block of 128 threads, with a dense tail: what many rows with few tail tokens take (see
// tq_set_combine_tail).  Sixteen of its blocks fit an SM, so that hundreds of rows are one wave where the blocks of
// tq_combine_group_kernel, one to an SM, are several.  What bounds it is one trip to memory per four tail tokens.
template <typename T>
__global__ void __launch_bounds__(TQ_D) tq_combine_row_kernel(CombineArgs a) {
    __shared__ float s_logit[kRowTailTokens];
    __shared__ float s_o[TQ_D], s_q[TQ_D], s_red[4];
    const int64_t row = blockIdx.x;  // b * Hq + hq
    const int e = threadIdx.x, warp = e >> 5, lane = e & 31;
    const int b = (int)(row / a.Hq), hkv = (int)(row % a.Hq) / a.G;
    const float hs = 0.08838834764831845f;
    int n_valid = a.n_splits;
    if (a.seg_chunk > 0) {
        const int64_t lo = (row / a.G) * (int64_t)a.seg_npad;
        n_valid = (int)((lo + a.seg_npad - 1) / a.seg_chunk - lo / a.seg_chunk) + 1;
    }
    float M = -INFINITY;
    for (int s = 0; s < n_valid; ++s) M = fmaxf(M, a.part_m[row * a.n_splits + s]);
    const T *tk = (const T *)a.tail_k + b * a.tk_sb + hkv * a.tk_sh;
    const T *tv = (const T *)a.tail_v + b * a.tv_sb + hkv * a.tv_sh;
    s_q[e] = tq_to_float<T>(((const T *)a.q)[row * TQ_D + e]);
    __syncthreads();
    float wmax = -INFINITY;
    for (int t = warp; t < a.n_tail; t += 4) {
        const T *kr = tk + (int64_t)t * a.tk_st + 4 * lane;
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) dot = fmaf(s_q[4 * lane + i], tq_to_float<T>(kr[i]), dot);
        dot = tq_warp_sum(dot) * hs;
        if (lane == 0) s_logit[t] = dot;
        wmax = fmaxf(wmax, dot);
    }
    if (lane == 0) s_red[warp] = wmax;
    __syncthreads();
    M = fmaxf(M, fmaxf(fmaxf(s_red[0], s_red[1]), fmaxf(s_red[2], s_red[3])));
    float L = 0.f, o = 0.f;
    for (int s = 0; s < n_valid; ++s) {
        const float ms = a.part_m[row * a.n_splits + s];
        const float w = ms == -INFINITY ? 0.f : expf(ms - M);
        L += a.part_l[row * a.n_splits + s] * w;
        o += a.part_acc[(row * a.n_splits + s) * TQ_D + e] * w;
    }
    s_o[e] = o;
    __syncthreads();
    float out = 0.f;
#pragma unroll 8
    for (int d = 0; d < TQ_D; ++d) out = fmaf(s_o[d], __ldg(a.rot_v + d * TQ_D + e), out);
    for (int t = 0; t < a.n_tail; ++t) {
        const float p = expf(s_logit[t] - M);
        L += p;
        out = fmaf(p, tq_to_float<T>(tv[(int64_t)t * a.tv_st + e]), out);
    }
    ((T *)a.out)[row * TQ_D + e] = tq_from_float<T>(out / fmaxf(L, 1e-8f));
}

__device__ __forceinline__ unsigned long long tq_global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
    return t;
}

// Waits until every rank's word of this rank's flag block has reached step * rows_per_step (the
// peers' combine kernels add the rows they have stored), for at most `limit_ns` nanoseconds of the
// GPU's wall clock; a wait that runs out sets the status word to 5 and the kernel returns without
// copying.  Otherwise, optionally, every block copies its slice of this rank's gathered buffer of
// the step to `dst`.  A step numbered on the device (seq_ptr: the number of the last completed
// step) is number *seq_ptr + 1; the last block to finish stores it back, after every block has
// read it.
__global__ void tq_gather_wait_kernel(const unsigned *flags, int world, unsigned seq_arg, unsigned *seq_ptr,
                                      unsigned rows_per_step, unsigned *counter, int *error_flag,
                                      unsigned long long limit_ns, const uint4 *src0, long long stride, uint4 *dst,
                                      size_t n16, size_t row_len16, size_t row_stride16, size_t src_off16) {
    // (the combine kernel of a device-numbered step reads the same word: it must be complete
    // before this kernel may advance it; a host-numbered step may start polling early)
    if (seq_ptr) tq_grid_dependency_wait();
    tq_launch_dependents();  // the next kernel of the stream may be placed while this one polls
    const unsigned seq = seq_ptr ? *seq_ptr + 1u : seq_arg;
    const unsigned target = seq * rows_per_step;
    __shared__ int s_failed;
    if (threadIdx.x == 0) s_failed = 0;
    __syncthreads();
    if ((int)threadIdx.x < world) {
        const unsigned long long t0 = tq_global_ns();
        unsigned polls = 0;
        while ((int)(tq_acquire_load_sys(flags + threadIdx.x) - target) < 0) {  // (the words only grow; a peer may already be a step ahead)
            if ((++polls & 63u) == 0 && tq_global_ns() - t0 > limit_ns) {
                atomicExch(error_flag, 5);
                s_failed = 1;
                break;
            }
        }
    }
    __syncthreads();
    if (dst && !s_failed) {
        // dst is dense; piece i of it is piece (i % row_len16) of source row (i / row_len16), rows being
        // row_stride16 apart and starting src_off16 into the buffer (a whole-buffer copy is one row)
        const uint4 *src = reinterpret_cast<const uint4 *>(reinterpret_cast<const char *>(src0) + ((seq & 1u) ? stride : 0));
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += (size_t)gridDim.x * blockDim.x)
            dst[i] = src[(i / row_len16) * row_stride16 + src_off16 + i % row_len16];
    }
    if (seq_ptr && !s_failed) {
        __syncthreads();
        if (threadIdx.x == 0 && atomicAdd(counter, 1u) == gridDim.x - 1) {
            *counter = 0;
            *seq_ptr = seq;
        }
    }
    // (a host-numbered wait began before the combine kernel was done: it ends only after it)
    if (!seq_ptr) tq_grid_dependency_wait();
}

// The decode kernels run with the largest shared-memory carve-out.  The small kernels around
// them ask for the same carve-out, so the SMs are not reconfigured (and drained) between the
// launches of one decode step.
template <typename K> static void prefer_max_shared(K kernel) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}
static void configure_small_kernels() {
    static bool done = false;
    if (done) return;
    done = true;
    prefer_max_shared(tq_qprep_kernel<float>);
    prefer_max_shared(tq_qprep_kernel<__half>);
    prefer_max_shared(tq_qprep_kernel<__nv_bfloat16>);
    prefer_max_shared(tq_qprep_frag_kernel<__half>);
    prefer_max_shared(tq_qprep_frag_kernel<__nv_bfloat16>);
    prefer_max_shared(tq_combine_group_kernel<float, false>);
    prefer_max_shared(tq_combine_group_kernel<__half, false>);
    prefer_max_shared(tq_combine_group_kernel<__nv_bfloat16, false>);
    prefer_max_shared(tq_combine_row_kernel<float>);
    prefer_max_shared(tq_combine_row_kernel<__half>);
    prefer_max_shared(tq_combine_row_kernel<__nv_bfloat16>);
    prefer_max_shared(tq_combine_group_kernel<float, true>);
    prefer_max_shared(tq_combine_group_kernel<__half, true>);
    prefer_max_shared(tq_combine_group_kernel<__nv_bfloat16, true>);
    prefer_max_shared(tq_step_prologue_kernel<__half, true, true>);
    prefer_max_shared(tq_step_prologue_kernel<__half, true, false>);
    prefer_max_shared(tq_step_prologue_kernel<__half, false, false>);
    prefer_max_shared(tq_step_prologue_kernel<__nv_bfloat16, true, true>);
    prefer_max_shared(tq_step_prologue_kernel<__nv_bfloat16, true, false>);
    prefer_max_shared(tq_step_prologue_kernel<__nv_bfloat16, false, false>);
}

template <typename T>
static cudaError_t launch_qprep(tq_ctx *ctx, const void *q, int64_t rows, float *qrot, float *qproj, cudaStream_t stream) {
    const unsigned grid = (unsigned)((rows + 3) / 4) * (ctx->use_qjl ? 2 : 1);
    return tq_launch_kernel(tq_qprep_kernel<T>, dim3(grid), dim3(4 * TQ_D), 0, stream, true, (const T *)q, ctx->rot_k_t,
                            ctx->qjl_t, qrot, qproj, rows);
}

int32_t tq_launch_qprep(tq_ctx *ctx, const void *q, int32_t q_dtype, int64_t rows, float *qrot, float *qproj,
                        cudaStream_t stream) {
    configure_small_kernels();
    cudaError_t e;
    if (q_dtype == TQ_DTYPE_F32) e = launch_qprep<float>(ctx, q, rows, qrot, qproj, stream);
    else if (q_dtype == TQ_DTYPE_F16) e = launch_qprep<__half>(ctx, q, rows, qrot, qproj, stream);
    else e = launch_qprep<__nv_bfloat16>(ctx, q, rows, qrot, qproj, stream);
    TQ_CUDA_CHECK(e);
    return TQ_OK;
}

template <typename T>
static cudaError_t launch_prologue(tq_ctx *ctx, const TqQprepArgs &qa, const TqPackArgs *append, cudaStream_t stream) {
    const int n_qprep = (int)qa.kv_rows * ((qa.G + 3) / 4) * (qa.use_qjl ? 2 : 1);
    if (!append) return tq_launch_kernel(tq_qprep_frag_kernel<T>, dim3(n_qprep), dim3(4 * TQ_D), 0, stream, true, qa);
    const int n_pack = append->n_kinds * append->B * append->H * append->S;
    const dim3 grid(n_qprep + n_pack), block(4 * TQ_D);
    if (!ctx->use_qjl) return tq_launch_kernel(tq_step_prologue_kernel<T, false, false>, grid, block, 0, stream, true, qa, *append, n_qprep);
    if (!tq_stages_matrices(ctx, n_qprep + n_pack))
        return tq_launch_kernel(tq_step_prologue_kernel<T, true, false>, grid, block, 0, stream, true, qa, *append, n_qprep);
    const cudaError_t e = tq_allow_shared<tq_step_prologue_kernel<T, true, true>>(ctx->device, kStagedMatrices);
    if (e != cudaSuccess) return e;
    return tq_launch_kernel(tq_step_prologue_kernel<T, true, true>, grid, block, kStagedMatrices, stream, true, qa, *append, n_qprep);
}

int32_t tq_launch_qprep_frag(tq_ctx *ctx, const void *q, int32_t q_dtype, int64_t kv_rows, int G, uint32_t *frag,
                             const TqPackArgs *append, cudaStream_t stream) {
    configure_small_kernels();
    if (G > 8 || q_dtype == TQ_DTYPE_F32) return TQ_ERR_UNSUPPORTED;  // (fp32 caches take the exact kernel, with tq_launch_qprep)
    TqQprepArgs qa;
    qa.q = q, qa.rot_k_t = ctx->rot_k_t, qa.qjl_t = ctx->qjl_t, qa.frag = frag;
    qa.G = G, qa.use_qjl = ctx->use_qjl, qa.kv_rows = kv_rows;
    cudaError_t e;
    if (q_dtype == TQ_DTYPE_F16) e = launch_prologue<__half>(ctx, qa, append, stream);
    else e = launch_prologue<__nv_bfloat16>(ctx, qa, append, stream);
    TQ_CUDA_CHECK(e);
    return TQ_OK;
}

template <typename T>
static cudaError_t launch_combine(const CombineArgs &a, dim3 grid, cudaStream_t stream, bool programmatic) {
    if (a.n_tail > 0 && a.tail_rows) {
        tq_combine_row_kernel<T><<<grid.x / ((a.G + 3) / 4) * a.G, TQ_D, 0, stream>>>(a);
        return cudaGetLastError();
    }
    if (a.n_tail == 0)
        return tq_launch_kernel(tq_combine_group_kernel<T, false>, grid, dim3(4 * TQ_D), 0, stream, programmatic, a);
    return tq_launch_cluster(tq_combine_group_kernel<T, true>, dim3(grid.x * a.tail_ctas), dim3(4 * TQ_D), sizeof(TailShared),
                             stream, programmatic, a.tail_ctas, a);
}

int32_t tq_launch_combine(const CombineArgs &a, int32_t q_dtype, int64_t rows, cudaStream_t stream, bool programmatic) {
    configure_small_kernels();
    if (a.G > 8) return TQ_ERR_UNSUPPORTED;
    const dim3 grid((unsigned)(rows / a.G) * ((a.G + 3) / 4));  // one block per four heads of a KV row
    cudaError_t e;
    if (q_dtype == TQ_DTYPE_F32) e = launch_combine<float>(a, grid, stream, programmatic);
    else if (q_dtype == TQ_DTYPE_F16) e = launch_combine<__half>(a, grid, stream, programmatic);
    else e = launch_combine<__nv_bfloat16>(a, grid, stream, programmatic);
    TQ_CUDA_CHECK(e);
    return TQ_OK;
}

// The tail fields of the combine arguments: `tail_vec` when every row of both tensors starts on a 16-byte boundary, and
// which kernel attends the tail of `kv_rows` KV rows.
//
// tq_combine_group_kernel needs an SM per block (four heads of a KV row), so that it takes 5 us more for every wave of blocks after
// the first; tq_combine_row_kernel takes a sixteenth of an SM per head, but a trip to memory for every four tail tokens.  So the
// more blocks there are to an SM, the longer the tail up to which the second is faster.  Measured where they cross (148 SMs,
// 512 / 4096 packed tokens, the tail in L2 / in HBM; us row kernel against group kernel): 64 blocks nowhere (17.1 against 14.4 at
// one token); 128 blocks at 12 / 8 tokens (19.7 against 21.0 at one, 38.9 against 37.7 at 16); 256 at 58 / 17 (35.6 against 38.7,
// 75.8 against 71.0 at 33); 512 at 125 / 96 (62 against 74, 137.8 against 137.0 at 96): 8 tokens times the square of blocks per SM.
//
// In the group kernel a row's tail is split over the CTAs of a cluster where that pays.  A CTA takes 28 ns per token; a
// cluster costs less than 64 tokens' time while its CTAs find half of the SMs free, 100 to 190 tokens' time up to all of them
// (its CTAs need free SMs of one GPC at once), and more beyond (us for 1 / 2 / 4 CTAs, 512 packed tokens: 8 blocks, 300 tail
// tokens 20.5 / 16.4 / 15.6, 128: 14.6 / 14.8; 32 blocks, 300: 20.7 / 16.8 / 20.2, 1000: 38.1 / 25.2 / 22.8; 64 blocks, 128:
// 16.3 / 20.4, 512: 25.4 / 23.4 / 32.3; 128 blocks, 300: 28.7 / 35.8 / 53.8).
int32_t tq_set_combine_tail(CombineArgs &c, const tq_dense_desc *k, const tq_dense_desc *v, int32_t n_tail, int32_t q_dtype,
                            int64_t kv_rows, int sm_count) {
    c.n_tail = n_tail, c.tail_k = c.tail_v = nullptr, c.tail_vec = c.tail_rows = false, c.tail_ctas = 0, c.tail_per_cta = 0;
    c.tk_sb = c.tk_sh = c.tk_st = c.tv_sb = c.tv_sh = c.tv_st = 0;
    if (n_tail == 0) return TQ_OK;
    if (k->dtype != q_dtype || v->dtype != q_dtype) return TQ_ERR_ARG;
    const int64_t blocks = kv_rows * ((c.G + 3) / 4);
    c.tail_rows = 2 * blocks > sm_count && n_tail <= kRowTailTokens && n_tail <= 8 * blocks * blocks / ((int64_t)sm_count * sm_count);
    int ctas = 1;
    int64_t cost = n_tail;
    for (int n = 2; n <= kTailCtas && n * blocks <= sm_count; n *= 2) {
        const int64_t with = (n_tail + n - 1) / n + (2 * n * blocks <= sm_count ? 64 : 192);
        if (with < cost) ctas = n, cost = with;
    }
    c.tail_per_cta = (n_tail + ctas - 1) / ctas;
    c.tail_ctas = (n_tail + c.tail_per_cta - 1) / c.tail_per_cta;  // (none of them empty)
    c.tail_k = k->data, c.tail_v = v->data;
    c.tk_sb = k->stride_b, c.tk_sh = k->stride_h, c.tk_st = k->stride_t;
    c.tv_sb = v->stride_b, c.tv_sh = v->stride_h, c.tv_st = v->stride_t;
    const int64_t strides = c.tk_sb | c.tk_sh | c.tk_st | c.tv_sb | c.tv_sh | c.tv_st;
    const int64_t elem = q_dtype == TQ_DTYPE_F32 ? 4 : 2;
    c.tail_vec = !((strides * elem | (int64_t)(uintptr_t)k->data | (int64_t)(uintptr_t)v->data) & 15);
    return TQ_OK;
}

int32_t tq_launch_gather_wait(const tq_gather_desc *g, int *error_flag, int limit_ms, int32_t batch, size_t elem_bytes,
                              void *out_final, cudaStream_t stream, int64_t rows_per_step) {
    if (rows_per_step <= 0) rows_per_step = (int64_t)batch * (g->q_heads_total / g->world);
    // out_final: the whole gathered output [batch, q_heads_total, 128], or (out_local_only) this
    // rank's heads of it [batch, q_heads_total / world, 128]
    size_t n16 = 0, row_len16 = 1, row_stride16 = 0, src_off16 = 0;
    if (out_final) {
        const size_t head16 = TQ_D * elem_bytes / 16;
        const size_t heads_local = (size_t)g->q_heads_total / g->world;
        if (g->out_local_only) {
            row_len16 = heads_local * head16, row_stride16 = (size_t)g->q_heads_total * head16;
            src_off16 = (size_t)g->rank * heads_local * head16, n16 = (size_t)batch * row_len16;
        } else {
            n16 = (size_t)batch * g->q_heads_total * head16, row_len16 = n16;
        }
    }
    const int blocks = out_final ? (int)((n16 + 255) / 256 < 64 ? (n16 + 255) / 256 : 64) : 1;
    // Launched as a programmatic dependent: with a host-side step number it begins polling while the
    // combine kernel that raises this rank's own flag is still finishing (harmless: the flags carry
    // the step number); what follows it in the stream still starts only after it has seen every
    // rank's flag, this rank's included.
    cudaError_t e = tq_launch_kernel(tq_gather_wait_kernel, dim3(blocks < 1 ? 1 : blocks), dim3(256), 0, stream, true,
                                     (const unsigned *)g->flags[g->rank], (int)g->world, (unsigned)g->seq,
                                     (unsigned *)g->seq_dev, (unsigned)rows_per_step,
                                     (unsigned *)g->counter, error_flag,
                                     (unsigned long long)(limit_ms < 1 ? 1 : limit_ms) * 1000000ull,
                                     reinterpret_cast<const uint4 *>(g->out[g->rank]), (long long)g->out_stride,
                                     reinterpret_cast<uint4 *>(out_final), n16, row_len16, row_stride16, src_off16);
    TQ_CUDA_CHECK(e);
    return TQ_OK;
}

DecodeWorkspace tq_carve_workspace(void *workspace, int64_t rows, int n_splits) {
    DecodeWorkspace w;
    float *p = (float *)workspace;
    w.qrot = p;
    p += rows * TQ_D;
    w.qproj = p;
    p += rows * TQ_D;
    p += rows * 8;
    w.part_m = p;
    p += rows * n_splits;
    w.part_l = p;
    p += rows * n_splits;
    w.part_acc = p;
    return w;
}

int32_t tq_launch_decode_exact(tq_ctx *ctx, const void *q, int32_t q_dtype, int32_t q_heads,
                               const tq_cache_desc *cache, int32_t seq_len, const tq_dense_desc *tail_k,
                               const tq_dense_desc *tail_v, int32_t n_tail, int32_t n_splits, void *workspace,
                               void *out, cudaStream_t stream) {
    const int64_t rows = (int64_t)cache->batch * q_heads;
    DecodeWorkspace w = tq_carve_workspace(workspace, rows, n_splits);
    const bool packed = seq_len > 0;  // else the tail alone: the combine kernel merges no splits (1024 rows of 4 heads, 16 tail tokens: 86 -> 24 us)
    int rc = packed ? tq_launch_qprep(ctx, q, q_dtype, rows, w.qrot, w.qproj, stream) : TQ_OK;
    if (rc) return rc;

    ExactArgs a;
    a.k_codes = cache->k_codes, a.k_norms = cache->k_norms;
    a.k_signs = cache->k_signs, a.k_rnorms = cache->k_rnorms;
    a.v_codes = cache->v_codes, a.v_norms = cache->v_norms;
    a.cache_sb = cache->stride_b, a.cache_sh = cache->stride_h;
    a.Hkv = cache->kv_heads, a.G = q_heads / cache->kv_heads, a.N = seq_len, a.n_splits = n_splits;
    a.seq_start = cache->seq_start;
    a.qrot = w.qrot, a.qproj = w.qproj;
    a.part_m = w.part_m, a.part_l = w.part_l, a.part_acc = w.part_acc;
    a.centers_k = ctx->centers_k, a.centers_v = ctx->centers_v;
    dim3 grid(n_splits, cache->batch * cache->kv_heads);
    const int mode = ctx->use_qjl * 10 + ctx->bits;
    tq_prof_count(ctx, packed ? 3 : 1);
    if (packed) {
        tq_prof_begin(ctx, stream);
        cudaError_t e;
        switch (mode) {
            case 2: e = launch_exact<2, 2, false>(a, ctx->device, grid, stream); break;
            case 3: e = launch_exact<3, 3, false>(a, ctx->device, grid, stream); break;
            case 4: e = launch_exact<4, 4, false>(a, ctx->device, grid, stream); break;
            case 12: e = launch_exact<1, 2, true>(a, ctx->device, grid, stream); break;
            case 13: e = launch_exact<2, 3, true>(a, ctx->device, grid, stream); break;
            case 14: e = launch_exact<3, 4, true>(a, ctx->device, grid, stream); break;
            default: return TQ_ERR_UNSUPPORTED;
        }
        tq_prof_end(ctx, stream);
        TQ_CUDA_CHECK(e);
    }

    CombineArgs c;
    c.part_m = w.part_m, c.part_l = w.part_l, c.part_acc = w.part_acc;
    c.n_splits = packed ? n_splits : 0, c.Hq = q_heads, c.G = a.G;
    c.seg_chunk = 0, c.seg_npad = 0;
    c.len_ptr = nullptr, c.len_add = 0, c.capacity = 0, c.plan_rows = 0, c.plan_ctas = 0, c.plan_step = 0;
    c.sm_count = 0, c.next_blocks = 0;
    c.gather_world = 0, c.parts = 0, c.part = 0, c.head_group = 0, c.exch_rows = 0;
    c.rot_v = ctx->rot_v;
    c.q = q, c.out = out, c.out_f32 = nullptr;
    rc = tq_set_combine_tail(c, tail_k, tail_v, n_tail, q_dtype, (int64_t)cache->batch * cache->kv_heads, ctx->sm_count);
    if (rc) return rc;
    // (a combine kernel reads the tail without a wait of its own, see tq_combine_group_kernel: alone it starts the ordinary way)
    return tq_launch_combine(c, q_dtype, rows, stream, /*programmatic=*/packed);
}
