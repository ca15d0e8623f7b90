// Prefix combine of per-segment (state, transition) pairs: the step that joins the segments of one long sequence, and
// the ranks of a context-parallel group, into the states entering each segment.
#include "common.cuh"
#include "host.h"

namespace mkda {

constexpr int LDA = 132;   // [128][128] matrix, row stride
constexpr int CW = 32;     // state columns per CTA
constexpr int LDS = CW + 8;   // [128][CW] tile, row stride

// ---------------------------------------------------------------------------------------------------------
// prefix combine over the segments of a group: one CTA per (32-column block, v-head, group).
//   forward:  X <- M_s X + H_s          backward: X <- M_s^T X + D_s
// X enters segment s before the update (stored to s_in[s]).  Plain fp32 keeps the carried state at fp32 accuracy however many segments are
// chained.  The chain is serial, so the next segment's transition matrix is copied into the second buffer (cp.async) and its H / D block into
// registers while the current product runs.
// The product of a step (128 x 32 x 128) is what takes the time.  A thread computes 8 x 4 outputs over half of the 128 terms: what its tile
// loads from shared memory, 128 B per cycle into registers, is the bound (6.1 k cycles; the multiplications alone 4.1 k).  The halves are added
// through shared memory, and each of the two threads keeps four of the eight rows.  (Compensated TF32 products of the older tensor
// instructions take 12 k; 32 segments of 32 heads 194 -> 163 us, 16 segments 93 -> 81 us.)
// ---------------------------------------------------------------------------------------------------------
constexpr int COMBINE_SMEM = (DK * LDS + 2 * DK * LDA + 16 * 256) * 4;

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(gsrc) : "memory");
}

// acc[r][e] += a[r] b[e]
__device__ __forceinline__ void add_outer(float (&acc)[8][4], const float (&a)[8], const float4& b) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        acc[r][0] = fmaf(a[r], b.x, acc[r][0]); acc[r][1] = fmaf(a[r], b.y, acc[r][1]);
        acc[r][2] = fmaf(a[r], b.z, acc[r][2]); acc[r][3] = fmaf(a[r], b.w, acc[r][3]);
    }
}

__global__ void __launch_bounds__(256, 1) combine_kernel(const MkdaCombine p) {
    follow_stream();
    extern __shared__ __align__(16) float smem[];
    float* sX = smem;                                  // [128][LDS]
    float* sM = sX + DK * LDS;                         // 2 x [128][LDA]  M[m][k] (forward) or M[k][m] (reverse)
    float4* sHalf = reinterpret_cast<float4*>(sM + 2 * DK * LDA);     // [4][256] partial sums on their way to the other half's thread
    const int cb = blockIdx.x, h = blockIdx.y, grp = blockIdx.z, HV = p.HV;
    const int col0 = cb * CW;
    const int tid = threadIdx.x, half = tid >> 7, lane = tid & 31;
    const int row8 = 8 * (((tid >> 5) & 3) * 4 + (lane >> 3)), c4 = 4 * (lane & 7), row = row8 + 4 * half;      // keeps rows row .. row + 3, columns c4 .. c4 + 3
    float X[4][4], Hn[4][4];
    {
        const float* src = p.carry ? p.carry + ((size_t)grp * HV + h) * DK * DV : nullptr;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int kk = row + i, cc = col0 + c4 + e;
                X[i][e] = src ? (p.carry_v_first ? src[(size_t)cc * DK + kk] : src[(size_t)kk * DV + cc]) : 0.f;
            }
    }
    const int s_beg = p.grp_seg_off[grp], s_end = p.grp_seg_off[grp + 1], n = s_end - s_beg;
    auto seg = [&](int i) { return p.reverse ? s_end - 1 - i : s_beg + i; };
    auto fetch_m = [&](int i, float* dst) {            // 64 KB, 16 x 16 bytes per thread
        const float* src = p.ms + ((size_t)seg(i) * HV + h) * DK * DK;
        for (int j = tid; j < DK * 32; j += 256) {
            const int r = j >> 5, c = (j & 31) * 4;
            cp_async16(dst + r * LDA + c, src + (size_t)r * DK + c);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto fetch_h = [&](int i) {
        const size_t base = ((size_t)seg(i) * HV + h) * DK * DV;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float4 a = p.hs ? *reinterpret_cast<const float4*>(p.hs + base + (size_t)(row + r) * DV + col0 + c4) : make_float4(0.f, 0.f, 0.f, 0.f);
            Hn[r][0] = a.x; Hn[r][1] = a.y; Hn[r][2] = a.z; Hn[r][3] = a.w;
        }
    };
    const int products = p.s_out ? n : n - 1;          // the last one leads to s_out only (16 segments of 32 heads 83 -> 78 us without)
    if (products > 0) { fetch_m(0, sM); fetch_h(0); }
    for (int i = 0; i < n; ++i) {
        const int cur = i & 1;
        const size_t base = ((size_t)seg(i) * HV + h) * DK * DV;
        if (i + 1 < products) fetch_m(i + 1, sM + (cur ^ 1) * DK * LDA);   // its last reader, the product of step i - 1, is behind a barrier
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float4 x = make_float4(X[r][0], X[r][1], X[r][2], X[r][3]);
            *reinterpret_cast<float4*>(sX + (row + r) * LDS + c4) = x;
            if (p.s_in) *reinterpret_cast<float4*>(p.s_in + base + (size_t)(row + r) * DV + col0 + c4) = x;
        }
        if (i == products) break;
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int e = 0; e < 4; ++e) X[r][e] = Hn[r][e];
        if (i + 1 < products) {
            fetch_h(i + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");     // this step's matrix has landed, the next may be in flight
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        float acc[8][4];
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
        const float *m = sM + cur * DK * LDA, *x = sX + c4;
        if (p.reverse) {
#pragma unroll 4
            for (int k = 64 * half; k < 64 * half + 64; ++k) {
                const float4 a0 = *reinterpret_cast<const float4*>(m + k * LDA + row8), a1 = *reinterpret_cast<const float4*>(m + k * LDA + row8 + 4);
                const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
                add_outer(acc, a, *reinterpret_cast<const float4*>(x + k * LDS));
            }
        } else {
#pragma unroll 1
            for (int k = 64 * half; k < 64 * half + 64; k += 4) {
                float4 a4[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) a4[r] = *reinterpret_cast<const float4*>(m + (row8 + r) * LDA + k);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float a[8];
#pragma unroll
                    for (int r = 0; r < 8; ++r) a[r] = e == 0 ? a4[r].x : e == 1 ? a4[r].y : e == 2 ? a4[r].z : a4[r].w;
                    add_outer(acc, a, *reinterpret_cast<const float4*>(x + (k + e) * LDS));
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
            sHalf[r * 256 + tid] = half ? make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]) : make_float4(acc[4 + r][0], acc[4 + r][1], acc[4 + r][2], acc[4 + r][3]);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float4 o = sHalf[r * 256 + (tid ^ 128)];
            const float other[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) X[r][e] += (half ? acc[4 + r][e] : acc[r][e]) + other[e];
        }
    }
    if (p.s_out) {
        float* out = p.s_out + ((size_t)grp * HV + h) * DK * DV;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if (p.out_v_first) {
#pragma unroll
                for (int e = 0; e < 4; ++e) out[(size_t)(col0 + c4 + e) * DK + row + r] = X[r][e];
            } else {
                *reinterpret_cast<float4*>(out + (size_t)(row + r) * DV + col0 + c4) = make_float4(X[r][0], X[r][1], X[r][2], X[r][3]);
            }
        }
    }
}

}  // namespace mkda

using namespace mkda;

extern "C" int mkda_state_combine(const MkdaCombine* p, void* stream) {
    if (!p || !p->grp_seg_off || !p->ms || (!p->s_in && !p->s_out)) return set_error(MKDA_ERR_ARG, "state_combine: null argument");
    if (p->NG == 0) return MKDA_OK;
    if (any_misaligned(p->ms, p->hs, p->s_in, p->s_out)) return set_error(MKDA_ERR_ARG, "state_combine: ms, hs, s_in and s_out must be 16-byte aligned");
    if (int e = ensure_smem((const void*)combine_kernel, COMBINE_SMEM, "state_combine")) return e;
    launch(combine_kernel, dim3(DV / CW, p->HV, p->NG), 256, COMBINE_SMEM, (cudaStream_t)stream, *p);
    return check_launch("state_combine");
}
