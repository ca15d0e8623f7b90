// Shared device helpers for the KDA / GDN kernels (sm_100a).
//
// Numerics policy: the contractions of the chunk kernels run on the tensor cores with the error-compensated three-product split
// (a = hi + lo, a*b ~ lo_a*hi_b + hi_a*lo_b + hi_a*hi_b) and fp32 accumulation: bf16 halves on tcgen05 (umma.cuh), and TF32 halves on
// mma.sync in the 16- and 32-row merges of the triangular inverse (warp_mma_short below).  The prefix combine and the step kernel are plain
// fp32.  Inputs may be fp32, bf16 or fp16 in global memory; they are widened to fp32 when staged.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/mkda.h"

namespace mkda {

constexpr int CH = 64;    // chunk length
constexpr int DK = 128;   // key dim
constexpr int DV = 128;   // value dim
constexpr float RCP_LN2 = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

// ---------------------------------------------------------------------------------------------------------
// typed global access: 4 consecutive elements starting at element index `idx` (idx % 4 == 0)
// ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float4 ld4(const void* base, int dtype, size_t idx) {
    if (dtype == MKDA_F32) return *reinterpret_cast<const float4*>(static_cast<const float*>(base) + idx);
    uint2 raw = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(base) + idx);
    float4 r;
    if (dtype == MKDA_BF16) {
        r.x = __uint_as_float(raw.x << 16);
        r.y = __uint_as_float(raw.x & 0xffff0000u);
        r.z = __uint_as_float(raw.y << 16);
        r.w = __uint_as_float(raw.y & 0xffff0000u);
    } else {
        __half2 a = *reinterpret_cast<__half2*>(&raw.x), b = *reinterpret_cast<__half2*>(&raw.y);
        float2 fa = __half22float2(a), fb = __half22float2(b);
        r = make_float4(fa.x, fa.y, fb.x, fb.y);
    }
    return r;
}

// 8 consecutive elements starting at element index `idx` (idx % 8 == 0): one 16-byte load for the 16-bit types
__device__ __forceinline__ void ld8(const void* base, int dtype, size_t idx, float (&v)[8]) {
    if (dtype == MKDA_F32) {
        const float4 a = *reinterpret_cast<const float4*>(static_cast<const float*>(base) + idx);
        const float4 b = *reinterpret_cast<const float4*>(static_cast<const float*>(base) + idx + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        return;
    }
    const uint4 raw = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(base) + idx);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (dtype == MKDA_BF16) {
            v[2 * e] = __uint_as_float(w[e] << 16);
            v[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
        } else {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
            v[2 * e] = f.x; v[2 * e + 1] = f.y;
        }
    }
}

// Every kernel of the library is launched (host.h: launch) so that the launch itself and the kernel's start-up lie under the end of the kernel
// in front of it in the stream.  Each thread calls this before it touches global memory: it waits until that kernel has completed and its
// writes are visible.  (Letting the next kernel's blocks in earlier, by griddepcontrol.launch_dependents, costs 1 to 5 %: they take up places
// and caches while they wait.)
__device__ __forceinline__ void follow_stream() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The same eight elements as raw bytes (one 16-byte piece, two for fp32), widened later by unpack8.  A conversion next to the
// load makes the thread wait for the data there and then; a load whose bytes are only parked in registers stays in flight
// until its first real use, which may be a whole phase (or the top of the next item) later.
struct Raw8 { uint4 a, b; };
template <int DT>
__device__ __forceinline__ void ldraw8(const void* base, size_t idx, Raw8& r) {
    if (DT == MKDA_F32) {
        r.a = *reinterpret_cast<const uint4*>(static_cast<const float*>(base) + idx);
        r.b = *reinterpret_cast<const uint4*>(static_cast<const float*>(base) + idx + 4);
    } else {
        r.a = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(base) + idx);
    }
}
template <int DT>
__device__ __forceinline__ void unpack8(const Raw8& r, float (&v)[8]) {
    if (DT == MKDA_F32) {
        v[0] = __uint_as_float(r.a.x); v[1] = __uint_as_float(r.a.y); v[2] = __uint_as_float(r.a.z); v[3] = __uint_as_float(r.a.w);
        v[4] = __uint_as_float(r.b.x); v[5] = __uint_as_float(r.b.y); v[6] = __uint_as_float(r.b.z); v[7] = __uint_as_float(r.b.w);
        return;
    }
    const uint32_t w[4] = {r.a.x, r.a.y, r.a.z, r.a.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (DT == MKDA_BF16) {
            v[2 * e] = __uint_as_float(w[e] << 16);
            v[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
        } else {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
            v[2 * e] = f.x; v[2 * e + 1] = f.y;
        }
    }
}

__device__ __forceinline__ float ld1(const void* base, int dtype, size_t idx) {
    if (dtype == MKDA_F32) return static_cast<const float*>(base)[idx];
    if (dtype == MKDA_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(base)[idx]);
    return __half2float(static_cast<const __half*>(base)[idx]);
}

__device__ __forceinline__ void st1(void* base, int dtype, size_t idx, float v) {
    if (dtype == MKDA_F32) static_cast<float*>(base)[idx] = v;
    else if (dtype == MKDA_BF16) static_cast<__nv_bfloat16*>(base)[idx] = __float2bfloat16_rn(v);
    else static_cast<__half*>(base)[idx] = __float2half_rn(v);
}


__device__ __forceinline__ void st4(void* base, int dtype, size_t idx, float4 v) {          // idx % 4 == 0
    if (dtype == MKDA_F32) {
        *reinterpret_cast<float4*>(static_cast<float*>(base) + idx) = v;
    } else if (dtype == MKDA_BF16) {
        __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
        uint2 raw = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
        *reinterpret_cast<uint2*>(static_cast<uint16_t*>(base) + idx) = raw;
    } else {
        __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
        uint2 raw = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
        *reinterpret_cast<uint2*>(static_cast<uint16_t*>(base) + idx) = raw;
    }
}

// two values rounded to the 16-bit type DT, in one word
template <int DT>
__device__ __forceinline__ uint32_t pack16(float a, float b) {
    if (DT == MKDA_BF16) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&v);
    }
    const __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// 8 consecutive elements, idx % 8 == 0
template <int DT>
__device__ __forceinline__ void st8(void* base, size_t idx, const float (&v)[8]) {
    if (DT == MKDA_F32) {
        st4(base, DT, idx, make_float4(v[0], v[1], v[2], v[3]));
        st4(base, DT, idx + 4, make_float4(v[4], v[5], v[6], v[7]));
        return;
    }
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = pack16<DT>(v[2 * e], v[2 * e + 1]);
    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(base) + idx) = make_uint4(w[0], w[1], w[2], w[3]);
}

// 32 bytes in one store, `dst` 32-byte aligned
__device__ __forceinline__ void st32b(void* dst, const uint32_t (&w)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 :: "l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}

// ---------------------------------------------------------------------------------------------------------
// tensor-core primitive: m16n8k8 TF32, fp32 accumulate.
// Fragment ownership (g = lane >> 2, t = lane & 3):
//   A (16x8):  a0 (g, t)  a1 (g+8, t)  a2 (g, t+4)  a3 (g+8, t+4)
//   B (8x8):   b0 (k = t, n = g)       b1 (k = t+4, n = g)
//   C (16x8):  c0 (g, 2t) c1 (g, 2t+1) c2 (g+8, 2t) c3 (g+8, 2t+1)
// ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ void mma_tf32_raw(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// a value as two TF32 parts
struct FragA {
    uint32_t hi[4], lo[4];
    __device__ __forceinline__ void set(int i, float x) {
        hi[i] = to_tf32(x);
        lo[i] = to_tf32(x - __uint_as_float(hi[i]));
    }
};
struct FragB {
    uint32_t hi[2], lo[2];
    __device__ __forceinline__ void set(int i, float x) {
        hi[i] = to_tf32(x);
        lo[i] = to_tf32(x - __uint_as_float(hi[i]));
    }
};

// acc[NT][4] = A(16 x KD) * B(KD x 8*NT) for one warp, KD a small multiple of 8.
//   A(m, k) = A[m * ARS + k * ACS]   (pointer already offset to the warp's first row)
//   B(k, n) = B[k * BKS + n * BNS]   (pointer already offset to the warp's first column)
// All fragments are loaded first, and the three products of the compensation are summed apart, so that the chain of products is short.
template <int NT, int KD, int ARS, int ACS, int BKS, int BNS>
__device__ __forceinline__ void warp_mma_short(float (&acc)[NT][4], const float* __restrict__ A, const float* __restrict__ B) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const float* ap = A + g * ARS + t * ACS;
    const float* bp = B + t * BKS + g * BNS;
    FragA fa[KD / 8];
    FragB fb[KD / 8][NT];
#pragma unroll
    for (int k = 0; k < KD / 8; ++k) {
        fa[k].set(0, ap[8 * k * ACS]);
        fa[k].set(1, ap[8 * ARS + 8 * k * ACS]);
        fa[k].set(2, ap[(8 * k + 4) * ACS]);
        fa[k].set(3, ap[8 * ARS + (8 * k + 4) * ACS]);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            fb[k][nt].set(0, bp[8 * k * BKS + nt * 8 * BNS]);
            fb[k][nt].set(1, bp[(8 * k + 4) * BKS + nt * 8 * BNS]);
        }
    }
    float lh[NT][4], hl[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) lh[nt][e] = hl[nt][e] = acc[nt][e] = 0.f;
#pragma unroll
    for (int k = 0; k < KD / 8; ++k)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            mma_tf32_raw(lh[nt], fa[k].lo, fb[k][nt].hi);
            mma_tf32_raw(hl[nt], fa[k].hi, fb[k][nt].lo);
            mma_tf32_raw(acc[nt], fa[k].hi, fb[k][nt].hi);
        }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[nt][e] += lh[nt][e] + hl[nt][e];
}

// acc[2][4] = A(16 x 16) * B(16 x 16) for one warp with A as the accumulators of an earlier product (its columns 2 t, 2 t + 1 of every eight
// taken as the terms t, t + 4), B(k, n) = B[k * ld + n]
__device__ __forceinline__ void warp_mma_chained(float (&acc)[2][4], const float (&A)[2][4], const float* __restrict__ B, int ld) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    FragA fa[2];
    FragB fb[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        fa[k].set(0, A[k][0]); fa[k].set(1, A[k][2]); fa[k].set(2, A[k][1]); fa[k].set(3, A[k][3]);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            fb[k][nt].set(0, B[(8 * k + 2 * t) * ld + 8 * nt + g]);
            fb[k][nt].set(1, B[(8 * k + 2 * t + 1) * ld + 8 * nt + g]);
        }
    }
    float lh[2][4], hl[2][4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) lh[nt][e] = hl[nt][e] = acc[nt][e] = 0.f;
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            mma_tf32_raw(lh[nt], fa[k].lo, fb[k][nt].hi);
            mma_tf32_raw(hl[nt], fa[k].hi, fb[k][nt].lo);
            mma_tf32_raw(acc[nt], fa[k].hi, fb[k][nt].hi);
        }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[nt][e] += lh[nt][e] + hl[nt][e];
}

// Two fp32 operations in one instruction (a pair of registers each): the staging and epilogue code is bound by instruction issue.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ f32x2 both(float a) { return pack2(a, a); }

// 2^x in one MUFU instruction (max relative error ~2^-22); used where 2^x scales tensor-core operands
__device__ __forceinline__ float ex2f_(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Stable scalar math on the MUFU unit (ex2 / lg2 / rcp approximations, relative error ~1e-7 each, absolute error of
// softplus < 1e-7): the gate and epilogue kernels evaluate several of these per element and were ALU-bound with the
// precise library versions.
__device__ __forceinline__ float expf_(float x) { return ex2f_(x * RCP_LN2); }
__device__ __forceinline__ float sigmoidf_(float z) { return __fdividef(1.f, 1.f + expf_(-z)); }
__device__ __forceinline__ float softplusf_(float s) { return fmaxf(s, 0.f) + __log2f(1.f + expf_(-fabsf(s))) * LN2; }

__device__ __forceinline__ float rcpf_(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ f32x2 ex2f2_(f32x2 v) {
    float a, b;
    unpack2(v, a, b);
    return pack2(ex2f_(a), ex2f_(b));
}
__device__ __forceinline__ f32x2 sigmoidf2_(f32x2 z) {
    float a, b;
    unpack2(add2(ex2f2_(mul2(z, both(-RCP_LN2))), both(1.f)), a, b);
    return pack2(rcpf_(a), rcpf_(b));
}

// Gated RMSNorm of a 128-value row.  Two kernels evaluate it (with the state chain, or on its own), chosen by sizes; results must not depend on
// that choice, so the order of every operation is fixed here.  A row is 32 pieces of four values; piece c + 8 i belongs to column c = 0..7,
// a column adds its four pieces in order, and the eight columns are then added by a butterfly (xor 4, 2, 1).
__device__ __forceinline__ float norm_piece(const float4& x) { return __fadd_rn(fmaf(x.x, x.x, __fmul_rn(x.y, x.y)), fmaf(x.z, x.z, __fmul_rn(x.w, x.w))); }
__device__ __forceinline__ float norm_butterfly(float s) {
#pragma unroll
    for (int sft = 4; sft > 0; sft >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, sft));
    return s;
}
__device__ __forceinline__ float norm_rs(float sum, float eps) { return rsqrtf(fmaf(sum, 1.f / 128.f, eps)); }
__device__ __forceinline__ float4 norm_gate(const float4& x, const float4& w, const float4& z, float rs, bool silu) {
    f32x2 a = sigmoidf2_(pack2(z.x, z.y)), b = sigmoidf2_(pack2(z.z, z.w));
    if (silu) { a = mul2(a, pack2(z.x, z.y)); b = mul2(b, pack2(z.z, z.w)); }
    a = mul2(mul2(a, both(rs)), mul2(pack2(w.x, w.y), pack2(x.x, x.y)));
    b = mul2(mul2(b, both(rs)), mul2(pack2(w.z, w.w), pack2(x.z, x.w)));
    float4 r;
    unpack2(a, r.x, r.y);
    unpack2(b, r.z, r.w);
    return r;
}


}  // namespace mkda
