// Helpers shared by the chunk-local forward (tc_intra.cu) and backward (tc_bwd_chunk.cu) kernels.
#pragma once
#include "common.cuh"
#include "umma.cuh"

namespace mkda {

using umma::store_split8;

__device__ __forceinline__ void lds8(const float* p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void sts8(float* p, const float (&v)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void lds8(const float* p, f32x2 (&v)[4]) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p), b = *reinterpret_cast<const ulonglong2*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void sts8(float* p, const f32x2 (&v)[4]) {
    *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v[0], v[1]);
    *reinterpret_cast<ulonglong2*>(p + 4) = make_ulonglong2(v[2], v[3]);
}
__device__ __forceinline__ void lds4(const float* p, f32x2 (&v)[2]) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p);
    v[0] = a.x; v[1] = a.y;
}
// channels 8 k8 .. 8 k8 + 7 of a 128-float row that is stored as two planes: the lower, then the upper four of every eight
__device__ __forceinline__ void lds_halves(const float* row, int k8, f32x2 (&v)[4]) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(row + 4 * k8), b = *reinterpret_cast<const ulonglong2*>(row + 64 + 4 * k8);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void sts_halves(float* row, int k8, const f32x2 (&v)[4]) {
    *reinterpret_cast<ulonglong2*>(row + 4 * k8) = make_ulonglong2(v[0], v[1]);
    *reinterpret_cast<ulonglong2*>(row + 64 + 4 * k8) = make_ulonglong2(v[2], v[3]);
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) { return fma2(b, both(-1.f), a); }
// out = x 2^(a - b), eight values as four pairs
__device__ __forceinline__ void scale_ex2(f32x2 (&out)[4], const f32x2 (&x)[4], const f32x2 (&a)[4], const f32x2 (&b)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) out[e] = mul2(x[e], ex2f2_(sub2(a[e], b[e])));
}
template <int DT>
__device__ __forceinline__ void unpack8(const Raw8& r, f32x2 (&v)[4]) {
    float f[8];
    unpack8<DT>(r, f);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = pack2(f[2 * e], f[2 * e + 1]);
}
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"(umma::smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void publish() {
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
}
// Sums of 2 N columns over the 32 lanes of a warp: every exchange halves the number of columns a lane carries, so 16 columns take
// 16 shuffles and 8 columns 9 instead of 5 per column.  Afterwards v[0] of the lane whose bits below 32 / N ... spell the column
// holds the sum: 16 columns -> column (lane >> 1) & 15, 8 columns -> column (lane >> 2) & 7 (all lanes of a group hold it).
template <int COLS>
__device__ __forceinline__ void warp_colsum(float (&v)[COLS], int lane) {
    int bit = 16;
#pragma unroll
    for (int w = COLS / 2; w >= 1; w >>= 1, bit >>= 1) {
#pragma unroll
        for (int j = 0; j < w; ++j) {
            const float recv = __shfl_xor_sync(0xffffffffu, (lane & bit) ? v[j] : v[j + w], bit);
            v[j] = ((lane & bit) ? v[j + w] : v[j]) + recv;
        }
    }
#pragma unroll
    for (; bit >= 1; bit >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], bit);
}

}  // namespace mkda
