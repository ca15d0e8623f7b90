// Helpers shared by the chunk-local forward (tc_intra.cu) and backward (tc_bwd_chunk.cu) kernels.
#pragma once
#include "common.cuh"
#include "umma.cuh"

namespace mkda {

using umma::store_split8;

__device__ __forceinline__ void ldg8(const void* base, int dtype, size_t idx, float (&v)[8]) {
    ld8(base, dtype, idx, v);
}
__device__ __forceinline__ void lds8(const float* p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void sts8(float* p, const float (&v)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
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
