// Host-side helpers shared by the launchers: error text behind mkda_last_error() and launch checking.
#pragma once
#include <stdint.h>
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/mkda.h"

namespace mkda {
int set_error(int code, const char* msg);
int check_launch(const char* what);
// Raises the dynamic shared memory limit of `func` (the attribute is set once per function and device; later calls
// return at once); returns 0 or an error code.
int ensure_smem(const void* func, int bytes, const char* what);
// Registers per thread the kernel is launched with (0 if unknown): a kernel whose warps redistribute registers checks its build with it.
int kernel_registers(const void* func);
// Tensor map over a row-major [rows][row_elems] tensor of 2- or 4-byte elements whose boxes are `box_rows` (64) rows x 128 elements,
// not swizzled: one tiled TMA copy then brings 64 strided 128-element rows (token rows of one head) into shared memory as a dense
// [64][128] block.  box_cols = 64 (2-byte elements): boxes of 64 elements with the 128-byte swizzle, a column block of an operand tile
// (umma.cuh).  Rows past the end of the tensor read as zeros.  Returns 0, or an error code when the tensor cannot be
// described (base not 16-byte aligned, row pitch not a multiple of 16 bytes, or the driver lacks the encoder).
int make_rows_map(CUtensorMap* out, const void* base, int elem_bytes, unsigned long long rows, unsigned long long row_elems, const char* what,
                  int box_rows = 64, int box_cols = 128);
// True if any of the (possibly null) pointers is not 16-byte aligned: the kernels read and write their tensors with
// 16-byte vector accesses and bulk copies, and a misaligned address would fault the device instead of returning an error.
template <typename... P>
inline bool any_misaligned(P... ptrs) {
    return (((reinterpret_cast<uintptr_t>(static_cast<const void*>(ptrs)) & 15) != 0) || ...);
}
// ... and the tiles and states that leave in 32-byte pieces
template <typename... P>
inline bool any_misaligned32(P... ptrs) {
    return (((reinterpret_cast<uintptr_t>(static_cast<const void*>(ptrs)) & 31) != 0) || ...);
}
// Launches a kernel that calls follow_stream(): the launch and the kernel's start-up then lie under the end of the kernel in front of it.
// Three to five us per kernel boundary less than a plain launch: 77-token prompt 35.1 -> 29.8 us, fp16 4 x 1000 tokens 323 -> 299 us.
template <typename... K, typename... A>
inline void launch(void (*kern)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, const A&... args) {
    cudaLaunchAttribute overlap{};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream; cfg.attrs = &overlap; cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, kern, args...);         // an error is picked up by check_launch
}
// Number of SMs of the current device (cached per device).
int sm_count();
int launch_out_fwd_tc(const MkdaOutFwd* p, cudaStream_t stream);
int tc_chunk_status(unsigned int* out);
int tc_chunk_status_clear();
int launch_rows_to_tiles(const MkdaLayout& L, const void* rows, int dtype, void* tiles, cudaStream_t stream);
int launch_ragged_rows_to_tiles(const MkdaLayout& L, const void* rows, void* tiles, cudaStream_t stream);
int launch_recur_fwd_tc(const MkdaRecurFwd* p, const int* seg_order, cudaStream_t stream);
int launch_chain_fwd_tc(const MkdaChainFwd* p, const int* seg_order, cudaStream_t stream);
int launch_bwd_dh_tc(const MkdaBwdDh* p, const int* seg_order, bool rows, cudaStream_t stream);
int tc_recur_status(unsigned int* out);
int tc_recur_status_clear();
int launch_intra_fwd_tc(const MkdaIntraFwd* p, const MkdaGateFwd* gate, cudaStream_t stream);      // gate: formed there, or NULL
int launch_bwd_chunk_tc(const MkdaBwdChunk* p, const void* d_o, void* dq, void* dk, cudaStream_t stream);      // rows instead of tiles, or NULL
int tc_bwd_chunk_status(unsigned int* out);
int tc_bwd_chunk_status_clear();
int step_status(unsigned int* out);
int step_status_clear();
int tc_intra_status(unsigned int* out);
int tc_intra_status_clear();
}  // namespace mkda
