// Error reporting and ABI self-description.
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <mutex>

#include "../../include/mkda.h"
#include "host.h"

namespace mkda {

static thread_local char g_err[512] = "";
static std::atomic<unsigned long long> g_launches{0};

int set_error(int code, const char* msg) {
    snprintf(g_err, sizeof(g_err), "%s", msg);
    return code;
}

int check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        snprintf(g_err, sizeof(g_err), "%s: %s", what, cudaGetErrorString(e));
        return MKDA_ERR_LAUNCH;
    }
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return MKDA_OK;
}

int sm_count() {
    static std::atomic<int> cached[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!cached[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

int make_rows_map(CUtensorMap* out, const void* base, int elem_bytes, unsigned long long rows, unsigned long long row_elems, const char* what,
                  int box_rows, int box_cols) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static std::atomic<Encode> resolved{nullptr};      // through the runtime: the library does not link against the driver
    Encode encode = resolved.load(std::memory_order_relaxed);
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) {
            (void)cudaGetLastError();
            snprintf(g_err, sizeof(g_err), "%s: the driver does not provide cuTensorMapEncodeTiled", what);
            return MKDA_ERR_LAUNCH;
        }
        encode = reinterpret_cast<Encode>(fn);
        resolved.store(encode, std::memory_order_relaxed);
    }
    const unsigned long long pitch = row_elems * (unsigned long long)elem_bytes;
    if ((reinterpret_cast<uintptr_t>(base) & 15) || (pitch & 15) || row_elems < 128 || rows == 0) {
        snprintf(g_err, sizeof(g_err), "%s: tensor not 16-byte aligned for tiled copies", what);
        return MKDA_ERR_ARG;
    }
    const cuuint64_t gdim[2] = {row_elems, rows};
    const cuuint64_t gstride[1] = {pitch};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, estr[2] = {1, 1};
    const CUresult r = encode(out, elem_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(base), gdim,
                              gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        snprintf(g_err, sizeof(g_err), "%s: cuTensorMapEncodeTiled failed (%d)", what, (int)r);
        return MKDA_ERR_LAUNCH;
    }
    return MKDA_OK;
}

int kernel_registers(const void* func) {
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, func) != cudaSuccess) { (void)cudaGetLastError(); return 0; }
    return a.numRegs;
}

int ensure_smem(const void* func, int bytes, const char* what) {
    // (function, device) pairs whose limit is already raised; a launcher asks before every launch.  Launches come from several threads: callers
    // that have released the GIL, and the autograd engine's thread of each device.
    struct Done { const void* func; int dev; int bytes; };
    static Done done[256];
    static int ndone = 0;
    static std::mutex mutex;
    int dev = 0;
    (void)cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mutex);
    for (int i = 0; i < ndone; ++i)
        if (done[i].func == func && done[i].dev == dev && done[i].bytes >= bytes) return MKDA_OK;
    cudaError_t e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) {
        snprintf(g_err, sizeof(g_err), "%s: cannot reserve %d bytes of shared memory: %s", what, bytes, cudaGetErrorString(e));
        (void)cudaGetLastError();
        return MKDA_ERR_LAUNCH;
    }
    if (ndone < 256) done[ndone++] = Done{func, dev, bytes};
    return MKDA_OK;
}

}  // namespace mkda

namespace mkda {
int selftest_status(unsigned int* out);
int selftest_status_clear();
}
extern "C" int mkda_device_status(void) {
    unsigned int f = 0, any = 0;
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    if (mkda::selftest_status(&f) == 0) any |= f;
    if (mkda::tc_chunk_status(&f) == 0) any |= f;
    if (mkda::tc_recur_status(&f) == 0) any |= f;
    if (mkda::tc_intra_status(&f) == 0) any |= f;
    if (mkda::tc_bwd_chunk_status(&f) == 0) any |= f;
    return (int)any;
}
extern "C" int mkda_device_status_clear(void) {
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    int rc = 0;
    rc |= mkda::selftest_status_clear();
    rc |= mkda::tc_chunk_status_clear();
    rc |= mkda::tc_recur_status_clear();
    rc |= mkda::tc_intra_status_clear();
    rc |= mkda::tc_bwd_chunk_status_clear();
    return rc;
}
extern "C" const char* mkda_last_error(void) { return mkda::g_err; }
extern "C" unsigned long long mkda_launch_count(void) { return mkda::g_launches.load(std::memory_order_relaxed); }
extern "C" int mkda_abi_version(void) { return 4; }
extern "C" int mkda_struct_sizes(int* out, int n) {
#define MKDA_SIZE(S) (int)sizeof(S),
    const int sizes[] = {MKDA_STRUCTS(MKDA_SIZE)};
    const int cnt = (int)(sizeof(sizes) / sizeof(sizes[0]));
    for (int i = 0; i < n && i < cnt; ++i) out[i] = sizes[i];
    return cnt;
}
