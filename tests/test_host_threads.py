"""CPU: the library's host state under threads.  csrc/host.cu is compiled as plain C++ against a fake of the CUDA runtime, with the thread sanitizer
where the compiler has one."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include "host.cu"
#include <mutex>
#include <set>
#include <thread>
#include <vector>
static thread_local int device = 0;
static std::mutex fake_mutex;
static std::set<std::pair<const void*, int>> raised;
static CUresult fake_encode(CUtensorMap* m, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                            CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) { memset(m, 0, sizeof(*m)); return CUDA_SUCCESS; }
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { memset(a, 0, sizeof(*a)); return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int) {
    std::lock_guard<std::mutex> lock(fake_mutex);
    raised.insert({f, device});
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *fn = reinterpret_cast<void*>(fake_encode);
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}
namespace mkda {
int selftest_status(unsigned int*) { return 0; }
int selftest_status_clear() { return 0; }
int tc_chunk_status(unsigned int*) { return 0; }
int tc_chunk_status_clear() { return 0; }
int tc_recur_status(unsigned int*) { return 0; }
int tc_recur_status_clear() { return 0; }
int tc_intra_status(unsigned int*) { return 0; }
int tc_intra_status_clear() { return 0; }
int tc_bwd_chunk_status(unsigned int*) { return 0; }
int tc_bwd_chunk_status_clear() { return 0; }
}
static char kernels[40], tensor[16] __attribute__((aligned(16)));
int main() {
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([t] {
            device = t % 4;
            CUtensorMap map;
            for (int r = 0; r < 50; ++r)
                for (char& k : kernels)
                    if (mkda::ensure_smem(&k, 1000, "k") || mkda::sm_count() != 148 || mkda::make_rows_map(&map, tensor, 2, 64, 128, "m")) _Exit(2);
        });
    for (std::thread& t : threads) t.join();
    return raised.size() == 4 * sizeof(kernels) ? 0 : 3;          // every pair that was called ready has been raised
}
"""


def test_launches_from_several_threads(tmp_path):
    cxx, nvcc = shutil.which("g++"), shutil.which("nvcc")
    if not cxx or not nvcc:
        pytest.skip("needs g++ and the CUDA headers")
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    src, exe = tmp_path / "threads.cpp", tmp_path / "threads"
    src.write_text(HARNESS)
    base = [cxx, "-std=c++17", "-O1", "-g", "-pthread", "-I", os.path.join(ROOT, "mogankda_b200", "csrc"), "-I", include, str(src), "-o", str(exe)]
    if subprocess.run([*base, "-fsanitize=thread"], capture_output=True).returncode:
        subprocess.run(base, check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[:3000]
