"""Builds libmkda.so (the C-ABI kernel library) with nvcc for sm_100a and _host.so (the native host path over it, a torch
extension module) in-tree.

    python -m mogankda_b200.build [--force] [-v]

Objects are cached under ``build/`` and recompiled only when their source or a header is newer.
"""
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
SOURCES = ("host.cu", "entry.cu", "prologue.cu", "combine.cu", "step.cu", "selftest.cu", "tc_chunk.cu", "tc_recur.cu", "tc_intra.cu", "tc_bwd_chunk.cu")
HOST_SOURCES = ("layer.cpp", "binding.cpp")
CXX_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-w"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
              "-Wno-deprecated-gpu-targets"]


def lib_path():
    return os.path.join(HERE, "libmkda.so")


def _newer(target, deps):
    if not os.path.exists(target):
        return False
    t = os.path.getmtime(target)
    return all(os.path.getmtime(d) <= t for d in deps)


def build(force=False, verbose=False):
    """Compiles (only what is stale) and links; returns the library path."""
    nvcc = os.environ.get("NVCC", "nvcc")
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    headers.append(os.path.join(HERE, "..", "include", "mkda.h"))
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    jobs, objs = [], []
    for src in SOURCES:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        objs.append(obj)
        path = os.path.join(CSRC, src)
        if not force and _newer(obj, [path, *headers]):
            continue
        cmd = [nvcc, *NVCC_FLAGS, "-c", path, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        jobs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    # the host sources need torch's headers, found without importing torch
    torch_dir = os.path.dirname(importlib.util.find_spec("torch").origin)
    cuda_inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(nvcc) or nvcc))), "include")
    incs = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"), cuda_inc,
            sysconfig.get_paths()["include"]]
    cxx = os.environ.get("CXX", "g++")
    host_jobs, host_objs = [], []
    for src in HOST_SOURCES:
        obj = os.path.join(objdir, src.replace(".cpp", ".o"))
        host_objs.append(obj)
        path = os.path.join(CSRC, src)
        if force or not _newer(obj, [path, *headers]):
            cmd = [cxx, *CXX_FLAGS, *("-isystem" + i for i in incs), "-c", path, "-o", obj]
            host_jobs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, pr in jobs:
        log, _ = pr.communicate()
        if pr.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{log}")
        if verbose:
            print(log)
    out = lib_path()
    if force or jobs or not _newer(out, objs):
        subprocess.check_call([nvcc, "-shared", "-Wno-deprecated-gpu-targets", "-Xlinker", "-soname=libmkda.so", "-o", out, *objs])
    for src, pr in host_jobs:
        log, _ = pr.communicate()
        if pr.returncode != 0:
            raise RuntimeError(f"{cxx} failed on {src}:\n{log}")
    host = os.path.join(HERE, "_host.so")
    if force or host_jobs or not _newer(host, [*host_objs, out]):
        torch_lib = os.path.join(torch_dir, "lib")
        # The C++ runtime that torch has loaded, by name: a compiler that brings only an archive of it would put a second copy into the module,
        # whose streams have no locale (the first number in an error message ended the process)
        subprocess.check_call([cxx, "-shared", "-o", host, *host_objs, "-L" + HERE, "-lmkda", "-L" + torch_lib, "-lc10", "-lc10_cuda", "-ltorch_cpu",
                               "-ltorch_cuda", "-ltorch", "-ltorch_python", "-l:libstdc++.so.6", "-Wl,-rpath,$ORIGIN", "-Wl,-rpath," + torch_lib])
    return out


def main(argv):
    print(build(force="--force" in argv, verbose="-v" in argv))


if __name__ == "__main__":
    main(sys.argv[1:])
