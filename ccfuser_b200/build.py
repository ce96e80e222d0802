"""Builds the CUDA library in-tree with nvcc for sm_100a (cross-compiles without a GPU).

``python -m ccfuser_b200.build`` or ``ccfuser_b200.build.build()``. The result is
``ccfuser_b200/lib/libccfuser_b200.so``; it is rebuilt only when a source is newer than it.
The reference builds a torch CUDAExtension against NVSHMEM and MPI with relocatable device code
(mix_moe/setup.py:108-196); this library has no dependency besides the CUDA runtime. Beside it lies a small Python
module with the autograd functions in C++, built with g++ against the installed torch and named after its version.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libccfuser_b200.so")
TORCH_SOURCES = [os.path.join(CSRC, f) for f in ("torch_norm.cpp", "norm.h")]
SOURCES = ["gemm.cu", "gemm2.cu", "gemm_swap.cu", "gemm_wgrad.cu", "moe_kernels.cu", "route.cu", "combine.cu", "router.cu", "runtime.cu",
           "no_alloc.cu", "norm.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; cannot build the sm_100a kernels")
    return nvcc


def sources():
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def needs_build() -> bool:
    """Whether the CUDA library is missing or older than a source."""
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))]
    return any(os.path.getmtime(d) > t for d in deps)


def torch_path() -> str:
    """The module of this torch and this Python: one built against others is never loaded."""
    import torch
    return os.path.join(LIB_DIR, f"_ccf_torch-{torch.__version__}-{sys.implementation.cache_tag}.so")


def needs_torch_module() -> bool:
    path = torch_path()
    return not os.path.exists(path) or any(os.path.getmtime(f) > os.path.getmtime(path) for f in TORCH_SOURCES)


def build(force: bool = False, verbose: bool = False) -> str:
    """The CUDA library and the torch module, where they are missing or stale."""
    if force or needs_build():
        build_library(verbose)
    if force or needs_torch_module():
        build_torch_module()
    return LIB_PATH


def build_library(verbose: bool = False) -> str:
    os.makedirs(LIB_DIR, exist_ok=True)
    objs = []
    obj_dir = os.path.join(HERE, "build")
    os.makedirs(obj_dir, exist_ok=True)
    procs = []
    for src in sources():
        obj = os.path.join(obj_dir, os.path.basename(src) + ".o")
        cmd = [_nvcc(), *NVCC_FLAGS, "-c", src, "-o", obj] + (["-Xptxas", "-v"] if verbose else [])
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for cmd, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode:
            sys.stderr.write(out)
        if p.returncode:
            raise RuntimeError("nvcc failed: " + " ".join(cmd))
    tmp = LIB_PATH + ".tmp"
    subprocess.check_call([_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", tmp, *objs, "-lcudart"])
    os.replace(tmp, LIB_PATH)
    return LIB_PATH


def build_torch_module() -> str:
    """``torch_path()``: a Python module against the installed torch, linked to the CUDA library beside it."""
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include"), sysconfig.get_paths()["include"]]
    path = torch_path()
    tmp = path + ".tmp"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared",
                           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                           *("-I" + i for i in inc), TORCH_SOURCES[0], "-o", tmp, "-L", LIB_DIR, "-lccfuser_b200", "-Wl,-rpath,$ORIGIN",
                           "-L", os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
                           "-ltorch_python"])
    os.replace(tmp, path)
    return path


def build_selftest() -> str:
    """Build ``lib/ccf_selftest``, the stand-alone C++ check of the library (csrc/selftest.cu: numerics against a CPU
    loop, throughput against cuBLAS). Not part of the default build: it links cuBLAS."""
    build()
    exe = os.path.join(LIB_DIR, "ccf_selftest")
    subprocess.check_call([_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                           os.path.join(CSRC, "selftest.cu"), "-o", exe, "-L", LIB_DIR, "-lccfuser_b200", "-lcublas",
                           "-Xlinker", "-rpath", "-Xlinker", "$ORIGIN"])
    return exe


if __name__ == "__main__":
    if "--selftest" in sys.argv:
        print(build_selftest())
    else:
        print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
