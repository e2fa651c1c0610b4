"""Builds libgranite4_b200.so (the CUDA kernels + C ABI) in-tree with nvcc for sm_100a."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libgranite4_b200.so")

SOURCES = ["runtime.cu", "embed.cu", "add_rmsnorm.cu", "rope_kv.cu", "rope_bf16.cu", "swiglu.cu", "decode_glue.cu", "attn_decode.cu", "attn_prefill.cu", "attn_prefill_tc.cu", "gemm_fp8.cu", "kv_pool.cc", "kv_pool_controller.cc", "host_glue.cu"]
HEADERS = ["g4_host.h", "g4_math.cuh", "g4_tma.cuh", "g4_cluster.cuh", "g4_tcgen05.cuh"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared",
]


def _nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.isfile(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA extension cannot be built")


def dispatch_path() -> str:
    """The Python extension (csrc/py_dispatch.cc). It is compiled against one torch and one Python, whose
    versions its name carries: under another one there is no such file, and an extension built for a different
    C++ ABI is never loaded."""
    import torch
    return os.path.join(PKG_DIR, f"_dispatch-{sys.implementation.cache_tag}-torch{torch.__version__}.so")


def is_stale() -> bool:
    dispatch = dispatch_path()
    if not os.path.isfile(LIB_PATH) or not os.path.isfile(dispatch):
        return True
    built = min(os.path.getmtime(LIB_PATH), os.path.getmtime(dispatch))
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS + ["py_dispatch.cc"]]
    deps += [os.path.join(PKG_DIR, "..", "include", f) for f in ("granite4_b200.h", "granite4_b200.hpp")]
    return any(os.path.getmtime(d) > built for d in deps)


def _dispatch_cmd() -> list:
    """g++ command of the Python extension: host code only, against the torch that will load it."""
    import torch
    inc = os.path.join(os.path.dirname(torch.__file__), "include")
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-I" + inc, "-I" + os.path.join(inc, "torch", "csrc", "api", "include"),
            "-I" + sysconfig.get_paths()["include"],
            "-I" + os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include"),
            os.path.join(CSRC, "py_dispatch.cc"), "-o", dispatch_path(),
            "-L" + os.path.join(os.path.dirname(torch.__file__), "lib"), "-ltorch_python", "-ltorch", "-lc10", "-lc10_cuda"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every CUDA source into one shared library and the Python extension that calls it;
    returns the library's path."""
    if not force and not is_stale():
        return LIB_PATH
    cmd = [_nvcc(), *NVCC_FLAGS]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", LIB_PATH] + [os.path.join(CSRC, s) for s in SOURCES]
    side = subprocess.Popen(_dispatch_cmd(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    proc = subprocess.run(cmd, capture_output=True, text=True)
    said = side.communicate()[0]
    if proc.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + proc.stdout + proc.stderr)
    if side.returncode != 0:
        raise RuntimeError("g++ failed:\n" + said)
    if verbose:
        print(proc.stderr)
    return LIB_PATH
