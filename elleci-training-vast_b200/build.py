"""Builds libelleci_int2.so (the C-ABI CUDA library) in-tree for sm_100a with nvcc, and elleci_host_ops.so (the operators' host
side, against the installed torch) with the C++ compiler.

    python elleci-training-vast_b200/build.py [--force]

The outputs, lib/libelleci_int2.so and lib/elleci_host_ops.<python>.torch-<version>.so, are git-ignored; they are rebuilt when a
source file is newer, and the second one when Python or torch is another one.
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libelleci_int2.so")
SOURCES = ["api.cu", "pack_quant.cu", "hysteresis.cu", "gemm_simple.cu", "gemm_skinny.cu", "tensor_maps.cu", "gemm_dw.cu", "gemm_wt.cu", "decode_static.cu", "gemv_small.cu", "gemv_mma.cu", "rmsnorm.cu", "swiglu.cu", "peer_sync.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-fmad=false",                       # the integer state must not depend on fused multiply-adds
    "-Xcompiler", "-fPIC,-fvisibility=hidden",
]


def host_path() -> str:
    """The extension module of csrc/host_ops.cpp for the running Python and torch.  It is compiled against their headers and holds for
    no other version, so its name carries both: after an upgrade the file is missing (and built again), not loaded and wrong."""
    import torch
    return os.path.join(LIB_DIR, f"elleci_host_ops.{sys.implementation.cache_tag}.torch-{torch.__version__}.so")


def _nvcc() -> str:
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _stale() -> bool:
    if not os.path.exists(LIB_PATH) or not os.path.exists(host_path()):
        return True
    t = min(os.path.getmtime(LIB_PATH), os.path.getmtime(host_path()))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(HERE, "..", "include", "elleci_int2.h"),
                                                                 os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    obj_dir = os.path.join(LIB_DIR, "obj")
    os.makedirs(obj_dir, exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: str) -> str:
        obj = os.path.join(obj_dir, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-c", os.path.join(CSRC, src), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    cmd = [nvcc, "-shared", "-o", LIB_PATH, *objs, "-cudart", "static"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stderr}")
    build_host_ops()
    return LIB_PATH


def build_host_ops() -> str:
    """The extension module of csrc/host_ops.cpp: host code against the installed torch's headers, no CUDA code."""
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f"-I{root}/include",
           f"-I{root}/include/torch/csrc/api/include", f"-I{sysconfig.get_paths()['include']}", f"-I{cuda}/include",
           os.path.join(CSRC, "host_ops.cpp"), "-o", host_path(), f"-L{root}/lib", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch",
           "-ltorch_python", "-ldl"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"building host_ops.cpp failed:\n{r.stderr}")
    return host_path()


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
