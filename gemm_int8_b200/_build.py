"""Builds libgemm_int8_b200.so in-tree with nvcc for sm_100a (no libtorch, no CUTLASS), and libgemm_int8_b200_torch.so, the
torch operators over it, with g++ against the installed torch.

Replaces the reference's CMake/ninja build of gemm_int8_CUDA.so (CMakeLists.txt, build.sh): one
translation unit, one nvcc command, a few seconds.
"""
from __future__ import annotations

import os
import shutil
import subprocess

_PKG = os.path.dirname(os.path.abspath(__file__))
LIB_NAME = "libgemm_int8_b200.so"
LIB_PATH = os.path.join(_PKG, LIB_NAME)
SOURCES = [os.path.join(_PKG, "csrc", "api.cu")]
HEADERS = [os.path.join(_PKG, "csrc", f) for f in ("ptx.cuh", "k_dense.cuh", "k_dense_splitk.cuh", "k_blockwise.cuh", "k_blockwise_smallm.cuh", "k_smallm.cuh", "k_quant.cuh")]
HEADERS.append(os.path.join(os.path.dirname(_PKG), "include", "gemm_int8_b200.h"))

OPS_NAME = "libgemm_int8_b200_torch.so"
OPS_PATH = os.path.join(_PKG, OPS_NAME)
OPS_SOURCE = os.path.join(_PKG, "csrc", "torch_ops.cpp")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; cannot build " + LIB_NAME)
    return cand


def _stale(target: str, sources: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.exists(f) and os.path.getmtime(f) > t for f in sources)


def _ops_tag() -> str:
    """What the operator library is tied to besides its sources: it is compiled against one torch and one Python ABI."""
    import sysconfig

    import torch

    return f"torch {torch.__version__} abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)} {sysconfig.get_config_var('SOABI')}"


def _built_for_other_torch() -> bool:
    with open(OPS_PATH, "rb") as f:
        return _ops_tag().encode() + b"\0" not in f.read()  # gi8_torch_ops_built_for of torch_ops.cpp


def _ops_stale() -> bool:
    return _stale(OPS_PATH, [OPS_SOURCE, HEADERS[-1]]) or _built_for_other_torch()


def is_stale() -> bool:
    return _stale(LIB_PATH, SOURCES + HEADERS) or _ops_stale()


def _run(cmd: list[str], verbose: bool) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(os.path.basename(cmd[0]) + " failed:\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stderr)


def _build_ops(verbose: bool) -> None:
    import sysconfig

    import torch

    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    _run([shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", *(f"-I{d}" for d in include),
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DGI8_BUILT_FOR="{_ops_tag()}"', "-o", OPS_PATH, OPS_SOURCE,
          f"-L{os.path.join(root, 'lib')}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch",
          f"-L{_PKG}", f"-l:{LIB_NAME}", "-Wl,-rpath,$ORIGIN"], verbose)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile both libraries if they are missing or older than their sources, the operators also if the installed torch or
    Python is another one; returns the path of the first."""
    if force or _stale(LIB_PATH, SOURCES + HEADERS):
        _run([_nvcc(), *(["-Xptxas", "-v"] if verbose else []), *NVCC_FLAGS, "-o", LIB_PATH, *SOURCES], verbose)
    if force or _ops_stale():
        _build_ops(verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force=True, verbose=True))
