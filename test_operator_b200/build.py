"""Builds the C-ABI shared library (hand-written sm_100a kernels) in-tree with nvcc, and the host module of the operator calls.

    python -m test_operator_b200.build          # build if sources are newer than the library
    python -m test_operator_b200.build --force
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
ROOT = os.path.dirname(PKG)
LIB_DIR = os.path.join(PKG, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libsmla_bwd.so")

HOST_SOURCE = os.path.join(CSRC, "smla_host.cpp")
HOST_PATH = os.path.join(LIB_DIR, "_smla_host.so")

SOURCES = ["smla_api.cu"]
HEADERS = ["sm100_ptx.cuh", "smla_kernels.cuh", "smla_index_inverse.cuh"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-shared",
    "-Xptxas", "-v",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found: the CUDA kernels cannot be built")
    return cand


def needs_build() -> bool:
    return _older(LIB_PATH, [os.path.join(CSRC, f) for f in SOURCES + HEADERS])


def host_needs_build() -> bool:
    return _older(HOST_PATH, [HOST_SOURCE])


def _older(path: str, sources) -> bool:
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    return any(os.path.getmtime(d) > t for d in [*sources, os.path.join(ROOT, "include", "smla_bwd.h")])


def build(force: bool = False, verbose: bool = False) -> str:
    if force or needs_build():
        _run([_nvcc()] + NVCC_FLAGS + [os.path.join(CSRC, s) for s in SOURCES] + ["-o", LIB_PATH], "build.log", verbose)
    if force or host_needs_build():
        build_host(verbose)
    return LIB_PATH


def build_host(verbose: bool = False) -> str:
    """The CPython module of csrc/smla_host.cpp (no kernels in it): the host compiler against torch's headers."""
    import sysconfig

    from torch.utils import cpp_extension
    cuda_home = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [sysconfig.get_paths()["include"], os.path.join(cuda_home, "include"), *cpp_extension.include_paths()]
    cmd = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-shared", "-fPIC", *(f"-I{d}" for d in inc), HOST_SOURCE, "-o", HOST_PATH,
           *(f"-L{d}" for d in cpp_extension.library_paths()), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]
    _run(cmd, "build_host.log", verbose)
    return HOST_PATH


def _run(cmd, log_name: str, verbose: bool) -> None:
    os.makedirs(LIB_DIR, exist_ok=True)
    res = subprocess.run(cmd, capture_output=True, text=True)
    log = res.stdout + res.stderr
    with open(os.path.join(LIB_DIR, log_name), "w") as f:
        f.write(" ".join(cmd) + "\n" + log)
    if res.returncode != 0:
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed:\n" + log[-4000:])
    if verbose:
        print(log)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
