"""Builds the C-ABI shared library (hand-written sm_100a kernels) in-tree with nvcc, and the host module of the operator calls.

    python -m test_operator_b200.build          # build if sources are newer than the library
    python -m test_operator_b200.build --force
"""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
ROOT = os.path.dirname(PKG)
LIB_DIR = os.path.join(PKG, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libsmla_bwd.so")

HOST_SOURCE = os.path.join(CSRC, "smla_host.cpp")
HOST_HEADER = os.path.join(ROOT, "include", "smla_bwd.h")
HOST_DELTA = os.path.join(CSRC, "smla_host_delta.h")

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
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS] + [os.path.join(ROOT, "include", "smla_bwd.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def host_path() -> str:
    """Where the host module for this interpreter, this torch and these sources lies.  All of them are in its name: it goes by torch's
    C++ interface and by the structs of the C header, so one that was built for others must not be loaded."""
    import torch
    tag = hashlib.sha256(torch.__version__.encode())
    for path in (HOST_SOURCE, HOST_HEADER, HOST_DELTA):
        with open(path, "rb") as f:
            tag.update(f.read())
    return os.path.join(LIB_DIR, "_smla_host." + tag.hexdigest()[:16] + sysconfig.get_config_var("EXT_SUFFIX"))


def build(force: bool = False, verbose: bool = False) -> str:
    if force or needs_build():
        _compile([_nvcc()] + NVCC_FLAGS + [os.path.join(CSRC, s) for s in SOURCES], LIB_PATH, "build.log", verbose)
    if force or not os.path.exists(host_path()):
        build_host(verbose)
    return LIB_PATH


def build_host(verbose: bool = False) -> str:
    """The CPython module of csrc/smla_host.cpp (no kernels in it): the host compiler against torch's headers."""
    from torch.utils import cpp_extension
    path = host_path()
    cuda_home = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [sysconfig.get_paths()["include"], os.path.join(cuda_home, "include"), *cpp_extension.include_paths()]
    _compile([shutil.which("g++") or "c++", "-O2", "-std=c++17", "-shared", "-fPIC", *(f"-I{d}" for d in inc), HOST_SOURCE,
              *(f"-L{d}" for d in cpp_extension.library_paths()), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"], path,
             "build_host.log", verbose)
    return path


def _compile(cmd, path: str, log_name: str, verbose: bool) -> None:
    """Runs the compiler.  `path` shows up when the file is whole: ranks that start together may all build it, and load it meanwhile."""
    os.makedirs(LIB_DIR, exist_ok=True)
    part = f"{path}.{os.getpid()}.part"
    cmd = [*cmd, "-o", part]
    try:
        res = subprocess.run(cmd, capture_output=True, text=True)
        log = res.stdout + res.stderr
        with open(os.path.join(LIB_DIR, log_name), "w") as f:
            f.write(" ".join(cmd) + "\n" + log)
        if res.returncode != 0:
            raise RuntimeError(f"{os.path.basename(cmd[0])} failed:\n" + log[-4000:])
        os.replace(part, path)
    finally:
        if os.path.exists(part):
            os.remove(part)
    if verbose:
        print(log)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
