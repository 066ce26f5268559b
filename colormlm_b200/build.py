"""Builds libpolaris_s14_cuda.so (sm_100a only) next to this file with nvcc.

Run as ``python -m colormlm_b200.build``.  The library is built in-tree so that it
travels with the source tree; there is no JIT cache and no other architecture.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_NAME = "libpolaris_s14_cuda.so"
LIB_PATH = os.path.join(HERE, LIB_NAME)
SOURCES = ["s14_kernels.cu", "s14_router.cu", "s14_moe_umma.cu", "s14_moe_block.cu", "s14_moe_pair.cu", "s14_glue.cu", "s14_head.cu", "s14_fp8_expert.cu", "s14_api.cu", "s14_host.cpp"]
# the Python mirror's per-token calls, a CPython extension over the library (no CUDA, no torch headers)
PYCALL_SOURCE = "s14_pycall.cpp"
PYCALL_PATH = os.path.join(HERE, "_s14call.so")
HEADERS = ["s14_internal.h", "s14_device.cuh", "s14_router.cuh", "s14_umma.cuh", "s14_moe_block.cuh", "s14_host.hpp", os.path.join("..", "..", "include", "polaris_s14_cuda.h")]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA library cannot be built")


def _older(target: str, sources) -> bool:
    if not os.path.exists(target):
        return True
    built = os.path.getmtime(target)
    return any(os.path.getmtime(os.path.join(CSRC, d)) > built for d in sources)


def is_stale() -> bool:
    return _older(LIB_PATH, SOURCES + HEADERS)


def build_pycall(force: bool = False) -> str:
    """The extension links the library by name and finds it next to itself."""
    if force or _older(PYCALL_PATH, [PYCALL_SOURCE, HEADERS[-1]]):
        subprocess.run([
            shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-shared",
            "-I" + sysconfig.get_paths()["include"], "-o", PYCALL_PATH, os.path.join(CSRC, PYCALL_SOURCE),
            "-L" + HERE, "-l:" + LIB_NAME, "-Wl,-rpath,$ORIGIN",
        ], check=True)
    return PYCALL_PATH


def build(force: bool = False, verbose: bool = False) -> str:
    if force or is_stale():
        _build_library(verbose)
    build_pycall(force)
    return LIB_PATH


def _build_library(verbose: bool) -> None:
    cmd = [
        _nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
        "-shared", "-Xcompiler", "-fPIC,-fvisibility=hidden", "-ccbin", shutil.which("g++") or "g++",
        "-o", LIB_PATH,
    ]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += [os.path.join(CSRC, s) for s in SOURCES]
    subprocess.run(cmd, check=True)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
