"""Build step: compiles libsarek_b200.so (CUDA, sm_100a only) and the extension _hostpath.so in-tree.

Run as ``python -m spoc_b200.build``.  nvcc cross-compiles without a GPU.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libsarek_b200.so")
HOSTPATH = os.path.join(HERE, "_hostpath.so")   # CPython extension: the marshalling half of run_vectors

SOURCES = ["sb200_shim.cu", "sb200_group.cu", "ir.cc", "fusion.cc", "map_jit.cc", "transfer.cc"]
HEADERS = ["gemm_tcgen05.cuh", "gemm_tcgen05_pair.cuh", "gemm_convert.cuh", "gemm_split.cuh", "map_fused.cuh",
           "ptx_sm100.cuh", "ir.hpp", "map_jit.hpp", "transfer.hpp", "internal.hpp",
           os.path.join("..", "..", "include", "sb200.h")]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden", "-shared", "-cudart", "static", "-ldl",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; libsarek_b200.so cannot be built")


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def build_library(force: bool = False, verbose: bool = False) -> str:
    build_hostpath(force)
    deps = [os.path.join(CSRC, s) for s in SOURCES + HEADERS] + [os.path.abspath(__file__)]
    if not force and not _stale(LIB, deps):
        return LIB
    cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB] + SOURCES
    res = subprocess.run(cmd, cwd=CSRC, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    if verbose:
        sys.stderr.write(res.stderr)
    return LIB


def build_hostpath(force: bool = False) -> str:
    src = os.path.join(CSRC, "hostpath.c")
    if not force and not _stale(HOSTPATH, [src, os.path.join(HERE, "..", "include", "sb200.h"), os.path.abspath(__file__)]):
        return HOSTPATH
    cmd = ["gcc", "-std=gnu11", "-O2", "-Wall", "-Wextra", "-fPIC", "-shared", "-I", sysconfig.get_paths()["include"], src, "-o", HOSTPATH]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("gcc failed:\n" + res.stdout + res.stderr)
    return HOSTPATH


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
