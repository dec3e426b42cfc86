"""Builds the in-tree CUDA library implexity_b200/liblbm_b200.so for sm_100a.

Run as ``python -m implexity_b200.build`` (or through ``__graft_entry__.build``).
nvcc cross-compiles without a GPU; the objects are rebuilt only when a
source or header is newer than the library.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
INCLUDE = PKG.parent / "include"
BUILD = PKG / "_build"
LIB = PKG / "liblbm_b200.so"
MMA_LIB = PKG / "libmma_cpu.so"
MMA_SOURCE = CSRC / "mma_cpu.cpp"

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"]
SOURCES = ["lbm_forward.cu", "lbm_adjoint.cu", "lbm_march.cu", "lbm_misc.cu", "lbm_io.cu", "lbm_noalloc.cu",
           "lbm_runtime.cpp"]
# The stepping kernels' instances compile as one unit per lattice and collision
# (LBM_PART: 10 * lattice + CollKind), in parallel with the rest.  (nvcc's own
# --split-compile makes them spill: 0 -> 108 bytes in the FP32 forward step,
# which then takes 149 instead of 124 us at 256x128x128.)
PARTS = {"lbm_forward.cu": [190, 191, 192, 270, 271, 272], "lbm_adjoint.cu": [190, 191, 192, 270, 271, 272],
         "lbm_march.cu": [190, 192, 270, 272]}
UNITS = [(src, part) for part in (191, 271, 190, 270, 192, 272, None) for src in SOURCES
         if part is None or part in PARTS.get(src, ())]
UNITS.sort(key=lambda u: u[0] != "lbm_misc.cu")  # the longest one first


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found: the CUDA toolkit is required to build liblbm_b200.so")


def _inputs() -> list[Path]:
    files = [CSRC / s for s in SOURCES]
    files += sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h")) + sorted(INCLUDE.glob("*.h"))
    return files


def up_to_date() -> bool:
    if not LIB.exists():
        return False
    t = LIB.stat().st_mtime
    return all(f.stat().st_mtime <= t for f in _inputs())


def host_cxx() -> str:
    """A host C++ compiler with OpenMP (the distribution g++ first)."""
    for cand in (os.environ.get("MMA_CXX"), "/usr/bin/g++", shutil.which("g++")):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("g++ not found: a host C++ compiler with OpenMP is required to build libmma_cpu.so")


def build_mma(force: bool = False, verbose: bool = False) -> Path:
    """The host MMA library (include/mma_cpu.h): C++17 with OpenMP."""
    deps = [MMA_SOURCE, INCLUDE / "mma_cpu.h"]
    if not force and MMA_LIB.exists() and all(d.stat().st_mtime <= MMA_LIB.stat().st_mtime for d in deps):
        return MMA_LIB
    tmp = MMA_LIB.with_suffix(".so.tmp")
    cmd = [host_cxx(), "-O3", "-std=c++17", "-fopenmp", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall",
           "-o", str(tmp), str(MMA_SOURCE)]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    os.replace(tmp, MMA_LIB)
    return MMA_LIB


def build(force: bool = False, verbose: bool = False) -> Path:
    build_mma(force, verbose)
    if not force and up_to_date():
        return LIB
    BUILD.mkdir(exist_ok=True)
    cc = nvcc()

    headers = sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h")) + sorted(INCLUDE.glob("*.h"))

    def compile_one(unit: tuple[str, int | None]) -> Path:
        src, part = unit
        obj = BUILD / (src + (".o" if part is None else f".{part}.o"))
        deps = [CSRC / src, *headers]
        if not force and obj.exists() and all(d.stat().st_mtime <= obj.stat().st_mtime for d in deps):
            return obj
        define = [] if part is None else [f"-DLBM_PART={part}"]
        cmd = [cc, *ARCH, *FLAGS, *define, "-c", str(CSRC / src), "-o", str(obj)]
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.run(cmd, check=True)
        return obj

    with ThreadPoolExecutor(max_workers=max(2, os.cpu_count() or 2)) as ex:
        objs = list(ex.map(compile_one, UNITS))
    tmp = LIB.with_suffix(".so.tmp")
    cmd = [cc, *ARCH, "-shared", "-o", str(tmp), *map(str, objs)]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
    print(LIB)
