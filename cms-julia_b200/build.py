"""Builds the native libraries of the package in-tree.

lib/libpxl_b200.so   hand-written sm_100a CUDA kernels + the C ABI of include/pxl.h
lib/libpxlgen.so     seeded synthetic event generator (input synthesis)

Run as ``python cms-julia_b200/build.py`` or through ``__graft_entry__.build()``.
"""
from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "lib"
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]

# Kernels whose FP32 results compare bit-exactly with the reference, which never contracts
# a*b+c, build without FMA contraction. The track fits build with it: their FP64 results hold
# to a tolerance, a contracted product loses nothing, and the fits are bound by the length of
# their instruction stream. Their FP32 part rounds each operation by itself (bl::f32).
FMA_SOURCES = {"k_fit.cu", "k_adjoint.cu", "k_riemann.cu"}
CUDA_SOURCES = [
    "scan.cu",
    "workqueue.cu",
    "k_raw.cu",
    "k_cluster.cu",
    "k_rechits.cu",
    "k_ca.cu",
    "k_fit.cu",
    "k_adjoint.cu",
    "k_riemann.cu",
    "k_select.cu",
    "k_products.cu",
    "k_export.cu",
    "k_validate.cu",
    "noalloc.cu",
    "pipeline.cu",
]


def flags(source: str) -> list[str]:
    return [] if source in FMA_SOURCES else ["--fmad=false"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (Path(cand).exists() or cand == "nvcc"):
            return cand
    return "nvcc"


def _newer(target: Path, deps: list[Path]) -> bool:
    if not target.exists():
        return False
    t = target.stat().st_mtime
    return all(d.stat().st_mtime <= t for d in deps)


def build_cuda(force: bool = False, verbose: bool = False) -> Path:
    LIB.mkdir(exist_ok=True)
    out = LIB / "libpxl_b200.so"
    srcs = [CSRC / s for s in CUDA_SOURCES if (CSRC / s).exists()]
    # the headers, and this file, which decides the flags
    common = [*CSRC.glob("*.cuh"), *CSRC.glob("*.h"), PKG.parent / "include" / "pxl.h", Path(__file__)]
    if not force and _newer(out, srcs + common):
        return out
    objdir = PKG / "_build"
    objdir.mkdir(exist_ok=True)
    objs = []
    for s in srcs:
        o = objdir / (s.stem + ".o")
        if force or not _newer(o, [s, *common]):
            cmd = [_nvcc(), *ARCH, "-O3", "-lineinfo", "-std=c++17", *flags(s.name), "-Xcompiler", "-fPIC",
                   "-Xptxas", "-v" if verbose else "-O3", "-c", str(s), "-o", str(o)]
            if verbose:
                print(" ".join(cmd), flush=True)
            subprocess.run(cmd, check=True)
        objs.append(str(o))
    cmd = [_nvcc(), *ARCH, "-shared", "-o", str(out), *objs, "-lcudart"]
    subprocess.run(cmd, check=True)
    return out


def build_gen(force: bool = False) -> Path:
    LIB.mkdir(exist_ok=True)
    out = LIB / "libpxlgen.so"
    src = CSRC / "gen" / "pxlgen.cpp"
    if not force and _newer(out, [src]):
        return out
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(out), str(src), "-lpthread"], check=True)
    return out


def build_all(force: bool = False, verbose: bool = False) -> None:
    build_gen(force)
    build_cuda(force, verbose)


if __name__ == "__main__":
    build_all(force="--force" in sys.argv, verbose="-v" in sys.argv)
