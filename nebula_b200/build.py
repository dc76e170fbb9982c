"""Builds the CUDA library in-tree with nvcc for sm_100a.

    python -m nebula_b200.build [--force]

Produces ``nebula_b200/lib/libnebula_b200.so`` (the C ABI declared in
``include/nebula_b200.h``).  nvcc cross-compiles without a GPU.
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIBDIR = PKG / "lib"
LIB = LIBDIR / "libnebula_b200.so"
# (source, object name, extra flags)
SOURCES = [(s, s, []) for s in ("api.cu", "network.cu", "plans.cu", "elementwise.cu", "gemm_simt.cu", "gemm_tcgen05.cu", "static_scratch.cu",
                                "arena.cu", "lstm_persistent.cu", "lstm_wide.cu", "recurrent_cluster.cu")]
# the CUDA-core contraction, a module per pair of copy modes (gemm_simt.cuh)
SOURCES += [("gemm_simt_kernels.cu", f"gemm_simt_kernels_{a}{b}", [f"-DNB_SIMT_A={a}", f"-DNB_SIMT_B={b}"]) for a in range(3) for b in range(3)]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _deps_mtime() -> float:
    files = list(CSRC.glob("*")) + [PKG.parent / "include" / "nebula_b200.h"]
    return max(f.stat().st_mtime for f in files)


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and LIB.exists() and LIB.stat().st_mtime >= _deps_mtime():
        return LIB
    LIBDIR.mkdir(exist_ok=True)
    objdir = LIBDIR / "obj"
    objdir.mkdir(exist_ok=True)
    nvcc = _nvcc()

    def compile_one(item):
        src, name, flags = item
        obj = objdir / (name + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *flags, "-c", str(CSRC / src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        (objdir / (name + ".log")).write_text(r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stderr[-4000:]}")
        if verbose:
            print(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(6, os.cpu_count() or 1)) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stderr[-4000:]}")
    return LIB


if __name__ == "__main__":
    p = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(p)
