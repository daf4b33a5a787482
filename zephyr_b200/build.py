"""Build the in-tree CUDA library ``zephyr_b200/libzephyr_gpu.so`` for sm_100a.

Each translation unit is compiled with nvcc to an object, then linked into one
shared library.  The parity kernels are compiled with ``-fmad=false`` so that
no multiply is fused into an add (bit-exact with the reference's x86-64
build); the other kernels keep nvcc's default contraction.

Run ``python -m zephyr_b200.build`` (or ``__graft_entry__.build()``).
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
OUT = PKG / "libzephyr_gpu.so"
BUILD = PKG / "_build"

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-ffp-contract=off",
          "--expt-relaxed-constexpr"]

# translation unit -> extra flags
UNITS = {
    "zg_api.cu": [],
    "smf_parity.cu": ["-fmad=false"],
    "mmf_parity.cu": ["-fmad=false"],
    # the multi-material mixed form: FP32 face arithmetic with IEEE division
    # and square root and no fused multiply-adds.  With either, the HLLC
    # terms of two equal states no longer cancel exactly: spurious mass
    # fluxes of a few ulps in quiescent water (1e-6 in density after 500
    # steps) and a slower step.
    "mmf_mixed.cu": ["-fmad=false"],
    # allocation-free first-order step; its device-built coordinate tables
    # must match the host-built ones, hence no fused multiply-adds
    "zg_noalloc.cu": ["-fmad=false"],
    # AMR refine: geometry and distributed states bit-exact with the reference
    "amr_refine.cu": ["-fmad=false"],
    # scalar VOF transport: polygon clipping and sections bit-exact with the reference
    "tr_vof.cu": ["-fmad=false"],
    "zg_vtu.cu": [],
    "host_copy.cu": [],
    "smf_fast.cu": [],
    "smf_slot_fast.cu": [],
    "smf_slot_order.cu": [],
    "smf_slot_mixed.cu": ["-prec-div=false", "-prec-sqrt=false", "-ftz=true"],
    "adj.cu": [],
    # FP32 face arithmetic: approximate single-precision division and square
    # root; FP64 operations are unaffected by these flags.
    "smf_mixed.cu": ["-prec-div=false", "-prec-sqrt=false", "-ftz=true"],
}


def nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(exe).exists():
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build zephyr_b200")
    return exe


def _stale(target: Path, deps) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> Path:
    BUILD.mkdir(exist_ok=True)
    headers = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + [PKG.parent / "include" / "zephyr_gpu.h"]
    objs, todo = [], []
    for unit, extra in UNITS.items():
        src = CSRC / unit
        obj = BUILD / (unit + ".o")
        objs.append(obj)
        if force or _stale(obj, [src, *headers, Path(__file__)]):
            todo.append([nvcc(), *ARCH, *COMMON, *extra, "-c", str(src), "-o", str(obj)])

    def compile_unit(cmd):
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.run(cmd, check=True)

    # the units are independent: one compiler per core
    with ThreadPoolExecutor(max_workers=max(1, min(len(todo), os.cpu_count() or 1))) as pool:
        list(pool.map(compile_unit, todo))
    if force or _stale(OUT, objs):
        cmd = [nvcc(), *ARCH, "-shared", "-o", str(OUT), *map(str, objs), "-cudart", "static"]
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.run(cmd, check=True)
    return OUT


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
    print(OUT)
