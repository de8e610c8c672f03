"""Builds libgfcuda.so (the CUDA engine and its C ABI) in-tree for sm_100a.

Usage: python -m genefer22_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libgfcuda.so")
INSTANCES = [f"gf_inst_{g}.cu" for g in ("small", "cluster_short", "cluster_long", "col", "colr", "row", "row_pair", "mid", "pcol")]
SOURCES = [os.path.join(CSRC, f) for f in ("gf_host.cu", "gf_probe.cu", *INSTANCES, "gf_gint.cpp", "gf_server.cpp",
                                           "gf_server_cuda.cpp")]
DEPS = SOURCES + [os.path.join(CSRC, f) for f in ("gf_arith.cuh", "gf_ntt.cuh", "gf_kernels.cuh", "gf_inst.cuh", "gf_server.h")] + \
    [os.path.join(ROOT, "include", "gfcuda.h")]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden",
    "-shared",
    "--threads", "0",       # the sources in parallel
    "-static-global-template-stub=false",   # kernel templates instantiated in one file, launched from another
]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def up_to_date() -> bool:
    if not os.path.exists(LIB):
        return False
    t = os.path.getmtime(LIB)
    return all(os.path.getmtime(d) <= t for d in DEPS)


def build(force: bool = False, verbose: bool = False, extra: list[str] | None = None) -> str:
    if not force and up_to_date():
        return LIB
    cmd = [nvcc(), *NVCC_FLAGS, *(extra or []), "-cudart=static", "-o", LIB + ".tmp", *SOURCES]
    if verbose:
        print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError(f"nvcc failed ({r.returncode})")
    if verbose and (r.stdout or r.stderr):
        sys.stderr.write(r.stdout + r.stderr)
    os.replace(LIB + ".tmp", LIB)
    return LIB


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    ap.add_argument("--ptxas-v", action="store_true", help="print register/smem usage per kernel")
    a = ap.parse_args()
    extra = ["-Xptxas", "-v"] if a.ptxas_v else []
    print(build(force=a.force or a.ptxas_v, verbose=a.verbose or a.ptxas_v, extra=extra))


if __name__ == "__main__":
    main()
