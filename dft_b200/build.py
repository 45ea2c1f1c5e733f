"""Build libdft_b200.so in-tree with nvcc for sm_100a.

    python -m dft_b200.build            # incremental
    python -m dft_b200.build --force    # rebuild everything

Each source compiles to an object under dft_b200/_build/ and the objects link into
dft_b200/libdft_b200.so (the .so travels with the source tree; no JIT cache is used).
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libdft_b200.so")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-O2",
          "--expt-relaxed-constexpr", "-I", CSRC, "-I", INCLUDE]

# per-source extra flags: the radial solver replays the reference's sequential arithmetic,
# so it is compiled without FMA contraction
SOURCES = {
    "capi.cu": [],
    "grid_ops.cu": [],
    "jacobi_resident.cu": [],
    "mg_fused.cu": [],
    "davidson.cu": [],
    "dense_fp64.cu": [],
    "scf.cu": [],
    "radial.cu": ["-fmad=false"],
    "gram_tc.cu": [],
    "neural.cu": [],
    "poisson_start.cu": [],
    "precond_mg.cu": [],
    "atomic_start.cu": [],
    "autotune.cu": [],
    "zslab.cu": [],
    "eigh.cpp": ["-Xcompiler", "-O3"],
}


def nvcc() -> str:
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if c and os.path.exists(c):
            return c
    raise RuntimeError("nvcc not found")


def headers_mtime() -> float:
    m = 0.0
    for d in (CSRC, INCLUDE):
        for f in os.listdir(d):
            if f.endswith((".h", ".cuh", ".hpp")):
                m = max(m, os.path.getmtime(os.path.join(d, f)))
    return m


def build(force: bool = False, verbose: bool = False, ptxas_info: bool = False) -> str:
    os.makedirs(BUILD, exist_ok=True)
    nv = nvcc()
    hm = headers_mtime()
    objs = []
    for src, extra in SOURCES.items():
        s = os.path.join(CSRC, src)
        o = os.path.join(BUILD, src + ".o")
        objs.append(o)
        if not force and os.path.exists(o) and os.path.getmtime(o) >= max(os.path.getmtime(s), hm):
            continue
        cmd = [nv, *ARCH, *COMMON, *extra, "-c", s, "-o", o]
        if ptxas_info and src.endswith(".cu"):
            cmd.insert(1, "-Xptxas=-v")
        if verbose:
            print(" ".join(cmd), flush=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError(f"nvcc failed on {src}")
        if ptxas_info:
            sys.stderr.write(r.stderr)
    if force or not os.path.exists(LIB) or os.path.getmtime(LIB) < max(os.path.getmtime(o) for o in objs):
        cmd = [nv, *ARCH, "-shared", "-o", LIB, *objs, "-lcudart"]
        if verbose:
            print(" ".join(cmd), flush=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("-v", "--verbose", action="store_true")
    ap.add_argument("--ptxas-info", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose, a.ptxas_info))
