"""Build libbaandi_b200.so in-tree for sm_100a (B200) with nvcc.

`python -m baandi_b200.build` compiles every CUDA/C++ source under csrc/ into one
shared library next to this file.  The host compiler keeps every multiply and add
separately rounded (-ffp-contract=off) because the basis sort depends on exact |G|^2.
"""
from __future__ import annotations

import os
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libbaandi_b200.so")
SOURCES = ["api.cu", "hpsi_kernels.cu", "planes_any.cu", "davidson.cu", "noalloc.cu", "fields.cu", "kset_davidson.cu", "mixer.cu",
           "learned.cu", "gemm_tc.cu", "gemm_rns.cu", "setup.cpp"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-ffp-contract=off,-O3,-fopenmp",
    "-Xptxas", "-v",
]


def nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    for root, _, files in os.walk(CSRC):
        for f in files:
            if os.path.getmtime(os.path.join(root, f)) > t:
                return True
    inc = os.path.join(HERE, "..", "include")
    return os.path.isdir(inc) and any(os.path.getmtime(os.path.join(inc, f)) > t for f in os.listdir(inc))


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not stale():
        return LIB
    tmp = LIB + ".tmp"
    with tempfile.TemporaryDirectory() as work, ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
        objects = [os.path.join(work, s + ".o") for s in SOURCES]

        def compile_one(args):
            src, obj = args
            return subprocess.run([nvcc(), *NVCC_FLAGS, "-c", "-o", obj, os.path.join(CSRC, src)], capture_output=True,
                                  text=True)
        done = list(pool.map(compile_one, zip(SOURCES, objects)))
        if all(r.returncode == 0 for r in done):
            done.append(subprocess.run([nvcc(), *NVCC_FLAGS, "-shared", "-o", tmp, *objects, "-lcudart", "-lgomp"],
                                       capture_output=True, text=True))
    if any(r.returncode != 0 for r in done):
        sys.stderr.write("".join(r.stdout + r.stderr for r in done if r.returncode != 0))
        raise RuntimeError("nvcc failed building libbaandi_b200.so")
    if verbose:
        sys.stderr.write("".join(r.stderr for r in done))
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
