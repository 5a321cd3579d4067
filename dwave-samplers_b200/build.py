"""Builds libb200sa.so (the sm_100a CUDA kernels plus the C ABI) in-tree.

    python dwave-samplers_b200/build.py [--force]

nvcc cross-compiles for sm_100a without a GPU.  The library links the CUDA
runtime statically and exports only the C ABI declared in include/b200sa.h.
"""
from __future__ import annotations

import argparse
import glob
import hashlib
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(ROOT, "include")
OUT = os.path.join(HERE, "b200sa", "libb200sa.so")

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC,-O3,-fvisibility=hidden",
         "-Xptxas", "-v", "--expt-relaxed-constexpr"]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cpp")))


def stale() -> bool:
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh"))
    deps += glob.glob(os.path.join(INCLUDE, "*.h")) + [__file__]
    return any(os.path.getmtime(d) > t for d in deps)


def digest() -> str:
    """Of the sources: part of the tuning cache's keys."""
    h = hashlib.sha256()
    for f in sorted(glob.glob(os.path.join(CSRC, "*"))):
        h.update(open(f, "rb").read())
    return h.hexdigest()[:12]


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not stale():
        return OUT
    tmp = OUT + ".tmp"
    cmd = [nvcc(), *ARCH, *FLAGS, f'-DB200SA_SOURCES="{digest()}"', "-shared", "-cudart", "static", "-I", INCLUDE, "-I", CSRC,
           *sources(), "-o", tmp]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("nvcc failed building libb200sa.so")
    if verbose:
        sys.stderr.write(res.stderr)
    os.replace(tmp, OUT)
    return OUT


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("-v", "--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
