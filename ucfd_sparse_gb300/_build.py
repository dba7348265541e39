"""Compile libucfd_gb300.so (the C-ABI library) in-tree for sm_103a.

Translation units are compiled in parallel with nvcc and linked into
``ucfd_sparse_gb300/lib/libucfd_gb300.so``; objects go to
``ucfd_sparse_gb300/_build/``.  ``kern_exact.cu`` is compiled with
``-fmad=false`` (the bit-exact FP64 mode), everything else with default
contraction.  A rebuild happens only when a source or header is newer than
the library.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INC = os.path.join(os.path.dirname(HERE), "include")
BUILD = os.path.join(HERE, "_build")
LIBDIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIBDIR, "libucfd_gb300.so")

ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
COMMON = ["-O3", "-std=c++20", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
          "-I", CSRC, "-I", INC]

# (source, extra flags)
UNITS = [
    ("kern_exact.cu", ["-fmad=false"]),
    ("kern_fast.cu", []),
    ("kern_gm.cu", []),
    ("runtime.cpp", []),
    ("graph.cpp", []),
    ("flowsys.cpp", []),
    ("legacy.cpp", []),
    ("krylov.cpp", []),
    ("noalloc.cu", []),
    ("selftest.cu", []),
    ("adjoint.cpp", []),
]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _deps_mtime() -> float:
    m = 0.0
    for d in (CSRC, INC):
        for f in os.listdir(d):
            m = max(m, os.path.getmtime(os.path.join(d, f)))
    return max(m, os.path.getmtime(__file__))


def up_to_date() -> bool:
    return os.path.exists(LIB) and os.path.getmtime(LIB) >= _deps_mtime()


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and up_to_date():
        return LIB
    os.makedirs(BUILD, exist_ok=True)
    os.makedirs(LIBDIR, exist_ok=True)
    cc = nvcc()

    def compile_one(unit):
        src, extra = unit
        obj = os.path.join(BUILD, os.path.splitext(src)[0] + ".o")
        # the kernel units: optimised in parallel parts (halves the longest unit's build time)
        split = ["--split-compile=0"] if src.endswith(".cu") else []
        cmd = [cc, *ARCH, *COMMON, *split, *extra, "-c", os.path.join(CSRC, src), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{' '.join(cmd)}\n{r.stdout}\n{r.stderr}")
        if verbose and (r.stdout or r.stderr):
            print(r.stdout + r.stderr, file=sys.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(len(UNITS), os.cpu_count() or 4)) as ex:
        objs = list(ex.map(compile_one, UNITS))
    tmp = LIB + ".tmp"
    cmd = [cc, *ARCH, "-shared", "-o", tmp, *objs, "-Xlinker", "--no-undefined"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{' '.join(cmd)}\n{r.stdout}\n{r.stderr}")
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
