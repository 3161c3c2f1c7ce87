"""Builds the sm_100a extension in-tree with plain nvcc (no torch headers: seconds per file).

Every ``csrc/*.cu`` is compiled to an object and linked into ``_lib/libmm_b200_ops.so``.  The
kernels expose a C ABI (raw pointers + a CUDA stream) and are called through ctypes, so the
library has no dependency on the PyTorch C++ ABI and can be loaded by any host program.

    python -m mindspeed_mm_b200.ops.build [--force] [--verbose]
"""
from __future__ import annotations

import hashlib
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIBDIR = os.path.join(HERE, "_lib")
LIBNAME = "libmm_b200_ops.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]
# Sources whose fp32 functions are the full ones: under --use_fast_math expf() is the fast exponential, whose relative error grows
# with its argument, and these replace PyTorch forms that had the full one.
FULL_MATH = ("gdn_prologue.cu",)


def _flags(src: str) -> list:
    return NVCC_FLAGS if src in FULL_MATH else [*NVCC_FLAGS, "--use_fast_math"]


def _nvcc() -> str:
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.isabs(c) and os.path.exists(c) or not os.path.isabs(c)):
            return c
    raise RuntimeError("nvcc not found")


def lib_path() -> str:
    return os.path.join(LIBDIR, LIBNAME)


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _digest() -> str:
    h = hashlib.sha256()
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h")):
            h.update(f.encode())
            h.update(open(os.path.join(CSRC, f), "rb").read())
            h.update(" ".join(_flags(f)).encode())
    return h.hexdigest()


def is_current() -> bool:
    stamp = os.path.join(LIBDIR, "build.stamp")
    return os.path.exists(lib_path()) and os.path.exists(stamp) and open(stamp).read().strip() == _digest()


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile (if sources changed) and return the path of the shared library."""
    if not force and is_current():
        return lib_path()
    os.makedirs(LIBDIR, exist_ok=True)
    nvcc = _nvcc()
    logs = {}

    def one(src):
        obj = os.path.join(LIBDIR, src[:-3] + ".o")
        cmd = [nvcc, *_flags(src), "-I", CSRC, "-c", os.path.join(CSRC, src), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        logs[src] = r.stdout + r.stderr
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        objs = list(ex.map(one, _sources()))
    cmd = [nvcc, "-shared", "-o", lib_path(), *objs, "-lcudart", "-Xcompiler", "-fPIC"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    with open(os.path.join(LIBDIR, "ptxas.log"), "w") as f:
        for k, v in logs.items():
            f.write(f"==== {k}\n{v}\n")
    with open(os.path.join(LIBDIR, "build.stamp"), "w") as f:
        f.write(_digest())
    if verbose:
        for k, v in logs.items():
            print(f"==== {k}\n{v}")
    return lib_path()


if __name__ == "__main__":
    p = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(p)
