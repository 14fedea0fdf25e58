"""Builds libqmcb200.so in-tree for sm_100a with nvcc (no JIT cache)."""
from __future__ import annotations

import os
import subprocess
import sys
import tempfile

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIBDIR = os.path.join(PKG, "lib")
LIB = os.path.join(LIBDIR, "libqmcb200.so")
SOURCES = ["qmcb200.cu", "sweep.cu", "invert.cu", "move.cu", "group.cu", "md.cu", "full.cu", "rows64.cu", "cusp_fit.c"]
HEADERS = ["device_common.cuh", "kernels.cuh", "kernels_population.cuh", "population.cuh", "kernels_md.cuh",
           "kernels_rows.cuh", "rows64_device.cuh", "group.h", "launches.h", "rows64.h", "sweep.h", "invert.h", "cusp_fit.h"]
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = [*ARCH_FLAGS, "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.isabs(c) and os.path.exists(c) or not os.path.isabs(c)):
            return c
    return "nvcc"


def stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS] + [os.path.join(ROOT, "include", "qmcb200.h")]
    return any(os.path.getmtime(p) > t for p in deps if os.path.exists(p))


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not stale():
        return LIB
    os.makedirs(LIBDIR, exist_ok=True)
    # the sources side by side: each takes up to two minutes
    with tempfile.TemporaryDirectory() as tmp:
        objects = [os.path.join(tmp, f + ".o") for f in SOURCES]
        jobs = []
        for f, o in zip(SOURCES, objects):
            cmd = [_nvcc(), *NVCC_FLAGS, "-c", "-o", o, os.path.join(CSRC, f)]
            if verbose:
                print(" ".join(cmd), file=sys.stderr)
            jobs.append((cmd, subprocess.Popen(cmd)))
        failed = [(cmd, job.returncode) for cmd, job in jobs if job.wait() != 0]
        if failed:
            raise subprocess.CalledProcessError(failed[0][1], failed[0][0])
        subprocess.check_call([_nvcc(), *ARCH_FLAGS, "-shared", "-o", LIB, *objects])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
