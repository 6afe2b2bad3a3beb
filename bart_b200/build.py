"""Build the sm_100a shared library ``bart_b200/lib/libbnufft.so`` in-tree.

``python -m bart_b200.build`` (or ``build()``) runs nvcc directly; the
library has a plain C ABI (include/bnufft.h, include/bespirit.h) and links only the CUDA
runtime; the ESPIRiT calibration loads cuSOLVER on first use. The FFT pass
kernels compile in several translation units at once.
"""

from __future__ import annotations

import os
import subprocess
import sys
import tempfile
import zlib
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "lib", "libbnufft.so")
# objects: outside the tree, one folder per checkout and user
OBJ = os.path.join(tempfile.gettempdir(), f"bnufft_build_{os.getuid()}_{zlib.crc32(HERE.encode()):08x}")
PASS_GROUPS = 7     # groups of FFT lengths (csrc/passes.cuh), one translation unit each
# object -> (source, extra flags, headers it depends on; None: all)
PASS_HEADERS = ("fft_core.cuh", "fft_passes.cuh", "passes.cuh", "host.cuh")
UNITS = {"bnufft": ("bnufft.cu", [], None),
         **{f"passes_{g}": ("passes.cu", [f"-DPASS_GROUP={g}"], PASS_HEADERS) for g in range(PASS_GROUPS)}}

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
         "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall", "--cudart", "shared",
         "-I" + os.path.join(ROOT, "include")]


def _inputs(unit):
    src, _, headers = UNITS[unit]
    hs = [f for f in os.listdir(CSRC) if f.endswith(".cuh")] if headers is None else headers
    return [os.path.join(CSRC, f) for f in (src, *hs)] + \
        [os.path.join(ROOT, "include", f) for f in ("bnufft.h", "bespirit.h")]


def _stale(target, unit) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(f) > os.path.getmtime(target) for f in _inputs(unit))


def needs_build() -> bool:
    return any(_stale(LIB, u) for u in UNITS)


def _compile(unit, force, verbose) -> str:
    obj = os.path.join(OBJ, unit + ".o")
    if force or _stale(obj, unit):
        src, extra, _ = UNITS[unit]
        cmd = [NVCC, "-c"] + FLAGS + extra + (["-Xptxas", "-v"] if verbose else []) + [os.path.join(CSRC, src), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed ({unit}):\n" + r.stdout + r.stderr)
        if verbose:
            sys.stderr.write(r.stderr)
    return obj


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    os.makedirs(OBJ, exist_ok=True)
    os.makedirs(os.path.dirname(LIB), exist_ok=True)
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
        objs = list(pool.map(lambda u: _compile(u, force, verbose), UNITS))
    r = subprocess.run([NVCC, "-shared", "--cudart", "shared"] + objs + ["-o", LIB], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n" + r.stdout + r.stderr)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
