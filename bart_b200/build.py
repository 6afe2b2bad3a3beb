"""Build the sm_100a shared library ``bart_b200/lib/libbnufft.so`` in-tree.

``python -m bart_b200.build`` (or ``build()``) runs nvcc directly; the
library has a plain C ABI (include/bnufft.h, include/bespirit.h) and links only the CUDA
runtime; the ESPIRiT calibration loads cuSOLVER on first use. The FFT pass
kernels compile in several translation units at once.
"""

from __future__ import annotations

import hashlib
import os
import subprocess
import sys
import tempfile
import time
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "lib", "libbnufft.so")
OBJ = os.path.join(HERE, "_build")      # objects, in the checkout (ignored by git)
STAMP = os.path.join(OBJ, "command")    # the command the library was built with
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


def _command(unit):
    src, extra, _ = UNITS[unit]
    return [NVCC, "-c"] + FLAGS + extra + [os.path.join(CSRC, src)]


def _hash(words) -> str:
    """Of a command (its paths relative to the checkout) and the compiler's version."""
    v = subprocess.run([NVCC, "--version"], capture_output=True, text=True).stdout if os.path.exists(NVCC) else ""
    return hashlib.sha256((repr(words).replace(ROOT, ".") + v).encode()).hexdigest()[:16]


def _library_hash() -> str:
    return _hash([_command(u) for u in UNITS])


def _older(target, unit) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(f) > os.path.getmtime(target) for f in _inputs(unit))


def needs_build() -> bool:
    """The library is missing, older than a source, or was built by another command."""
    if any(_older(LIB, u) for u in UNITS):
        return True
    try:
        with open(STAMP) as f:
            # without the compiler the library at hand is used as it is
            return os.path.exists(NVCC) and f.read() != _library_hash()
    except OSError:
        return os.path.exists(NVCC)


def _run(cmd, target, what, begun, verbose=False) -> None:
    """Run cmd with -o, under a name of its own, then move the output to target: a build
    that fails or runs beside another one leaves no half-written file. The output
    is dated begun: a source that changed since is newer."""
    fd, tmp = tempfile.mkstemp(dir=os.path.dirname(target), prefix=".", suffix=os.path.basename(target))
    os.close(fd)
    try:
        r = subprocess.run(cmd + ["-o", tmp], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed ({what}):\n" + r.stdout + r.stderr)
        if verbose:
            sys.stderr.write(r.stderr)
        os.utime(tmp, (begun, begun))
        os.chmod(tmp, 0o755)
        os.replace(tmp, target)
    finally:
        if os.path.exists(tmp):
            os.unlink(tmp)


def _compile(unit, force, verbose) -> str:
    """The object of a unit, named by its command."""
    obj = os.path.join(OBJ, f"{unit}-{_hash(_command(unit))}.o")
    if force or _older(obj, unit):
        _run(_command(unit) + (["-Xptxas", "-v"] if verbose else []), obj, unit, time.time(), verbose)
    return obj


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    begun = time.time()
    os.makedirs(OBJ, exist_ok=True)
    os.makedirs(os.path.dirname(LIB), exist_ok=True)
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
        objs = list(pool.map(lambda u: _compile(u, force, verbose), UNITS))
    _run([NVCC, "-shared", "--cudart", "shared"] + objs, LIB, "link", begun)
    with open(STAMP, "w") as f:
        f.write(_library_hash())
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
