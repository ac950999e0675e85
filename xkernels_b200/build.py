"""Builds ``libxkb200.so`` (the C-ABI library of sm_100a kernels) in-tree with nvcc, and the native call path of the small
ops (``_torch_calls.*.so``, for the torch and Python that run the build) with the host compiler.

Run ``python -m xkernels_b200.build`` or call :func:`build`.  The objects are
compiled in parallel, one nvcc process per ``.cu`` file, and linked into
``xkernels_b200/libxkb200.so``.  nvcc cross-compiles, so no GPU is needed.
"""

from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
import warnings
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

from ._lib import CALLS_PATH

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_PATH = PKG_DIR / "libxkb200.so"
OBJ_DIR = PKG_DIR / "build"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: cannot build libxkb200.so")
    return exe


def _sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _fingerprint() -> str:
    h = hashlib.sha256()
    for p in sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h"))
                    + [PKG_DIR.parent / "include" / "xkb200.h"]):
        h.update(p.name.encode())
        h.update(p.read_bytes())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def is_current() -> bool:
    stamp = OBJ_DIR / "fingerprint"
    return LIB_PATH.exists() and stamp.exists() and stamp.read_text() == _fingerprint()


def _calls_fingerprint() -> str:
    h = hashlib.sha256((CSRC / "torch_calls.cpp").read_bytes())
    h.update((PKG_DIR.parent / "include" / "xkb200.h").read_bytes())
    return f"{CALLS_PATH.name} {sys.version} {h.hexdigest()}"


def calls_are_current() -> bool:
    stamp = OBJ_DIR / "calls_fingerprint"
    return CALLS_PATH.exists() and stamp.exists() and stamp.read_text() == _calls_fingerprint()


def _compile_calls() -> None:
    import torch
    from torch.utils import cpp_extension as ext

    cxx = os.environ.get("CXX") or shutil.which("g++") or "c++"
    dirs = [*ext.include_paths(), sysconfig.get_paths()["include"], str(Path(_nvcc()).resolve().parents[1] / "include")]
    cmd = [cxx, "-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           *(f"-I{d}" for d in dirs), str(CSRC / "torch_calls.cpp"), "-o", str(CALLS_PATH),
           *(f"-L{d}" for d in ext.library_paths()), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"build of {CALLS_PATH.name} failed:\n{res.stdout}\n{res.stderr}")


def build_calls(force: bool = False) -> bool:
    """Compile the native call path for this torch and Python.  Returns whether it is there: it needs a host compiler and
    both's headers, and without them the ops take their Python form, so a failure is a warning."""
    if not force and calls_are_current():
        return True
    OBJ_DIR.mkdir(exist_ok=True)
    CALLS_PATH.unlink(missing_ok=True)   # never the path of another source
    try:
        _compile_calls()
    except (ImportError, OSError, RuntimeError) as e:
        warnings.warn(f"the small ops take their Python form, 5 to 8 us more of host time a call: {e}", stacklevel=2)
        return False
    (OBJ_DIR / "calls_fingerprint").write_text(_calls_fingerprint())
    return True


def build_library(force: bool = False, verbose: bool = False) -> None:
    """Compile every ``csrc/*.cu`` for sm_100a and link the shared library."""
    if not force and is_current():
        return
    nvcc = _nvcc()
    OBJ_DIR.mkdir(exist_ok=True)
    extra = ["-Xptxas", "-v"] if verbose else []

    def compile_one(src: Path) -> Path:
        obj = OBJ_DIR / (src.stem + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", str(src), "-o", str(obj)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
        if verbose:
            sys.stderr.write(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        objs = list(pool.map(compile_one, _sources()))
    cmd = [nvcc, "-shared", "-o", str(LIB_PATH), *map(str, objs)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link of libxkb200.so failed:\n{res.stdout}\n{res.stderr}")
    (OBJ_DIR / "fingerprint").write_text(_fingerprint())


def build(force: bool = False, verbose: bool = False) -> Path:
    """Build what is not current: the library, and the call path beside it."""
    with ThreadPoolExecutor(max_workers=1) as pool:
        calls = pool.submit(build_calls, force)
        build_library(force, verbose)
        calls.result()
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
