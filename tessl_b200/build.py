"""Builds the CUDA library in-tree: `tessl_b200/_lib/libtessl_b200.so`.

One `nvcc` invocation for sm_100a (the only target this library has). nvcc
cross-compiles without a GPU, so this also runs on a CPU-only build box.

    python -m tessl_b200.build [--force] [--verbose-ptxas]
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
LIB = HERE / "_lib" / "libtessl_b200.so"
STEP_DRIVER = HERE / "_lib" / "tessl_step_driver"
PY_CALL = HERE / "_lib" / ("_tessl_call" + sysconfig.get_config_var("EXT_SUFFIX"))  # of this interpreter
SOURCES = ["capi.cu", "nn_q4.cu", "nn_q8.cu", "q4_weight.cu", "prefill_gemm.cu", "peer_gather.cu", "qwen35_norm.cu", "mlx_q4_loader.cu"]


def nvcc_path() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found (set NVCC or add it to PATH)")


HEADER = HERE.parent / "include" / "tessl_b200.h"


def _older(built, deps) -> bool:
    return not all(b.exists() for b in built) or any(d.stat().st_mtime > min(b.stat().st_mtime for b in built) for d in deps)


def is_stale() -> bool:
    deps = [d for pattern in ("*.cu", "*.cuh", "*.h", "*.cpp") for d in CSRC.glob(pattern)]
    return _older((LIB, STEP_DRIVER), deps + [HEADER])


def build(force: bool = False, verbose_ptxas: bool = False) -> Path:
    if force or is_stale():
        build_library(verbose_ptxas)
    if force or _older((PY_CALL,), (CSRC / "py_call.c", HEADER)):
        try:
            build_py_call()
        except RuntimeError as e:  # no C compiler, or no headers of this interpreter
            sys.stderr.write(f"tessl_b200: operator calls from Python will go through ctypes: {e}\n")
    return LIB


def build_library(verbose_ptxas: bool = False) -> None:
    """The CUDA library and the step driver."""
    LIB.parent.mkdir(parents=True, exist_ok=True)
    host_cxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else None
    cmd = [nvcc_path(), "-std=c++17", "-O3", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a",
           "-shared", "-Xcompiler", "-fPIC,-fvisibility=hidden", "--expt-relaxed-constexpr",
           "-Xlinker", "--exclude-libs,ALL"]
    if host_cxx:
        cmd += ["-ccbin", host_cxx]
    if verbose_ptxas:
        cmd += ["-Xptxas", "-v"]
    cmd += os.environ.get("TESSL_B200_NVCC_FLAGS", "").split()
    cmd += ["-o", str(LIB)] + [str(CSRC / s) for s in SOURCES]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed:\n$ " + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    if verbose_ptxas:
        sys.stderr.write(r.stderr)
    build_step_driver(host_cxx)


def build_step_driver(host_cxx=None) -> Path:
    """The compiled host of the end-to-end measurement (csrc/host_step_driver.cpp): plain C++ over the
    public header, linked against the library beside it (found at run time through $ORIGIN)."""
    cmd = [nvcc_path(), "-std=c++17", "-O2", "-o", str(STEP_DRIVER), str(CSRC / "host_step_driver.cpp"),
           "-L", str(LIB.parent), "-ltessl_b200", "-Xlinker", "-rpath,$ORIGIN", "-Xcompiler", "-pthread"]
    if host_cxx:
        cmd += ["-ccbin", host_cxx]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("step driver build failed:\n$ " + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    return STEP_DRIVER


def build_py_call() -> Path:
    """The operator calls of the Python binding (csrc/py_call.c): a CPython extension for this interpreter, linked against the
    library beside it."""
    cc = next((c for c in ("/usr/bin/gcc", shutil.which("gcc"), shutil.which("cc")) if c and Path(c).exists()), None)
    if cc is None:
        raise RuntimeError("no C compiler found")
    cmd = [cc, "-O2", "-Wall", "-shared", "-fPIC", "-fvisibility=hidden", "-I", sysconfig.get_paths()["include"],
           "-o", str(PY_CALL), str(CSRC / "py_call.c"), "-L", str(LIB.parent), "-ltessl_b200", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("binding build failed:\n$ " + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    return PY_CALL


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose-ptxas", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose_ptxas=a.verbose_ptxas))
