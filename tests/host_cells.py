"""The per-cell device code of the FP64 step on the CPU (tests/host_cells/,
built with g++ and contraction off)."""
import ctypes
import pathlib
import subprocess
import tempfile

ROOT = pathlib.Path(__file__).resolve().parents[1]
_lib = None


def library(abi):
    global _lib
    if _lib is None:
        src, csrc = ROOT / "tests" / "host_cells", ROOT / "shmem-cuda-filtration_gb300" / "csrc"
        out = pathlib.Path(tempfile.mkdtemp()) / "libcells.so"
        subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-shared", "-fPIC", "-I", str(ROOT / "include"),
                        "-I", str(csrc), "-I", "/usr/local/cuda/include", "-include", str(src / "cuda_on_host.h"),
                        "-o", str(out), str(src / "cells.cpp")], check=True)
        lib = ctypes.CDLL(str(out))
        p = ctypes.c_void_p
        lib.host_pair_functions.argtypes = [ctypes.c_int, p, p, p, p, p]
        _lib = lib
    return _lib
