"""The per-cell device code of the FP64 step on the CPU (tests/host_cells/,
built with g++ and contraction off)."""
import ctypes
import pathlib
import subprocess
import tempfile

import numpy as np

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
        PM = ctypes.POINTER(abi.GbfModel)
        p = ctypes.c_void_p
        lib.host_f64_steps.argtypes = [PM, p, p, p, p, p, ctypes.c_int, ctypes.c_int, p]
        lib.host_f64_steps.restype = ctypes.c_uint
        lib.host_fp64_cells.restype = ctypes.c_long
        lib.host_pair_applies.argtypes = [PM]
        lib.host_pair_functions.argtypes = [ctypes.c_int, p, p, p, p, p]
        _lib = lib
    return _lib


def steps(abi, m, media, K, phi, P, S, n, pair):
    """(P, S, masses, status) after n steps by the pair step or the plain FP64 passes."""
    P, S = np.array(P, np.float64, order="C"), np.array(S, np.float64, order="C")
    masses = np.zeros((n, 2))
    ptr = lambda a: None if a is None else a.ctypes.data  # noqa: E731
    bad = library(abi).host_f64_steps(ctypes.byref(m), ptr(media), ptr(K), ptr(phi), P.ctypes.data, S.ctypes.data, n,
                                      int(pair), masses.ctypes.data)
    return P, S, masses, bad
