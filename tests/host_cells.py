"""The per-cell device code of the FP64 step on the CPU (tests/host_cells/,
built with g++ and contraction off), and the steps in extended precision."""
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


def exact_interior(abi, m, media, K, phi, P0, S0, iterations=6):
    """(P, S) of the interior after one step, in extended precision and increments (nothing cancels)."""
    F = np.longdouble
    P, S = P0.astype(F), S0.astype(F)
    tab = lambda v: np.asarray(v, F)[media] if media is not None else F(v[0])  # noqa: E731
    Kc = K.astype(F) if K is not None else tab(list(m.K))
    ph = phi.astype(F) if phi is not None else tab(list(m.m))
    swr, lam, pd = tab(list(m.S_wr)), tab(list(m.lam)), tab(list(m.P_d))
    h1, h2, h3, dt, g, kv = (F(v) for v in (m.h1, m.h2, m.h3, m.dt, m.g, m.kv))
    ro01, ro02, b1, b2, Pa = (F(v) for v in (m.ro01, m.ro02, m.beta1, m.beta2, m.P_atm))
    c = (slice(1, -1),) * 3
    at = lambda v: v[c] if np.ndim(v) else v  # noqa: E731
    om = S / (1 - swr)
    ln = np.log1p(-om)
    ro1, ro2 = ro01 * (1 + b1 * (P - Pa)), ro02 * (1 + b2 * (P - Pa))
    L1 = Kc * np.exp((2 + 3 * lam) / lam * ln) / F(m.mu1) * ro1
    L2 = Kc * om * om * -np.expm1((2 + lam) / lam * ln) / F(m.mu2) * ro2
    f = [F(0), F(0)]
    for axis, h, w in ((2, h1, F(1)), (1, h2, kv), (0, h3, F(1))):
        lo, hi = list(c), list(c)
        lo[axis], hi[axis] = slice(0, -2), slice(2, None)
        lo, hi = tuple(lo), tuple(hi)
        x1, x2 = (P[lo] - P[c]) / h, (P[c] - P[hi]) / h
        for a, (L, ro) in enumerate(((L1, ro1), (L2, ro2))):
            y1, y2 = x1, x2
            if axis == 1:
                y1, y2 = x1 + ro[c] * g, x2 + ro[c] * g
                if m.bc_mode == abi.GBF_BC_HYDROSTATIC_SIDES:
                    y2[:, -1, :] = 0
            f[a] = f[a] + w * (y2 * np.where(y2 >= 0, L[c], L[hi]) - y1 * np.where(y1 >= 0, L[lo], L[c])) / h
    r1, r2 = dt / at(ph) * f[0], dt / at(ph) * f[1]
    if m.source_mode == abi.GBF_SOURCE_RATE:
        n, i0, k0 = m.rate_cells, m.nx // 2 - m.rate_cells // 2, m.nz // 2 - m.rate_cells // 2
        src = (slice(max(k0, 1) - 1, min(k0 + n, m.nz - 1) - 1), 0, slice(max(i0, 1) - 1, min(i0 + n, m.nx - 1) - 1))
        r2[src] -= dt / (at(ph)[src] if np.ndim(ph) else ph) * (F(m.rate) / (n * n) / (h1 * h2 * h3))
    Pc, Sc, lamc, swrc, lnc = P[c], S[c], at(lam), at(swr), ln[c]
    Se = 1 - Sc / (1 - swrc)
    Pk = at(pd) * np.exp(-lnc / lamc)
    r2 = r2 + ro02 * b2 * Pk * Sc
    a, b = 1 + b1 * (Pc - Pa), 1 + b2 * (Pc - Pa + Pk)
    dp, ds = np.zeros_like(r1), np.zeros_like(r1)
    for _ in range(iterations):
        dPk = Pk * np.expm1(-np.log1p(-ds / ((1 - swrc) * Se)) / lamc)
        Sn = Sc + ds
        G1 = r1 + ro01 * (b1 * dp * (1 - Sn) - a * ds)
        G2 = r2 + ro02 * (b2 * (dp + dPk) * Sn + b * ds)
        slope = (Pk + dPk) / (lamc * ((1 - swrc) - Sn))
        J11, J12 = ro01 * b1 * (1 - Sn), -ro01 * (a + b1 * dp)
        J21, J22 = ro02 * b2 * Sn, ro02 * (b + b2 * (dp + dPk + slope * Sn))
        det = J11 * J22 - J12 * J21
        dp, ds = dp - (J22 * G1 - J12 * G2) / det, ds - (J11 * G2 - J21 * G1) / det
    return Pc + dp, Sc + ds
