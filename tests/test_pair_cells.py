"""The FP64 step's per-cell code on the CPU (host_cells.py): the pair step where
its increments are hard to hold in FP32 pairs, against the oracle near residual
water and for small lambda, and against extended precision far from hydrostatic,
where it may err no more than the plain FP64 passes."""
import ctypes

import numpy as np
import pytest

import host_cells
from gpu_util import F64_TOL, p_tol

INNER = (slice(1, -1),) * 3
extended = pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="no extended precision")


def residual_state(abi, lib, lam, w, ini, iterations, n=8):
    """A block of DNAPL with S_e = w to 1.5 w in every cell."""
    rng = np.random.default_rng(int(1e6 * lam) + n)
    m = abi.reference_model(n, n, n, 1.0)
    if not ini:
        m.beta1 = m.beta2 = 1e-9
    m.lam[:], m.S_wr[:] = [lam, lam], [0.1, 0.1]
    m.newton_iterations, m.source = iterations, 1
    cells = abi.GbfCells()
    m.dt = 0.1 * lib.gbf_stable_dt(ctypes.byref(m), ctypes.byref(cells), 1.0)
    P = m.P_atm + np.arange(n)[None, :, None] * m.ro01 * m.g * m.h2 + rng.normal(0, 100, m.shape)
    return m, P, 0.9 * (1 - w * (1 + 0.5 * rng.random(m.shape)))


@pytest.mark.parametrize("iterations", [7, 20])
@pytest.mark.parametrize("ini", [True, False])
@pytest.mark.parametrize("lam", [0.05, 0.125, 0.2, 0.3, 0.5, 1.0, 2.0, 2.7])
def test_residual_water_matches_oracle(abi, O, oracle, lam, ini, iterations):
    for w in (0.5, 0.1, 1e-2, 3e-3, 1e-3, 6e-4, 4.5e-4, 1e-4, 1e-5, 1e-6, 1e-7, 1e-8, 1e-9, 1e-12):
        m, P, S = residual_state(abi, O.inputs_library(abi), lam, w, ini, iterations)
        st = O.State(m)
        st["P1"][...], st["S2"][...] = P, S
        oracle.step(st, 1)
        pair = host_cells.library(abi).host_pair_applies(ctypes.byref(m))
        Pn, Sn, _, bad = host_cells.steps(abi, m, None, None, None, P, S, 1, pair)
        want_S, want_P = st["S2"][INNER], st["P1"][INNER]
        if not (np.isfinite(want_S).all() and np.isfinite(want_P).all()):
            assert bad, w
            continue
        assert not bad, w
        assert np.abs(Sn[INNER] - want_S).max() <= F64_TOL, w
        assert np.abs(Pn[INNER] - want_P).max() <= p_tol(m) * np.abs(want_P).max(), w


def overpressure(abi, O, ini, amp, uniform, smooth):
    n = 20
    rng = np.random.default_rng(0)
    m = abi.reference_model(n, n, n, 1.0)
    if not ini:
        m.beta1 = m.beta2 = 1e-9
    m.source = 1
    media = (rng.random(m.shape) < 0.3).astype(np.int32)
    cells = abi.GbfCells()
    cells.media = media.ctypes.data_as(ctypes.POINTER(ctypes.c_int))
    m.dt = 0.5 * O.inputs_library(abi).gbf_stable_dt(ctypes.byref(m), ctypes.byref(cells), 1.0)
    z, y, x = np.meshgrid(*(np.linspace(-1, 1, n),) * 3, indexing="ij")
    d = np.sin(2 * x + 1) * np.cos(1.5 * y) * np.cos(z) if smooth else rng.normal(0, 1, m.shape)
    P = m.P_atm + np.arange(n)[None, :, None] * m.ro01 * m.g * m.h2 + uniform + amp * d
    return m, media, P, np.where(rng.random(m.shape) < 0.3, 0.0, 0.6 * rng.random(m.shape))


@extended
@pytest.mark.parametrize("smooth", [True, False])
@pytest.mark.parametrize("uniform", [0.0, 1e4, 1e6])
@pytest.mark.parametrize("amp", [0.0, 100.0, 1e3, 1e4])
@pytest.mark.parametrize("ini", [True, False])
def test_overpressure_errs_no_more_than_fp64(abi, O, ini, amp, uniform, smooth):
    """Mean errors against extended precision: the pair step's within a tenth of the plain passes'."""
    m, media, P, S = overpressure(abi, O, ini, amp, uniform, smooth)
    Pe, Se = host_cells.exact_interior(abi, m, media, None, None, P, S)
    err = []
    for pair in (True, False):
        Pn, Sn, _, bad = host_cells.steps(abi, m, media, None, None, P, S, 1, pair)
        assert not bad
        err.append((float(np.abs((Pn[INNER] - Pe) / Pe).mean()), float(np.abs(Sn[INNER] - Se).mean())))
    for a, b in zip(*err):
        assert a <= 1.1 * b, err
