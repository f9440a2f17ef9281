"""The eager FP64 kernels' exact shortcuts (divisions through reciprocals,
cells without DNAPL, P2 = P1, the Newton's fixed points and 2-cycles) against
the oracle, each function on its own inputs: S of exactly 0 (both signs),
tiny, large, above 1 - S_wr; P2 unlike P1 in places; DNAPL mobility zero in
the whole neighbourhood, in part of it, and with a NaN or an infinity behind
it; iteration counts of both parities; grids of one interior cell, below a
block, and of several blocks. Tolerances: those of the eager path (1e-12)."""
import ctypes

import numpy as np
import pytest

from gpu_util import DevState, assert_field

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (5, 7, 6), (15, 15, 15), (34, 9, 33)]


def state(abi, O, size, fields, seed):
    nx, ny, nz = size
    rng = np.random.default_rng(seed + nx)
    m = abi.reference_model(nx, ny, nz, 1e-3)
    m.source = (min(nx, nz) - 1) // 4
    K = phi = media = None
    if fields:
        K = (6.64e-11 * np.exp(rng.normal(0, 1, m.shape))).astype(np.float32)
        phi = (0.35 + 0.05 * rng.uniform(-1, 1, m.shape)).astype(np.float32)
        m.source_mode, m.rate_cells, m.rate = abi.GBF_SOURCE_RATE, 1, 1e-3
        m.bc_mode, m.kv = abi.GBF_BC_HYDROSTATIC_SIDES, 0.5
    else:
        media = (rng.random(m.shape) < 0.4).astype(np.int32)
    st = O.State(m, media, K, phi)
    j = np.arange(ny)[None, :, None]
    st["P1"][...] = m.P_atm + j * m.ro01 * m.g * m.h2 + rng.normal(0, 100, m.shape)
    S = np.where(rng.random(m.shape) < 0.3, 0.7 * rng.random(m.shape), 0.0)
    S[:, :, : nx // 2] *= rng.random(m.shape)[:, :, : nx // 2] < 0.2  # a half nearly without DNAPL
    pick = rng.random(m.shape)
    S[pick < 0.05] = -0.0
    S[(pick > 0.05) & (pick < 0.1)] = 1e-30
    S[(pick > 0.1) & (pick < 0.13)] = 0.87
    st["S2"][...] = S
    return m, st, rng


@pytest.mark.parametrize("fields", [False, True])
@pytest.mark.parametrize("size", SIZES)
def test_functions_match_oracle(gpu_lib, abi, O, oracle, size, fields):
    m, st, rng = state(abi, O, size, fields, 3)
    dev = DevState(st, abi)
    a, c, lib = dev.arrays(), dev.cells(), gpu_lib
    oracle.props(st)
    assert lib.gbf_props_f64(ctypes.byref(m), a, c, None) == 0
    for name in ("P2", "Xi1", "Xi2", "ro1", "ro2"):
        assert_field(name, dev.host(name), st[name])
    # P2 unlike P1 in some cells: the phases' potentials differ there
    st["P2"][...] = np.where(rng.random(m.shape) < 0.1, st["P1"] + 7.0, st["P1"])
    dev.t["P2"].copy_(dev.t["P2"].new_tensor(st["P2"]))
    oracle.velocity(st)
    assert lib.gbf_velocity_f64(ctypes.byref(m), a, None) == 0
    for name in ("u1x", "u1y", "u1z", "u2x", "u2y", "u2z"):
        assert_field(name, dev.host(name), st[name], tol=1e-10)
    oracle.mass(st)
    assert lib.gbf_mass_f64(ctypes.byref(m), a, c, None) == 0
    for name in ("roS1", "roS2", "roS1_old", "roS2_old"):
        assert_field(name, dev.host(name), st[name])


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("field", ["P2", "ro2"])
def test_mass_keeps_nonfinite_neighbours(gpu_lib, abi, O, oracle, field, bad):
    """0 x inf and 0 x NaN are NaN: a non-finite pressure or density next to
    cells of zero DNAPL mobility reaches the same cells as in the oracle."""
    m, st, _ = state(abi, O, (9, 8, 7), False, 5)
    st["S2"][...] = 0.0
    oracle.props(st)
    st[field][3, 4, 4] = bad
    dev = DevState(st, abi)
    oracle.mass(st)
    assert gpu_lib.gbf_mass_f64(ctypes.byref(m), dev.arrays(), dev.cells(), None) == 0
    for name in ("roS1", "roS2"):
        assert np.array_equal(np.isfinite(dev.host(name)), np.isfinite(st[name])), name
    assert not np.isfinite(st["roS2"]).all()


@pytest.mark.parametrize("iterations", [1, 2, 3, 6, 7, 8, 15])
@pytest.mark.parametrize("size", SIZES)
def test_newton_matches_oracle(gpu_lib, abi, O, oracle, size, iterations):
    m, st, rng = state(abi, O, size, False, 7)
    m.newton_iterations = iterations
    st.model = m
    for beta in ((1e-4, 1e-8), (1e-9, 1e-9)):
        m.beta1, m.beta2 = beta
        oracle.props(st)
        st["roS1"][...] = st["ro1"] * (1 - st["S2"]) * (1 + 1e-7 * rng.normal(0, 1, m.shape) * (beta[0] > 1e-8))
        st["roS2"][...] = st["ro2"] * st["S2"] * (1 + 1e-4 * rng.normal(0, 1, m.shape))
        s = st.copy()
        for name in st.f:
            s[name][...] = st[name]
        dev = DevState(s, abi)
        oracle.newton(s)
        assert gpu_lib.gbf_newton_f64(ctypes.byref(m), dev.arrays(), dev.cells(), None) == 0
        assert_field("S2", dev.host("S2"), s["S2"])
        cond = 1.0 / (min(beta) * m.P_atm)
        assert_field("P1", dev.host("P1"), s["P1"], tol=max(1e-12, 4e-15 * cond))
