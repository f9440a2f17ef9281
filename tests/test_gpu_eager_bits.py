"""The eager FP64 functions keep the bits of the plain expressions (the oracle's,
compiled without contraction), wherever no pow() of an S_e other than 1 enters:
velocities and mass updates of every cell, mobilities and densities of cells
without DNAPL. A zero divided by a constant keeps the quotient's sign, or is a
NaN, whatever the constant, and S = 0 is no S_e of 1 where S_wr = 1 (the stage
functions take any model)."""
import ctypes

import numpy as np
import pytest

from gpu_util import DevState
from test_gpu_eager_shortcuts import SIZES, state

pytestmark = pytest.mark.gpu


def same_bits(a, b):
    return np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(
        np.where(np.isnan(a), 0.0, a).view(np.int64), np.where(np.isnan(b), 0.0, b).view(np.int64))


@pytest.mark.parametrize("fields", [False, True])
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("h1", [0.02045, -0.02045, float("nan")])
def test_velocity_and_mass_bits(gpu_lib, abi, O, oracle, size, fields, h1):
    m, st, rng = state(abi, O, size, fields, 5)
    P = st["P1"]
    P[:, :, : size[0] // 2 + 1] = P[:, :, :1]  # no gradient along x in a half
    oracle.props(st)
    st["P2"][...] += np.where(rng.random(m.shape) < 0.1, rng.normal(0, 1, m.shape), 0.0)  # P2 unlike P1 in places
    m.h1 = h1
    st.model = m
    dev = DevState(st, abi)
    oracle.velocity(st)
    oracle.mass(st)
    assert gpu_lib.gbf_velocity_f64(ctypes.byref(m), dev.arrays(), None) == abi.GBF_OK
    assert gpu_lib.gbf_mass_f64(ctypes.byref(m), dev.arrays(), dev.cells(), None) == abi.GBF_OK
    for name in ("u1x", "u1y", "u1z", "u2x", "u2y", "u2z"):
        assert same_bits(dev.host(name), st[name]), name
    inner = (slice(1, -1),) * 3
    for name in ("roS1", "roS2", "roS1_old", "roS2_old"):
        assert same_bits(dev.host(name)[inner], st[name][inner]), name


@pytest.mark.parametrize("fields", [False, True])
@pytest.mark.parametrize("size", SIZES)
def test_props_bits_without_dnapl(gpu_lib, abi, O, oracle, size, fields):
    m, st, _ = state(abi, O, size, fields, 6)
    dev = DevState(st, abi)
    oracle.props(st)
    assert gpu_lib.gbf_props_f64(ctypes.byref(m), dev.arrays(), dev.cells(), None) == abi.GBF_OK
    dry = st["S2"] == 0
    for name in ("P2", "ro1", "ro2"):
        assert same_bits(dev.host(name), st[name]), name
    for name in ("Xi1", "Xi2"):
        assert same_bits(dev.host(name)[dry], st[name][dry]), name


@pytest.mark.parametrize("name,value", [("S_wr", 1.0), ("S_wr", float("nan")), ("lam", 0.0), ("P_d", float("inf"))])
def test_models_without_a_unit_saturation(gpu_lib, abi, O, oracle, name, value):
    """NaN where the plain expressions of cells without DNAPL are."""
    m, st, _ = state(abi, O, (9, 8, 7), False, 8)
    getattr(m, name)[:] = [value, value]
    st.model = m
    dev = DevState(st, abi)
    oracle.props(st)
    oracle.mass(st)
    oracle.newton(st)
    c = dev.cells()
    assert gpu_lib.gbf_props_f64(ctypes.byref(m), dev.arrays(), c, None) == abi.GBF_OK
    assert gpu_lib.gbf_mass_f64(ctypes.byref(m), dev.arrays(), c, None) == abi.GBF_OK
    assert gpu_lib.gbf_newton_f64(ctypes.byref(m), dev.arrays(), c, None) == abi.GBF_OK
    for f in ("Xi1", "Xi2", "roS1", "roS2", "P1", "S2"):
        assert np.array_equal(np.isnan(dev.host(f)), np.isnan(st[f])), f
