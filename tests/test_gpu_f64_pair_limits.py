"""The FP64 step on a GPU where its increments do not fit FP32 pairs: near
residual water and for small lambda (single domains, and an ensemble of them),
far from hydrostatic, and a drop-in whose parameters move from the pair step to
the plain passes and back. Against the oracle at the plain FP64 paths' tolerances."""
from importlib import import_module
from types import SimpleNamespace

import numpy as np
import pytest

from gpu_util import assert_field, p_tol
from test_pair_cells import overpressure, residual_state

pytestmark = pytest.mark.gpu

LAMBDAS = [0.05, 0.125, 0.3, 1.0, 2.0, 2.7]
WATER = [0.1, 1e-2, 1e-3, 4.5e-4, 1e-6, 1e-9]


def oracle_step(O, oracle, m, P, S, media=None, n=1):
    st = O.State(m, media)
    st["P1"][...], st["S2"][...] = P, S
    mass = oracle.step(st, n, want_mass=True)
    return st["P1"], st["S2"], mass


def check(m, got_P, got_S, mass, want):
    assert_field("S2", got_S, want[1])
    assert_field("P1", got_P, want[0], tol=p_tol(m))
    assert np.abs(mass - want[2]).max() <= 1e-12 * np.abs(want[2]).max()


@pytest.mark.parametrize("iterations", [7, 20])
@pytest.mark.parametrize("lam", LAMBDAS)
def test_residual_water(gpu_lib, abi, O, oracle, pkg, lam, iterations):
    pk = import_module(pkg.__name__ + ".domain")
    members = []
    for w in WATER:
        for ini in (True, False):
            m, P, S = residual_state(abi, O.inputs_library(abi), lam, w, ini, iterations)
            want = oracle_step(O, oracle, m, P, S)
            if not all(np.isfinite(a).all() for a in want):
                continue
            members.append((m, P, S, want))
            dom = pk.Domain(m)
            dom.set_outputs(abi.GBF_OUT_MASS, 1)
            dom.upload(P, S)
            dom.step(1)
            assert dom.status() == abi.GBF_OK, w
            check(m, dom.download("P1"), dom.download("S2"), dom.mass_history(1), want)
            dom.close()
    assert members
    Ensemble = import_module(pkg.__name__ + ".ensemble").Ensemble
    ens = Ensemble([SimpleNamespace(model=m, K=None, phi=None) for m, *_ in members], precision=abi.GBF_PREC_F64)
    ens.set_outputs(abi.GBF_OUT_MASS, 1)
    for r, (_, P, S, _) in enumerate(members):
        ens.upload(r, P, S)
    ens.step(1)
    assert ens.status() == abi.GBF_OK
    masses = ens.mass_history(1)
    for r, (m, _, _, want) in enumerate(members):
        check(m, ens.download(r, "P1"), ens.download(r, "S2"), masses[:, r], want)
    ens.close()


@pytest.mark.parametrize("smooth", [True, False])
@pytest.mark.parametrize("uniform", [0.0, 1e4, 1e6])
@pytest.mark.parametrize("amp", [100.0, 1e4])
@pytest.mark.parametrize("ini", [True, False])
def test_overpressure(gpu_lib, abi, O, oracle, pkg, ini, amp, uniform, smooth):
    Domain = import_module(pkg.__name__ + ".domain").Domain
    m, media, P, S = overpressure(abi, O, ini, amp, uniform, smooth)
    want = oracle_step(O, oracle, m, P, S, media)
    dom = Domain(m, media)
    dom.set_outputs(abi.GBF_OUT_MASS, 1)
    dom.upload(P, S)
    dom.step(1)
    assert dom.status() == abi.GBF_OK
    check(m, dom.download("P1"), dom.download("S2"), dom.mass_history(1), want)
    dom.close()


def test_dropin_parameters_change_the_step(gpu_lib, abi, O, oracle, pkg):
    """lambda 2 -> 0.05 (plain passes) -> 2 between fused steps."""
    dp = import_module(pkg.__name__ + ".dropin")
    import ctypes
    di = dp.DropIn()
    m, P, S = residual_state(abi, O.inputs_library(abi), 2.0, 0.6, True, 7, n=12)
    m.S_wr[:] = [0.1, 0.1]
    st = O.State(m)
    st["P1"][...], st["S2"][...] = P, S
    H, D, buf = dp.PtrArrays(), dp.PtrArrays(), ctypes.c_void_p()
    c = dp.consts_from_model(m)
    di.set_mode(1)
    try:
        di.f["device_memory_alloc"](ctypes.byref(D), ctypes.byref(buf), m.nx, c)
        media = np.zeros(m.shape, np.int32)
        di.f["load_data_to_device_int"](media.ctypes.data, D.media, m.nx, c)
        for a, dev in ((P, D.P1), (S, D.S2)):
            a = np.ascontiguousarray(a)
            di.f["load_data_to_device"](a.ctypes.data, dev, m.nx, c)
        for s, lam in enumerate((2.0, 2.0, 0.05, 0.05, 2.0)):
            m.lam[:] = [lam, lam]
            c = dp.consts_from_model(m)
            di.time_step(H, D, c, (s + 1) * m.dt)
            oracle.step(st, 1)
        got = [np.empty(m.shape) for _ in range(3)]
        for a, dev in zip(got, (D.P1, D.S2, D.Xi2)):
            di.f["load_data_to_host"](a.ctypes.data, dev, m.nx, c)
        assert_field("S2", got[1], st["S2"])
        assert_field("P1", got[0], st["P1"], tol=p_tol(m))
        assert_field("Xi2", got[2], st["Xi2"])
        di.f["device_memory_free"](D, buf)
    finally:
        di.set_mode(0)
