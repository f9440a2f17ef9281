"""Cells that the FP64 step's pairs refuse, in blocks of several thousand cells:
few (one list a block), more than a list holds, and most of a block (each thread
its own); a single domain and an ensemble against the oracle, and the same bits
of state and masses on a repeat."""
import ctypes
from importlib import import_module
from types import SimpleNamespace

import numpy as np
import pytest

from gpu_util import assert_field, p_tol

pytestmark = pytest.mark.gpu


def state(abi, lib, shape, share):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + int(1000 * share))
    m = abi.reference_model(nx, ny, nz, 1.0)
    cells = abi.GbfCells()
    m.dt = 1e-3 * lib.gbf_stable_dt(ctypes.byref(m), ctypes.byref(cells), 1.0)
    P = m.P_atm + np.arange(ny)[None, :, None] * m.ro01 * m.g * m.h2 + rng.normal(0, 10, m.shape)
    S = 0.3 + 0.01 * rng.random(m.shape)
    S[rng.random(m.shape) < share] = (1.0 - m.S_wr[0]) * (1.0 - 1e-5)  # near residual water
    return m, P, S


@pytest.mark.parametrize("share", [0.002, 0.06, 0.5])
def test_refused_cells_of_large_blocks(gpu_lib, abi, O, oracle, pkg, share):
    Domain = import_module(pkg.__name__ + ".domain").Domain
    Ensemble = import_module(pkg.__name__ + ".ensemble").Ensemble
    members, want = [], []
    for shape in ((128, 127, 126), (40, 33, 35)):
        m, P, S = state(abi, O.inputs_library(abi), shape, share)
        st = O.State(m)
        st["P1"][...], st["S2"][...] = P, S
        mass = oracle.step(st, 2, want_mass=True)
        assert np.isfinite(st["S2"]).all() and np.isfinite(st["P1"]).all()
        members.append((m, P, S))
        want.append((st["P1"], st["S2"], mass))

    def check(m, got, w):
        assert_field("S2", got[1], w[1])
        assert_field("P1", got[0], w[0], tol=p_tol(m))
        assert np.abs(got[2] - w[2]).max() <= 1e-12 * np.abs(w[2]).max()

    for (m, P, S), w in zip(members, want):
        runs = []
        for _ in range(2):
            dom = Domain(m)
            dom.set_outputs(abi.GBF_OUT_MASS, 2)
            dom.upload(P, S)
            dom.step(2)
            assert dom.status() == abi.GBF_OK
            runs.append((dom.download("P1"), dom.download("S2"), dom.mass_history(2)))
            dom.close()
        check(m, runs[0], w)
        for a, b in zip(*runs):
            assert np.array_equal(a, b)
    ens = Ensemble([SimpleNamespace(model=m, K=None, phi=None) for m, _, _ in members], precision=abi.GBF_PREC_F64)
    ens.set_outputs(abi.GBF_OUT_MASS, 2)
    for r, (_, P, S) in enumerate(members):
        ens.upload(r, P, S)
    ens.step(2)
    assert ens.status() == abi.GBF_OK
    mass = ens.mass_history(2)
    for r, w in enumerate(want):
        check(members[r][0], (ens.download(r, "P1"), ens.download(r, "S2"), mass[:, r]), w)
    ens.close()
