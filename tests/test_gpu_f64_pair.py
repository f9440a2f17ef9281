"""The FP64 step in increment form (FP32-pair arithmetic, gbf_f64_pair.cuh)
against the oracle: every combination of cell fields, source and boundary mode,
at sizes with one interior cell, a warp's remainder and several blocks, from
states that reach each branch: S exactly 0 (the water-only form), subnormal
and tiny S, S near residual water (beyond the logarithm's table), slightly
negative S. The models that keep the plain FP64 passes (fewer than 7 Newton
iterations) are held to the same oracle.

Tolerances are those of the plain FP64 paths (gpu_util: 1e-12 on S and on the
other arrays, p_tol on P, 1e-10 on velocities).
"""
import numpy as np
import pytest

from gpu_util import F64_TOL_GRADIENT, assert_field, p_tol

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (4, 3, 5), (5, 7, 6), (34, 9, 8), (33, 18, 35)]
FORMS = {  # media table, K field, phi field, rate source with hydrostatic sides, reference compressibilities
    "table_patch_ini": (True, False, False, False, True),
    "table_rate": (True, False, False, True, False),
    "K_only_rate_ini": (True, True, False, True, True),
    "phi_only_patch": (True, False, True, False, False),
    "fields_rate": (False, True, True, True, False),
    "fields_patch_ini": (False, True, True, False, True),
}


def make(abi, O, lib, size, form, iterations):
    import ctypes
    table, hasK, hasphi, rate, ini = FORMS[form]
    nx, ny, nz = size
    rng = np.random.default_rng(nx * 10007 + ny * 101 + nz)
    m = abi.reference_model(nx, ny, nz, 1.0)
    if not ini:
        m.beta1 = m.beta2 = 1e-9
    if rate:
        m.source_mode, m.rate_cells, m.rate = abi.GBF_SOURCE_RATE, 1, 1e-3
        m.bc_mode, m.kv = abi.GBF_BC_HYDROSTATIC_SIDES, 0.6
    else:
        m.source = (min(nx, nz) - 1) // 4
    m.newton_iterations = iterations
    media = (rng.random(m.shape) < 0.4).astype(np.int32) if table else None
    K = (6.64e-11 * np.exp(rng.normal(0, 1, m.shape))).astype(np.float32) if hasK else None
    phi = (0.35 + 0.05 * rng.uniform(-1, 1, m.shape)).astype(np.float32) if hasphi else None
    st = O.State(m, media, K, phi)
    cells = st.gbf_cells(abi)
    m.dt = 0.1 * lib.gbf_stable_dt(ctypes.byref(m), ctypes.byref(cells), 1.0)
    st.model = m
    j = np.arange(ny)[None, :, None]
    P = m.P_atm + j * m.ro01 * m.g * m.h2 + rng.normal(0, 100, m.shape)
    S = np.where(rng.random(m.shape) < 0.4, 0.0, 0.7 * rng.random(m.shape))
    # near residual water only in cells of the media with the larger S_wr: the
    # boundary rules copy S across media
    md = 1 if table else 0
    wet = 1.0 - m.S_wr[md]
    special = [1e-320, 1e-30, 1e-12, wet * (1 - 1e-2), wet * (1 - 1e-4), -1e-9]
    pick = rng.random(m.shape)
    for q, v in enumerate(special):
        where = (pick > 0.03 * q) & (pick < 0.03 * (q + 1))
        S[where & (st.media == md) if 0.8 < v else where] = v
    return m, st, P, S


@pytest.mark.parametrize("iterations", [7, 6])
@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("size", SIZES)
def test_pair_step_matches_oracle(gpu_lib, abi, O, oracle, pkg, size, form, iterations):
    from importlib import import_module
    Domain = import_module(pkg.__name__ + ".domain").Domain
    m, st, P0, S0 = make(abi, O, gpu_lib, size, form, iterations)
    st["P1"][...], st["S2"][...] = P0, S0
    steps = 4
    mass_ref = oracle.step(st, steps, want_mass=True)
    dom = Domain(m, st.media, st.K, st.phi)
    dom.set_outputs(abi.GBF_OUT_MASS | abi.GBF_OUT_VELOCITY | abi.GBF_OUT_MASS_ARRAYS | abi.GBF_OUT_PROPS, steps)
    dom.upload(P0, S0)
    dom.step(steps - 1)
    last = st.copy()  # the state the last step starts from, for its derived arrays
    last["P1"][...], last["S2"][...] = dom.download("P1"), dom.download("S2")
    dom.step(1)
    assert dom.status() == abi.GBF_OK
    assert_field("S2", dom.download("S2"), st["S2"])
    assert_field("P1", dom.download("P1"), st["P1"], tol=p_tol(m))
    oracle.step(last, 1)
    inner = (slice(1, -1),) * 3
    for name in ("P2", "ro1", "ro2", "Xi1", "Xi2", "u1x", "u1y", "u1z", "u2x", "u2y", "u2z"):
        assert_field(name, dom.download(name), last[name], tol=F64_TOL_GRADIENT if name[0] == "u" else p_tol(m))
    for name in ("roS1", "roS2", "roS1_old", "roS2_old"):
        assert_field(name, dom.download(name)[inner], last[name][inner], tol=p_tol(m))
    mass = dom.mass_history(steps)
    for ph in range(2):
        scale = np.abs(mass_ref[:, ph]).max()
        assert np.abs(mass[:, ph] - mass_ref[:, ph]).max() <= 1e-12 * scale
    dom.close()
