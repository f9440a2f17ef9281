"""The x-pair tile's shorter update of warps without DNAPL against the plain-load
tile, which has none: the same bits of P, S and CFL numbers where dry and wet
regions meet inside a warp, at its edges and between planes, S2 = -0, an FP64 S2
that is 0 in FP32 (a mass without a saturation), both sources in dry rock, and a
plume that moves into dry cells; a non-finite pressure in dry rock is reported."""
import numpy as np
import pytest

from test_gpu_split_pitch import FORMS, make

pytestmark = pytest.mark.gpu

SIZES = [(5, 4, 6), (35, 20, 9), (70, 21, 24), (131, 12, 40)]


def states(m, P, S):
    nz, ny, nx = m.shape
    box = np.zeros(m.shape, bool)
    box[nz // 3:nz // 3 + 2, 1:1 + ny // 2, nx // 3:nx // 2 + 1] = True
    one = np.zeros(m.shape, bool)
    one[nz // 2, ny // 2, nx // 2] = True
    yield "box", np.where(box, 0.1 + 0.5 * S, 0.0)
    yield "one_cell", np.where(one, 0.3, -0.0)
    yield "none", np.zeros(m.shape)
    yield "mass_only", np.where(one, 1e-50, 0.0)


def run(gpu_lib, abi, pkg, tma, case, form, S, P, steps):
    from importlib import import_module
    Domain = import_module(pkg.__name__ + ".domain").Domain
    m, media, K, phi = case
    prev = gpu_lib.gbf_set_tma(tma)
    try:
        dom = Domain(m, media, K, phi, precision=getattr(abi, FORMS[form]))
        assert gpu_lib.gbf_domain_uses_tma(dom.h) == tma
        dom.set_outputs(abi.GBF_OUT_MASS | abi.GBF_OUT_CFL, steps)
        dom.upload(P, S)
        dom.step(steps)
        out = dom.status(), dom.download("P1"), dom.download("S2"), dom.cfl_history(steps), dom.mass_history(steps)
        dom.close()
    finally:
        gpu_lib.gbf_set_tma(prev)
    return out


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("kind", ["media", "one_medium", "fields_rate", "fields_patch"])
@pytest.mark.parametrize("size", SIZES)
def test_dry_warps_equal_plain_loads(gpu_lib, abi, pkg, size, kind, form):
    m, media, K, phi, P, S0 = make(abi, gpu_lib, size, kind)
    for name, S in states(m, P, S0):
        a, b = (run(gpu_lib, abi, pkg, tma, (m, media, K, phi), form, S, P, 7) for tma in (0, 1))
        assert a[0] == b[0] == abi.GBF_OK, name
        for x, y in zip(a[1:4], b[1:4]):
            assert np.array_equal(x, y), name
        assert (a[4][:, 1] == 0).all() == (b[4][:, 1] == 0).all(), name


@pytest.mark.parametrize("form", list(FORMS))
def test_a_non_finite_pressure_in_dry_rock_is_reported(gpu_lib, abi, pkg, form):
    m, media, K, phi, P, _ = make(abi, gpu_lib, (70, 21, 24), "fields_patch")
    P[12, 10, 33] = np.inf
    a, b = (run(gpu_lib, abi, pkg, tma, (m, media, K, phi), form, np.zeros(m.shape), P, 1) for tma in (0, 1))
    gpu_lib.gbf_clear_status()
    assert a[0] == b[0] == abi.GBF_ERR_NONFINITE
    assert np.array_equal(np.isfinite(a[2]), np.isfinite(b[2])) and not np.isfinite(b[2]).all()
