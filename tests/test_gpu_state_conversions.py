"""FP64 state <-> split state conversions (integer bit-field arithmetic on the
device) against numpy's, bit for bit: an upload followed by a download gives
P_hs(j) + (float)(P - P_hs(j)) and (double)(float)S. Values: ties and
near-ties of the FP32 rounding, results that are subnormal in FP32 or round up
to a normal, both zeros, carries into the exponent; sizes of one cell beyond a
block's cells, below one, and odd rows. g h2 rho01 is a power of two times an
integer here, so that P_hs is exact and its rounding is not at issue."""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def state(m, seed):
    rng = np.random.default_rng(seed)
    j = np.arange(m.ny, dtype=np.float64)[None, :, None]
    phs = np.broadcast_to(m.P_atm + j * 1024.0, m.shape)

    def awkward(scale):
        """FP64 numbers at and next to the ties of FP32, and of every size."""
        f = (scale * rng.normal(0, 1, m.shape)).astype(np.float32)
        ulp = np.spacing(np.abs(f)).astype(np.float64)
        d = f.astype(np.float64) + ulp * rng.choice([0, 0.5, 0.25, -0.5], m.shape)
        d = np.where(rng.random(m.shape) < 0.3, np.nextafter(d, rng.choice([-1e300, 1e300], m.shape)), d)
        return d

    P = phs + awkward(300.0)
    S = np.abs(awkward(0.2)).clip(0, 0.8)
    pick = rng.random(m.shape)
    for q, v in enumerate([0.0, -0.0, 1e-40, 2.0 ** -149 * 1.5, 2.0 ** -126 * (1 - 2.0 ** -25), 2.0 ** -130, 1e-320, 1e-25,
                           0.25 - 2.0 ** -27]):
        S[(pick > 0.05 * q) & (pick < 0.05 * (q + 1))] = v
    return phs, P, S


@pytest.mark.parametrize("form", ["GBF_PREC_SPLIT", "GBF_PREC_SPLIT_DF", "GBF_PREC_SPLIT_DEFECT"])
@pytest.mark.parametrize("size", [(3, 3, 3), (5, 5, 41), (31, 3, 11), (67, 31, 33)])
def test_upload_download_equals_numpy(gpu_lib, abi, pkg, size, form):
    from importlib import import_module
    Domain = import_module(pkg.__name__ + ".domain").Domain
    Ensemble = import_module(pkg.__name__ + ".ensemble").Ensemble
    m = abi.reference_model(*size, 1e-6)
    m.ro01, m.g, m.h2, m.source = 1024.0, 8.0, 0.125, 0
    phs, P, S = state(m, sum(size))
    want_P = phs + (P - phs).astype(np.float32).astype(np.float64)
    want_S = S.astype(np.float32).astype(np.float64)

    def same(got, want):
        assert np.array_equal(got.view(np.uint64), np.ascontiguousarray(want).view(np.uint64))

    dom = Domain(m, precision=getattr(abi, form))
    dom.upload(P, S)
    same(dom.download("P1"), want_P)
    same(dom.download("S2"), want_S)
    dom.close()
    mems = [types.SimpleNamespace(model=m)] * 2
    ens = Ensemble(mems, precision=getattr(abi, form))
    Pa, Sa = np.concatenate([P.ravel()] * 2), np.concatenate([S.ravel()] * 2)
    ens.upload_all(Pa, Sa)
    Po, So = np.empty_like(Pa), np.empty_like(Sa)
    ens.download_all(Po, So)
    same(Po, np.concatenate([want_P.ravel()] * 2))
    same(So, np.concatenate([want_S.ravel()] * 2))
    ens.close()
