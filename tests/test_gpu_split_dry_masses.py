"""Phase masses of the x-pair tile's shorter update of warps without DNAPL
against the plain-load tile's, by value, for every state of test_gpu_split_dry
(rock without DNAPL among them) and every mass form and kind of cell fields, at
test_gpu_split_pitch's tolerance."""
import numpy as np
import pytest

from gpu_util import mass_order_rtol
from test_gpu_split_dry import SIZES, run, states
from test_gpu_split_pitch import FORMS, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("kind", ["media", "one_medium", "fields_rate", "fields_patch"])
@pytest.mark.parametrize("size", SIZES)
def test_masses_of_dry_warps(gpu_lib, abi, pkg, size, kind, form):
    m, media, K, phi, P, S0 = make(abi, gpu_lib, size, kind)
    rtol = mass_order_rtol(form, 1e-12)
    if form == "split_defect":  # its FP32 sums of phi D round at 2^-24 |D| each way, |D| / M up to beta |P - P_hs|
        j = np.arange(m.ny)[None, :, None]
        rtol += 2.0 ** -23 * m.beta1 * np.abs(P - m.P_atm - j * m.ro01 * m.g * m.h2).max()
    for name, S in states(m, P, S0):
        a, b = (run(gpu_lib, abi, pkg, tma, (m, media, K, phi), form, S, P, 7)[4] for tma in (0, 1))
        assert (np.abs(b - a).max(0) <= rtol * np.abs(a).max()).all(), name
