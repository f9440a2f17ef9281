"""The FP64 step's table-driven ln and 2^x (csrc/gbf_pair.cuh) on the CPU against
extended precision."""
import numpy as np
import pytest

import host_cells

extended = pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="no extended precision")


@extended
def test_table_functions(abi):
    """ln(1 - x) and 2^x to two units of FP64, 1 - 2^x to 2^-51 of 1: the tables' entries err by a unit,
    the pair polynomials by 2^-46 of the reduced part."""
    rng = np.random.default_rng(1)
    lib = host_cells.library(abi)

    def run(x, which):
        out = np.empty_like(x)
        args = [None] * 4
        args[which] = out.ctypes.data
        lib.host_pair_functions(len(x), x.ctypes.data, *args)
        return out

    F = np.longdouble
    om = np.concatenate([rng.uniform(-0.25, 0.9995, 200000), 1 - 2.0 ** -rng.uniform(0, 10.9, 50000),
                         10.0 ** -rng.uniform(0.7, 300, 50000), -(10.0 ** -rng.uniform(0.7, 300, 50000))])
    want = np.log1p(-om.astype(F))
    assert np.abs((run(om, 0) - want) / want).max() <= 2.0 ** -51
    u = np.concatenate([rng.uniform(-260, 110, 200000), rng.uniform(-1, 0.4, 100000), 10.0 ** -rng.uniform(2.8, 30, 50000) * -1])
    want = np.exp2(u.astype(F))
    assert np.abs(run(u, 1) / want - 1).max() <= 2.0 ** -51
    v = u[u < 0.5]
    want = -np.expm1(v.astype(F) * np.log(F(2)))
    assert np.abs(run(v, 2) - want).max() <= 2.0 ** -51
