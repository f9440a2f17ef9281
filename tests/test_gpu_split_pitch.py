"""The x-pair TMA tile on grids it used not to take (rows that are not whole
16-byte units, the media table, a single medium) against the plain-load tile:
the same bits of P and S, the same CFL numbers, phase masses up to the
summation order. Sizes at the tile's edges: one interior cell, an odd and an
even last column, one column beyond a 64-wide tile, several tiles and k chunks;
every split form, both sources, with and without media indices."""
import ctypes

import numpy as np
import pytest

from gpu_util import mass_order_rtol

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (4, 5, 3), (5, 4, 6), (7, 11, 20), (62, 6, 5), (65, 9, 4), (66, 10, 7), (67, 19, 5), (131, 12, 40)]
FORMS = {"split": "GBF_PREC_SPLIT", "split_df": "GBF_PREC_SPLIT_DF", "split_defect": "GBF_PREC_SPLIT_DEFECT"}


def make(abi, lib, size, kind):
    nx, ny, nz = size
    rng = np.random.default_rng(nx * 1009 + ny * 31 + nz)
    m = abi.reference_model(nx, ny, nz, 1.0)
    media = K = phi = None
    if kind != "one_medium":
        m.K[:], m.S_wr[:], m.lam[:] = [6.64e-11, 7.15e-12], [0.09, 0.12], [2.7, 2.0]
    if kind.startswith("fields"):
        K = (6.64e-11 * np.exp(rng.normal(0, 1, m.shape))).astype(np.float32)
        phi = (0.35 + 0.05 * rng.uniform(-1, 1, m.shape)).astype(np.float32)
    elif kind == "media":
        media = (rng.random(m.shape) < 0.4).astype(np.int32)
    if kind in ("fields_rate", "one_medium"):
        m.source_mode, m.rate_cells, m.rate = abi.GBF_SOURCE_RATE, 1, 1e-3
        m.bc_mode, m.kv = abi.GBF_BC_HYDROSTATIC_SIDES, 0.6
    else:
        m.source = (min(nx, nz) - 1) // 4
    cells = abi.GbfCells()
    for name, a, ct in (("media", media, ctypes.c_int), ("K", K, ctypes.c_float), ("phi", phi, ctypes.c_float)):
        if a is not None:
            setattr(cells, name, a.ctypes.data_as(ctypes.POINTER(ct)))
    m.dt = 0.3 * lib.gbf_stable_dt(ctypes.byref(m), ctypes.byref(cells), 1.0)
    j = np.arange(ny)[None, :, None]
    P = m.P_atm + j * m.ro01 * m.g * m.h2 + rng.normal(0, 50, m.shape)
    S = np.where(rng.random(m.shape) < 0.4, 0.0, 0.6 * rng.random(m.shape))
    return m, media, K, phi, P, S


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("kind", ["media", "one_medium", "fields_rate", "fields_patch"])
@pytest.mark.parametrize("size", SIZES)
def test_pitched_and_table_tiles_equal_plain_loads(gpu_lib, abi, pkg, size, kind, form):
    from importlib import import_module
    Domain = import_module(pkg.__name__ + ".domain").Domain
    m, media, K, phi, P, S = make(abi, gpu_lib, size, kind)
    steps, out = 5, []
    prev = gpu_lib.gbf_set_tma(-1)
    try:
        for tma in (0, 1):
            gpu_lib.gbf_set_tma(tma)
            dom = Domain(m, media, K, phi, precision=getattr(abi, FORMS[form]))
            assert gpu_lib.gbf_domain_uses_tma(dom.h) == tma
            dom.set_outputs(abi.GBF_OUT_MASS | abi.GBF_OUT_CFL, steps)
            dom.upload(P, S)
            dom.step(steps)
            assert dom.status() == abi.GBF_OK
            out.append((dom.download("P1"), dom.download("S2"), dom.cfl_history(steps), dom.mass_history(steps)))
            dom.close()
    finally:
        gpu_lib.gbf_set_tma(prev)
    (P0, S0, c0, m0), (P1, S1, c1, m1) = out
    assert np.array_equal(S1, S0) and np.array_equal(P1, P0) and np.array_equal(c1, c0)
    rtol = mass_order_rtol(form, 1e-12)
    if form == "split_defect":  # its FP32 sums of phi D round at 2^-24 |D| each way, |D| / M up to beta |P - P_hs|
        j = np.arange(m.ny)[None, :, None]
        rtol += 2.0 ** -23 * m.beta1 * np.abs(P - m.P_atm - j * m.ro01 * m.g * m.h2).max()
    assert (np.abs(m1 - m0).max(0) <= rtol * np.abs(m0).max()).all()


def test_plots_and_checkpoint_of_a_padded_grid(gpu_lib, abi, pkg, tmp_path):
    """What reads the split state beside the step, on rows with padding: the
    checkpoint (start-of-step masses) and the plot files equal those of the
    unpadded grid."""
    from importlib import import_module
    Domain = import_module(pkg.__name__ + ".domain").Domain
    m, media, K, phi, P, S = make(abi, gpu_lib, (7, 11, 20), "media")
    prev = gpu_lib.gbf_set_tma(-1)
    files = []
    try:
        for tma in (0, 1):
            gpu_lib.gbf_set_tma(tma)
            dom = Domain(m, media, precision=abi.GBF_PREC_SPLIT)
            dom.upload(P, S)
            dom.step(3)
            d = tmp_path / str(tma)
            d.mkdir()
            dom.save(d / "save.dat", 3)
            dom.write_plots(d, 0.5)
            files.append({p.relative_to(d): p.read_bytes() for p in sorted(d.rglob("*")) if p.is_file()})
            dom.close()
    finally:
        gpu_lib.gbf_set_tma(prev)
    assert files[0] == files[1] and len(files[0]) >= 6


def test_dropin_split_rereads_media_of_a_padded_grid(gpu_lib, abi, pkg):
    """A media array rewritten between steps reaches the drop-in's padded copy:
    the same state as with the plain-load tile, which reads it in place."""
    from importlib import import_module
    dp = import_module(pkg.__name__ + ".dropin")
    m, media, _, _, P, S = make(abi, gpu_lib, (13, 9, 12), "media")
    other = np.ascontiguousarray(1 - media)
    out = []
    prev = gpu_lib.gbf_set_tma(-1)
    di = dp.DropIn()
    try:
        for tma in (0, 1):
            gpu_lib.gbf_set_tma(tma)
            di.set_mode(2)
            c = dp.consts_from_model(m)
            H, D, buf = dp.PtrArrays(), dp.PtrArrays(), ctypes.c_void_p()
            di.f["device_memory_alloc"](ctypes.byref(D), ctypes.byref(buf), m.nx + 3, c)
            di.f["load_data_to_device_int"](media.ctypes.data, D.media, m.nx, c)
            di.f["load_data_to_device"](P.ctypes.data, D.P1, m.nx, c)
            di.f["load_data_to_device"](S.ctypes.data, D.S2, m.nx, c)
            for s in range(1, 4):
                di.time_step(H, D, c, s * m.dt)
            di.f["load_data_to_device_int"](other.ctypes.data, D.media, m.nx, c)
            for s in range(4, 7):
                di.time_step(H, D, c, s * m.dt)
            Po, So = np.empty_like(P), np.empty_like(S)
            di.f["load_data_to_host"](Po.ctypes.data, D.P1, m.nx, c)
            di.f["load_data_to_host"](So.ctypes.data, D.S2, m.nx, c)
            di.f["device_memory_free"](D, buf)
            out.append((Po, So))
    finally:
        di.set_mode(0)
        gpu_lib.gbf_set_tma(prev)
    assert gpu_lib.gbf_last_status() == abi.GBF_OK
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
