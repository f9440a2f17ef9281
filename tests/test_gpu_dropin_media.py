"""A drop-in in split mode whose media array the caller allocated, at any
address an int can have: the same state as with a 16-byte aligned array (which
the x-pair tile reads in place), with rows of whole 16-byte units and without,
and with media rewritten between the steps."""
import ctypes
from importlib import import_module

import numpy as np
import pytest

from gpu_util import torch
from test_gpu_split_pitch import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [16, 13])
def test_media_at_any_address(gpu_lib, abi, pkg, nx):
    dp = import_module(pkg.__name__ + ".dropin")
    m, media, _, _, P, S = make(abi, gpu_lib, (nx, 9, 12), "media")
    other = np.ascontiguousarray(1 - media)
    mem = torch().empty(m.ncells + 4, dtype=torch().int32, device="cuda")
    di = dp.DropIn()
    out = []
    try:
        for offset in (0, 1, 2, 3):
            di.set_mode(2)
            c = dp.consts_from_model(m)
            H, D, buf = dp.PtrArrays(), dp.PtrArrays(), ctypes.c_void_p()
            di.f["device_memory_alloc"](ctypes.byref(D), ctypes.byref(buf), m.nx + 3, c)
            own = D.media
            D.media = mem.data_ptr() + 4 * offset
            t = 0
            for a in (media, other):
                di.f["load_data_to_device_int"](a.ctypes.data, D.media, m.nx, c)
                if t == 0:
                    di.f["load_data_to_device"](P.ctypes.data, D.P1, m.nx, c)
                    di.f["load_data_to_device"](S.ctypes.data, D.S2, m.nx, c)
                for _ in range(3):
                    t += 1
                    di.time_step(H, D, c, t * m.dt)
            assert gpu_lib.gbf_last_status() == abi.GBF_OK, offset
            assert gpu_lib.gbf_domain_uses_tma(ctypes.c_void_p(di.domain(D.P1))) == 1
            Po, So = np.empty_like(P), np.empty_like(S)
            di.f["load_data_to_host"](Po.ctypes.data, D.P1, m.nx, c)
            di.f["load_data_to_host"](So.ctypes.data, D.S2, m.nx, c)
            D.media = own
            di.f["device_memory_free"](D, buf)
            out.append((Po, So))
    finally:
        di.set_mode(0)
        gpu_lib.gbf_clear_status()
    for Po, So in out[1:]:
        assert np.array_equal(Po, out[0][0]) and np.array_equal(So, out[0][1])
