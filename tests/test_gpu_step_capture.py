"""A caller's CUDA graph of a domain's steps: captured on the domain's stream and
replayed, it advances the state as plain steps do, bit for bit."""
import numpy as np
import pytest

from test_gpu_split_pitch import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["GBF_PREC_F64", "GBF_PREC_SPLIT"])
@pytest.mark.parametrize("size", [(13, 9, 12), (70, 21, 24)])
def test_captured_steps_equal_plain_steps(gpu_lib, abi, pkg, size, prec):
    from ctypes import c_void_p
    from importlib import import_module
    torch = pytest.importorskip("torch")
    Domain = import_module(pkg.__name__ + ".domain").Domain
    m, media, K, phi, P, S = make(abi, gpu_lib, size, "fields_rate")
    out = []
    for graph in (False, True):
        dom = Domain(m, media, K, phi, precision=getattr(abi, prec))
        st = torch.cuda.Stream()
        assert gpu_lib.gbf_domain_set_stream(dom.h, c_void_p(st.cuda_stream)) == abi.GBF_OK
        dom.upload(P, S)
        dom.step(2)
        dom.sync()
        if graph:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st):
                dom.step(2)
            with torch.cuda.stream(st):
                for _ in range(3):
                    g.replay()
        else:
            dom.step(6)
        dom.sync()
        assert dom.status() == abi.GBF_OK
        out.append((dom.download("P1"), dom.download("S2")))
        dom.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
