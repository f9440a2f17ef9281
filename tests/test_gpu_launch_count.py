"""gbf_domain_launches_per_step counts the kernels of a step: the kernel nodes of
a captured one, for every form of the FP64 step and its derived outputs, and
for the split step."""
import ctypes
from ctypes import c_void_p
from importlib import import_module

import pytest

from gpu_util import torch
from test_gpu_split_pitch import make

pytestmark = pytest.mark.gpu


def kernel_nodes(graph):
    cuda = ctypes.CDLL("libcuda.so.1")
    n = ctypes.c_size_t(0)
    assert cuda.cuGraphGetNodes(c_void_p(graph), None, ctypes.byref(n)) == 0
    nodes = (c_void_p * n.value)()
    assert cuda.cuGraphGetNodes(c_void_p(graph), nodes, ctypes.byref(n)) == 0
    kinds = []
    for node in nodes:
        t = ctypes.c_int(-1)
        assert cuda.cuGraphNodeGetType(c_void_p(node), ctypes.byref(t)) == 0
        kinds.append(t.value)
    return kinds.count(0)  # CU_GRAPH_NODE_TYPE_KERNEL


@pytest.mark.parametrize("outputs", ["none", "mass", "props", "velocity", "mass_arrays"])
@pytest.mark.parametrize("prec,iterations,kind", [("F64", 7, "fields_rate"), ("F64", 6, "fields_rate"),
                                                  ("SPLIT", 7, "fields_rate"), ("SPLIT", 7, "media")])
def test_count_equals_kernel_nodes(gpu_lib, abi, pkg, prec, iterations, kind, outputs):
    if prec == "SPLIT" and outputs in ("velocity", "mass_arrays"):
        pytest.skip("FP64-only outputs")
    Domain = import_module(pkg.__name__ + ".domain").Domain
    m, media, K, phi, P, S = make(abi, gpu_lib, (13, 9, 12), kind)
    m.newton_iterations = iterations
    dom = Domain(m, media, K, phi, precision=getattr(abi, "GBF_PREC_" + prec))
    flags = {"none": 0, "mass": abi.GBF_OUT_MASS, "props": abi.GBF_OUT_PROPS, "velocity": abi.GBF_OUT_VELOCITY,
             "mass_arrays": abi.GBF_OUT_MASS_ARRAYS}[outputs]
    dom.set_outputs(flags, 8)
    st = torch().cuda.Stream()
    assert gpu_lib.gbf_domain_set_stream(dom.h, c_void_p(st.cuda_stream)) == abi.GBF_OK
    dom.upload(P, S)
    dom.step(1)
    dom.sync()
    g = torch().cuda.CUDAGraph(keep_graph=True)
    with torch().cuda.graph(g, stream=st):
        dom.step(1)
    raw = g.raw_cuda_graph  # a method or a property, by torch's version
    assert dom.launches_per_step == kernel_nodes(raw() if callable(raw) else raw)
    dom.close()
