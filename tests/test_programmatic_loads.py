"""Kernels launched with programmatic stream serialization are resident while
the kernel before them writes: the non-coherent loads (__ldg, ld.global.nc, or
what __restrict__ lets the compiler make of a load) are for data that no kernel
of a step writes. Read off the sources of those kernels."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "shmem-cuda-filtration_gb300" / "csrc"
SOURCES = ["gbf_internal.h", "gbf_pair.cuh", "gbf_f64.cu", "gbf_f64_cell.cuh", "gbf_f64_pair.cuh", "gbf_split.cu",
           "gbf_split.h", "gbf_split_tile.cuh", "gbf_split_x2.cuh"]
# the cells' media, permeability and porosity, and the tables of ln and 2^x
READ_ONLY = re.compile(r"(cells|G)\.(media|K|phi) \+|&t->lnc|reinterpret_cast<const float2\*>\(t\)|&g_pf_tab\.")


def test_noncoherent_loads_are_of_data_that_no_step_writes():
    seen = 0
    for name in SOURCES:
        text = (CSRC / name).read_text()
        assert "ld.global.nc" not in text and "__restrict__" not in text, name
        for arg in re.findall(r"__ldg\((.*)", text):
            seen += 1
            assert READ_ONLY.match(arg), (name, arg)
    assert seen
