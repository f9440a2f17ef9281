"""bench.py's algorithmic bytes of the split step are those of the timed states, which hold no
DNAPL but at a source: not above the DRAM traffic that the profiles measured on
such states (1% for what stays in L2 from one launch to the next)."""
import json
import pathlib
import sys

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))
TRAFFIC = json.loads((ROOT / "profiles" / "traffic.json").read_text())


@pytest.mark.parametrize("workload,kernel", [(w, k) for w, e in TRAFFIC.items() for k in e if k == "ensemble_step"])
def test_algorithmic_bytes_are_at_most_the_measured_traffic(workload, kernel):
    import bench
    ent = TRAFFIC[workload][kernel]
    bpc, which = bench.algo_bytes(workload.split("_")[1], kernel)
    assert which == ent["cells"] and 0 < bpc <= 1.01 * ent["bytes_per_cell"], (bpc, ent)
