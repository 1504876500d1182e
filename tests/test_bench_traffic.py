"""The bench line's DRAM traffic is the running stage kernel's own."""
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


@pytest.mark.parametrize("kernel,precision,source", [("tile", "fp64", "k_stage_split"), ("tile", "mixed", "k_stage_split"),
                                                     ("lane", "fp64", "k_stage_ausm")])
def test_traffic_of_a_captured_kernel(kernel, precision, source):
    d = json.load(open(os.path.join(ROOT, "profiles", "stage2_traffic.json")))
    e = d["kernels"][kernel]
    assert e["kernel"] == source and source in e[precision]["source"]
    t = bench.stage2_traffic(kernel, precision, 1000)
    assert t == 1000 * e[precision]["dram_bytes_per_leaf_cell"]
    # lhs, rhs and tables once each are 145 bytes; some of it is still in the L2 from the stage before
    assert 0.8 * 145 < t / 1000 < 1.2 * 145


@pytest.mark.parametrize("kernel,precision", [("warp", "fp64"), ("lane", "mixed"), ("per_cell", "fp64")])
def test_no_traffic_for_a_kernel_that_was_not_captured(kernel, precision):
    assert bench.stage2_traffic(kernel, precision, 1000) is None
