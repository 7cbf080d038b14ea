"""The records bench.py writes, without a GPU."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import bench  # noqa: E402


@pytest.mark.parametrize("fused,launches,kernel,phases", [
    (False, 2, "k_element_forces", {"predictor": 0.1, "element_forces": 2.0, "node_update": 1.0}),
    (True, 1, "k_patch_step", {"predictor": 0.1, "fused_step": 2.0})])
def test_records_name_the_kernels_that_run(fused, launches, kernel, phases):
    """one launch per step of the fused step, two otherwise, the prescribed
    motion in one of them"""
    assert bench.launches_per_step(fused) == launches
    assert bench.roofline_entry(1e9, 1.0, 6550.0, "measured", None, fused)["kernel"] == kernel
    assert bench.phases_per_step((1.0, 20.0, 10.0), 10, fused) == phases
