"""Rules that the CUDA sources keep, read from the sources themselves (no GPU)."""
from __future__ import annotations

import os

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pico-engine_b200", "csrc")


@pytest.mark.parametrize("name", ["linear_simt", "linear_fused", "linear_batch", "gemm_splitk", "attention_decode", "attention_diff"])
def test_cluster_barriers_are_of_the_form_that_lanes_may_reach_apart(name):
    """The kernels that merge ranges over a cluster come to its barrier from loops that the lanes of a warp leave at different times;
    the .aligned form is only defined where they arrive together."""
    with open(os.path.join(CSRC, name + ".cu")) as f:
        lines = [line for line in f if "barrier.cluster" in line]
    assert lines and not any(".aligned" in line for line in lines)
