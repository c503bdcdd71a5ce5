"""Bounded waits in the tensor-core kernels, by their source (a wait that runs out
cannot be had on a GPU without holding it): where a whole warp waits for accumulators,
its lanes decide together, as .sync.aligned loads of tensor memory follow, and a
lane that left alone would wait at the block's last barrier for the others."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "tensornetworks.jl_gb300", "csrc")


@pytest.mark.parametrize("name,pattern", [("tc_zgemm.cu", r"mbar_wait\(&accf"), ("tc_gemm.cu", r"mbar_wait\(accf")])
def test_warps_leave_as_a_whole(name, pattern):
    with open(os.path.join(CSRC, name)) as f:
        src = f.read()
    waits = [m.start() for m in re.finditer(pattern, src)]
    assert waits
    for at in waits:
        assert src[:at].endswith("__all_sync(0xffffffffu, ")
