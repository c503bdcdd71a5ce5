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


def _read(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def test_a_failed_call_leaves_no_error_word():
    """Every way out of a C entry by an exception ends the call's kernels and clears their
    error words, so that the next call does not report them as its own."""
    end = re.search(r"#define TN_API_END(.*?)\n\n", _read("capi.cu"), re.S).group(1)
    catches = re.split(r"catch \(", end)[1:]
    assert len(catches) == 3
    for c in catches:
        assert "_c->forget()" in c


def test_results_reach_the_host_through_the_checked_wait():
    """A modular product's error word is looked at in Ctx::sync; no entry waits for the stream
    in another way before it hands results out (two destructors wait and return nothing)."""
    assert "h_err" in re.search(r"void sync\(\) \{(.*?)\n    \}", _read("common.cuh"), re.S).group(1)
    assert "cudaStreamSynchronize" not in re.search(r"#define TN_API_END(.*?)\n\n", _read("capi.cu"), re.S).group(1)
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu") and name not in ("linalg.cu", "capi.cu"):
            assert "cudaStreamSynchronize" not in _read(name), name
    assert _read("capi.cu").count("cudaStreamSynchronize") == 2
