"""The float forms divide by the density through the correctly rounded reciprocal: no kernel of
theirs has an approximate one of its own (the fixed-point arithmetic refines its seed)."""
import os

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dugks-gpu_gb300", "csrc")


@pytest.mark.parametrize("name", ["dugks_kernels.cuh", "flux_shared.cuh", "adjoint_kernels.cuh", "aux_kernels.cuh"])
def test_no_approximate_reciprocal(name):
    with open(os.path.join(CSRC, name)) as fh:
        text = fh.read()
    assert "rcp.approx" not in text and "__fdividef" not in text
