"""Barriers of flux_fx_kernel (csrc/fixed_kernels.cuh): its warps take different branches, one per
axis, so they meet at named barriers with a thread count (__syncthreads() is for one call site
that all threads reach)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dugks-gpu_gb300", "csrc")


def test_axis_warps_meet_at_named_barriers():
    with open(os.path.join(CSRC, "fixed_kernels.cuh")) as fh:
        text = fh.read()
    body = text[text.index(") flux_fx_kernel("):]
    body = body[:body.index("\n}\n")]
    assert "__syncthreads" not in body
    # a plane of every role: one barrier of the whole CTA on each path
    assert len(re.findall(r"fx_bar\(0, ALL\)", body)) == 6
