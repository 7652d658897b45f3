"""The fixed-point arithmetic of the FP64 step (csrc/fixed_kernels.cuh), compiled for
the host: stage (a) and the face flux over the whole range that the GPU kernels accept
are no further from quadruple precision than the same formulas in double."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fixed") / "fixed_check")
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-fwrapv", "-o", exe, os.path.join(HERE, "fixed_check.cpp")], check=True)
    return exe


# (viscosity, time step, force): the laminar channel, the Re_tau = 180 channel, the
# Taylor-Green box, a viscous and a small-step case
@pytest.mark.parametrize("visc,dt,force", [(0.166, 0.49, 3e-5), (0.00227, 0.126, 1e-6), (3.18e-4, 0.3535, 1e-4),
                                           (1.0, 0.35, 1e-3), (0.05, 0.01, 1e-4)])
def test_fixed_point_is_no_less_exact_than_double(checker, visc, dt, force):
    out = subprocess.run([checker, str(visc), str(dt), str(force)], check=True, capture_output=True, text=True).stdout
    rows = [r.split() for r in out.splitlines()]
    assert [r[0] for r in rows] == ["0", "1", "2", "3"]  # force along x, y, z and none
    for r in rows:
        for k in range(1, len(r), 3):
            fixed, double = float(r[k + 1]), float(r[k + 2])
            assert fixed <= double, f"axis {r[0]} {r[k]}: {fixed} against {double} (units of 2^-62)"
