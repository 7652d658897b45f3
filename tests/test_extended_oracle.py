"""The extended-precision instance of the oracle, and with it the error of the FP64 forms of the
step against the double scheme without the rounding of its arithmetic."""
import numpy as np
import pytest

import pydugks
import pyoracle
from seeded import seeded_state

FLOWS = {
    "channel": dict(nx=24, ny=5, nz=4, xwidth=24, ywidth=5, zwidth=4, periods_x=0, visc=0.032, ambient_fz=6.25e-6),
    "box": dict(nx=10, ny=8, nz=7, xwidth=10, ywidth=8, zwidth=7, periods_x=1, visc=0.005, ambient_fz=0.0),
}


def _flow(name):
    cfg = pydugks.make_config(CFL=0.5, **FLOWS[name])
    orc = pyoracle.Oracle.from_config(cfg)
    f0 = seeded_state(orc.cfg.nx, orc.cfg.ny, orc.cfg.nz, seed=3, umax=0.02, eps=0.005)
    return cfg, orc, f0


def _distance(f, x):
    """relative 2-norm of f - x"""
    return float(np.linalg.norm((f - x).astype(np.float64)) / np.linalg.norm(x.astype(np.float64)))


def _extended(orc, f0, n):
    g = np.ascontiguousarray(pyoracle.to_ghosted(f0).astype(np.longdouble))
    return pyoracle.interior(orc.run_extended(g, 1, n))


@pytest.mark.parametrize("name", sorted(FLOWS))
def test_double_oracle_rounds_around_it(name):
    _, orc, f0 = _flow(name)
    for n in (1, 100):
        x, g = _extended(orc, f0, n), pyoracle.to_ghosted(f0)
        orc.run(g, 1, n)
        # a few roundings of 2^-53 a step, walking as n^(1/2)
        assert 0 < _distance(pyoracle.interior(g), x) <= 8 * 2.0 ** -53 * n ** 0.5


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(FLOWS))
def test_fixed_point_step_is_no_further_from_it_than_the_fp64_kernels(name):
    cfg, orc, f0 = _flow(name)
    fixed, fp64 = pydugks.Engine(cfg), pydugks.Engine(cfg)
    fp64.device_ptr(pydugks.DG_BUF_FB)  # keeps f-bar-plus, and with it the step, in FP64
    fixed.set_state(f0)
    fp64.set_state(f0)
    done = 0
    for n in (1, 100):
        fixed.run(done + 1, n - done)
        fp64.run(done + 1, n - done)
        done = n
        x = _extended(orc, f0, n)
        a, b = _distance(fixed.get_state(), x), _distance(fp64.get_state(), x)
        print(f"{name}, {n} steps: fixed point {a:.2e}, FP64 kernels {b:.2e}")
        assert a <= b
        # the rounding of the stored values, 2^-54 on average, once a step
        assert a <= 2.0 ** -53 * n ** 0.5
