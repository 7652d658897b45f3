"""The fixed-point FP64 step at the ends of its density range (every population within
0.4 .. 1.98 of its weight), where the sums of a face's populations are largest."""
import numpy as np
import pytest

import pydugks
import pyoracle
from seeded import W, rel_err, seeded_state, uniform_sym

pytestmark = pytest.mark.gpu

TOL = 1e-12  # the FP64 parity bound


# densities within 2 % of the scale; between walls the ghost columns deviate three times as far
@pytest.mark.parametrize("scale,periodic_x", [(0.45, 1), (0.5, 0), (1.45, 0), (1.55, 0), (1.7, 0), (1.55, 1), (1.9, 1)])
@pytest.mark.parametrize("mesh", ["uniform", "tanh"])
def test_densities_within_the_range(scale, periodic_x, mesh):
    if mesh == "tanh" and periodic_x:
        pytest.skip("the stretched mesh is for walls")
    kw = dict(mesh="tanh", mesh_alpha=0.85) if mesh == "tanh" else {}
    nx, ny, nz = 40, 9, 7
    cfg = pydugks.make_config(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=12, zwidth=10, periods_x=periodic_x, CFL=0.5,
                              visc=0.02, ambient_fz=2e-5, **kw)
    eng, orc = pydugks.Engine(cfg), pyoracle.Oracle.from_config(cfg)
    f0 = scale * seeded_state(nx, ny, nz, seed=3, umax=0.003, eps=0.001)
    eng.set_state(f0)
    eng.run(1, 3)
    g = pyoracle.to_ghosted(f0)
    orc.run(g, 1, 3)
    assert rel_err(eng.get_state(), pyoracle.interior(g)) <= TOL


@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("pattern", ["random", "high and low"])
def test_populations_across_the_whole_box(pattern, seed):
    """Every population anywhere between 0.42 and 1.96 of its weight, or at either end; viscous, so
    that f-bar-plus stays near f-tilde and in the box."""
    nx, ny, nz = 33, 9, 6
    cfg = pydugks.make_config(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, periods_x=1, CFL=0.5, visc=20.0,
                              ambient_fz=1e-4)
    eng, fp64, orc = pydugks.Engine(cfg), pydugks.Engine(cfg), pyoracle.Oracle.from_config(cfg)
    fp64.device_ptr(pydugks.DG_BUF_FB)  # keeps f-bar-plus, and with it the step, in FP64
    r = uniform_sym(seed, nx * ny * nz * 19, 0).reshape(nz, ny, nx, 19)
    if pattern != "random":
        r = np.where(r > 0, 1.0, -1.0)
    f0 = W * (1.19 + 0.77 * r)
    eng.set_state(f0)
    fp64.set_state(f0)
    eng.step(1)
    fp64.step(1)
    got = eng.get_state()
    g = pyoracle.to_ghosted(f0)
    orc.run(g, 1, 1)
    assert not np.array_equal(got, fp64.get_state())  # in range: not redone
    assert rel_err(got, pyoracle.interior(g)) <= TOL
