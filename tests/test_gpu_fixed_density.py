"""The fixed-point FP64 step at the ends of its density range (every population within
0.4 .. 1.98 of its weight), where the sums of a face's populations are largest."""
import numpy as np
import pytest

import pydugks
import pyoracle
from seeded import rel_err, seeded_state

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
