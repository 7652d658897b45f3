"""The FP64 step over 10^4 steps of the laminar channel (64 cells between walls; uniform along
the walls, so two cells there are enough) against the oracle: the parity bound of the FP64
form, and the mass, which follows the rounding of the scheme's double coefficients."""
import numpy as np
import pytest

import pydugks
import pyoracle
from seeded import W, rel_err, seeded_state

pytestmark = pytest.mark.gpu


def test_laminar_channel_over_1e4_steps():
    cfg = pydugks.make_config(nx=64, ny=2, nz=2, xwidth=64, ywidth=2, zwidth=2, periods_x=0, CFL=0.5, visc=0.032,
                              ambient_fz=6.25e-6)
    eng, orc = pydugks.Engine(cfg), pyoracle.Oracle.from_config(cfg)
    f0 = np.ascontiguousarray(np.broadcast_to(W, (2, 2, 64, 19)))
    eng.set_state(f0)
    g = pyoracle.to_ghosted(f0)
    done = 0
    for upto in (1000, 10000):
        eng.run(done + 1, upto - done)
        orc.run(g, done + 1, upto - done)
        done = upto
        got, want = eng.get_state(), pyoracle.interior(g)
        # the oracle's own rounding: a walk of 2^-53 a step, 1.1e-14 after 10^4; ten times that
        assert rel_err(got, want) <= 1.1e-15 * upto ** 0.5
        assert abs(got.sum() - want.sum()) / want.sum() <= 1.1e-15 * upto ** 0.5


@pytest.mark.parametrize("kw", [
    dict(nx=16, ny=6, nz=5, xwidth=16, ywidth=6, zwidth=5, periods_x=1, visc=0.005, ambient_fz=0.0),
    # faces from a file: the engine's and the oracle's tanh differ in the last place
    dict(nx=32, ny=4, nz=3, xwidth=32, ywidth=8, zwidth=6, periods_x=0, visc=0.01, ambient_fz=1e-5, mesh="file",
         mesh_file="mesh.txt"),
], ids=["box", "stretched"])
def test_box_and_stretched_channel_over_1e4_steps(kw, tmp_path):
    t = np.tanh(1.2 * (np.arange(33) / 16.0 - 1.0))
    (tmp_path / "mesh.txt").write_text("\n".join(repr(float(x)) for x in 16.0 * (1.0 + t / t[-1])) + "\n")
    cfg = pydugks.make_config(CFL=0.5, **kw)
    eng, orc = pydugks.Engine(cfg, workdir=str(tmp_path)), pyoracle.Oracle.from_config(cfg, workdir=str(tmp_path))
    f0 = seeded_state(eng.nx, eng.ny, eng.nz, seed=3, umax=0.02, eps=0.005)
    eng.set_state(f0)
    g = pyoracle.to_ghosted(f0)
    eng.run(1, 10000)
    orc.run(g, 1, 10000)
    assert rel_err(eng.get_state(), pyoracle.interior(g)) <= 1.1e-13
