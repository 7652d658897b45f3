"""Ghosts of the periodic 16-bit forms, written by stage (a) with the cells.

With rounding to nearest a step on a uniform periodic box does not depend on where the
box is cut: a state rolled in y and z gives the rolled result, value for value.  Rolled in x
the face between columns nx and 1 takes its two weights in the other order (FP32 rounding,
which may tip a stored value by one quantum per step): two quanta of the largest deviation
after two steps.
"""
import numpy as np
import pytest

import pydugks
from seeded import seeded_state

pytestmark = pytest.mark.gpu

QUANT = {"fp16": 2.0 ** -11, "bf16": 2.0 ** -8}
W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


@pytest.mark.parametrize("prec", ["fp16", "bf16"])
@pytest.mark.parametrize("nx,ny,nz", [(3, 2, 2), (20, 1, 3), (31, 4, 1), (32, 5, 3), (33, 8, 9), (129, 3, 2)])
def test_the_cut_of_the_box_does_not_matter(prec, nx, ny, nz):
    eng = pydugks.Engine(pydugks.make_config(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, periods_x=1, CFL=0.5,
                                             visc=0.02, ambient_fz=1e-5, precision=prec, rounding="nearest"))
    f0 = seeded_state(nx, ny, nz, seed=8)

    def run(f):
        eng.set_state(f)
        eng.run(1, 2)
        return eng.get_state()

    ref = run(f0)
    assert np.array_equal(run(np.roll(f0, (1, 1), axis=(0, 1))), np.roll(ref, (1, 1), axis=(0, 1)))
    dev = np.max(np.abs(f0 - W) / W)
    x = run(np.roll(f0, 1, axis=2)) - np.roll(ref, 1, axis=2)
    assert np.max(np.abs(x) / W) <= 2 * QUANT[prec] * dev
