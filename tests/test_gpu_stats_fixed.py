"""Statistics with density and velocity of the cells in fixed point (stats_fx_kernel),
every form, cells out of its range among them, against numpy in extended precision."""
import numpy as np
import pytest

import pydugks
from seeded import CX, CY, CZ, seeded_state

pytestmark = pytest.mark.gpu

# sums of n values below 1 in FP64 round to a few n^(1/2) 2^-53: below 1e-13 for these grids
TOL = 1e-13


def _numpy_stats(eng):
    f = eng.get_state().astype(np.longdouble)
    info = eng.info
    rho = f.sum(-1)
    F = np.array(list(info.ambient), dtype=np.longdouble) * (0.5 * info.dt)
    u = [(f * c).sum(-1) / rho + F[a] for a, c in enumerate((CX, CY, CZ))]
    q = [rho] + u
    diag = [x.mean() for x in q] + [x.min() for x in q] + [x.max() for x in q]
    m = [x.mean((0, 1)) for x in u]
    cov = [(u[a] * u[b]).mean((0, 1)) - m[a] * m[b] for a, b in ((0, 2), (0, 1), (1, 2), (0, 0), (1, 1), (2, 2))]
    return np.array(diag, dtype=np.float64), np.stack(m + cov, -1).astype(np.float64)


# 131,072 cells and more (FP64 states below take the FP64 cells); nx across warp and block edges
@pytest.mark.parametrize("shape", [(31, 66, 65), (33, 64, 63), (257, 16, 32), (300, 23, 19)])
@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp16", "bf16"])
@pytest.mark.parametrize("odd", [False, True])
def test_statistics_match_numpy(shape, prec, odd):
    nx, ny, nz = shape
    cfg = pydugks.make_config(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, CFL=0.5, visc=0.02,
                              ambient_fx=1e-4, ambient_fy=-2e-4, ambient_fz=3e-4, precision=prec)
    eng = pydugks.Engine(cfg)
    f = seeded_state(nx, ny, nz, seed=6, umax=0.02, eps=0.005)
    if odd:  # some cells dense, some thin
        f[1, :, ::3] *= 1.9
        f[2, ::2, 1] *= 0.3
    eng.set_state(f)
    diag, prof = eng.stats_values()
    wd, wp = _numpy_stats(eng)
    assert np.abs(diag - wd).max() <= TOL
    assert np.abs(prof - wp).max() <= TOL


def test_a_non_finite_cell_is_reported():
    nx, ny, nz = 64, 48, 48
    cfg = pydugks.make_config(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, CFL=0.5, visc=0.02)
    eng = pydugks.Engine(cfg)
    f = seeded_state(nx, ny, nz, seed=7)
    f[3, 4, 5, 6] = np.inf
    eng.set_state(f)
    with pytest.raises(pydugks.DugksError) as e:
        eng.stats_values()
    assert e.value.code == pydugks.DG_ERR_NUMERIC
