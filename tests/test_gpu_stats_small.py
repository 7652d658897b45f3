"""Statistics of slow flows: velocities far below the density's scale keep the relative
precision of FP64, in every form, against exact integer moments."""
import ctypes

import numpy as np
import pytest

import pydugks
from seeded import CX, CY, CZ, W, seeded_state, uniform_sym

pytestmark = pytest.mark.gpu

# A cell's velocity is good to 2 ulp of FP64; a sum is a chain of at most 64 additions of
# values of one sign (rows of a block, blocks of a chain, chains), 2^-53 each.
CELL = 2 * 2.0 ** -52
MEAN = 64 * 2.0 ** -53 + CELL


def _state(nx, ny, nz, u0):
    n = nx * ny * nz
    u = [u0 * (1 + 0.4 * uniform_sym(8, n, s)) for s in range(3)]
    eu = sum(3 * c * x[:, None] for c, x in zip((CX, CY, CZ), u))
    return np.ascontiguousarray((W * (1 + eu)).reshape(nz, ny, nx, 19))


@pytest.mark.parametrize("prec,u0", [("fp64", 1e-4), ("fp64", 1e-7), ("fp64", 1e-10), ("fp32", 1e-4), ("fp32", 1e-5),
                                     ("fp16", 1e-3)])
@pytest.mark.parametrize("force", [0.0, 2e-9])
def test_slow_flows_keep_their_digits(prec, u0, force):
    nx, ny, nz = 64, 48, 48
    cfg = pydugks.make_config(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, CFL=0.5, visc=0.02, ambient_fx=0.0,
                              ambient_fy=force, ambient_fz=0.0, precision=prec)
    eng = pydugks.Engine(cfg)
    eng.set_state(_state(nx, ny, nz, u0))
    diag, prof = eng.stats_values()
    f = eng.get_state()
    if prec == "fp16":
        # 16-bit deviations decode to FP32 values: the populations as the statistics see them
        f = f.astype(np.float32).astype(np.float64)
    x = np.ldexp(f, 62).astype(np.int64)  # exact: 53 bits of values between 2^-6 and 1
    assert np.array_equal(np.ldexp(x.astype(np.float64), -62), f)
    rho = x.sum(-1).astype(np.longdouble)
    u = [(x * c).sum(-1).astype(np.longdouble) / rho for c in (CX, CY, CZ)]
    u[1] = u[1] + np.longdouble(eng.info.ambient[1] * (0.5 * eng.info.dt))
    assert min(abs(q).min() for q in u) > 0.2 * u0 and min(q.min() for q in u) > 0
    for a in range(3):
        want = u[a].mean((0, 1))
        assert np.abs(prof[:, a] / want - 1).max() <= MEAN
        assert abs(diag[5 + a] / u[a].min() - 1) <= CELL
        assert abs(diag[9 + a] / u[a].max() - 1) <= CELL
        # variances: <uu> and <u>^2 carry the errors of two factors each and cancel down to them
        var = (u[a] * u[a]).mean((0, 1)) - want * want
        assert np.abs(prof[:, 6 + a] - var).max() <= 4 * MEAN * float((u[a] * u[a]).max())


def test_both_entry_points_agree_where_the_cells_are_in_fixed_point():
    """dg_stats_values_noalloc has FP64 cells and one chain of sums at every size; here
    dg_stats_values has neither.  Sums of n values below 1 in any order: a few n^(1/2) 2^-53."""
    torch = pytest.importorskip("torch")
    nx, ny, nz = 65, 64, 63
    cfg = pydugks.make_config(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, CFL=0.5, visc=0.02, ambient_fz=1e-5)
    eng = pydugks.Engine(cfg)
    eng.set_state(seeded_state(nx, ny, nz, seed=6, umax=0.02, eps=0.005))
    diag, prof = eng.stats_values()
    out = torch.full((12 + 9 * nx + 1,), float("nan"), dtype=torch.float64, device="cuda")
    i = eng.info
    rc = pydugks.lib().dg_stats_values_noalloc(
        ctypes.c_void_p(eng.device_ptr(pydugks.DG_BUF_F)), nx, ny, nz, i.pitch, i.pop_stride, i.dt / 2.0, i.ambient[0],
        i.ambient[1], i.ambient[2], ctypes.c_void_p(out.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    o = out.cpu().numpy()
    assert o[-1] == 0
    assert np.abs(diag - o[:12]).max() <= 1e-13
    assert np.abs(prof - o[12:-1].reshape(nx, 9)).max() <= 1e-13
