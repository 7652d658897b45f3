"""The fixed-point FP64 step: tile and chunk edges, every force axis, and states
outside its range, which the FP64 kernels take over."""
import numpy as np
import pytest

import pydugks
import pyoracle
from seeded import rel_err, seeded_state

pytestmark = pytest.mark.gpu

TOL = 1e-12  # the FP64 parity bound


def _state(nx, ny, nz, seed):
    """In range, wall ghosts (extrapolated from two cells) included."""
    return seeded_state(nx, ny, nz, seed=seed, umax=0.02, eps=0.005)


def _pair(seed=1, f0=None, **kw):
    cfg = pydugks.make_config(**dict(dict(CFL=0.6, visc=0.02, ambient_fz=0.0), **kw))
    eng, orc = pydugks.Engine(cfg), pyoracle.Oracle.from_config(cfg)
    f0 = _state(eng.nx, eng.ny, eng.nz, seed) if f0 is None else f0
    eng.set_state(f0)
    return eng, orc, f0


def _oracle(orc, f0, n):
    g = pyoracle.to_ghosted(f0)
    orc.run(g, 1, n)
    return pyoracle.interior(g)


@pytest.mark.parametrize("nx,ny,nz", [(3, 1, 1), (16, 2, 3), (31, 7, 5), (32, 8, 2), (33, 14, 9), (63, 15, 4),
                                      (64, 6, 17), (65, 11, 6), (97, 23, 3)])
@pytest.mark.parametrize("periodic_x", [0, 1])
def test_edges_of_tiles(nx, ny, nz, periodic_x):
    eng, orc, f0 = _pair(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, periods_x=periodic_x, ambient_fz=2e-5)
    eng.run(1, 3)
    assert rel_err(eng.get_state(), _oracle(orc, f0, 3)) <= TOL


@pytest.mark.parametrize("nx,ny,nz", [(5, 3, 2), (31, 4, 1), (32, 5, 3), (33, 9, 16), (65, 13, 2), (40, 4, 33)])
@pytest.mark.parametrize("periodic_x", [0, 1])
def test_edges_of_four_row_tiles(nx, ny, nz, periodic_x):
    """Tiles of four rows with warps per axis; z chunks of unequal length; the FP64 parity bound."""
    eng, orc, f0 = _pair(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=1.3 * ny, zwidth=nz, periods_x=periodic_x,
                         ambient_fy=2e-5)
    eng.run(1, 4)
    assert rel_err(eng.get_state(), _oracle(orc, f0, 4)) <= TOL


@pytest.mark.parametrize("nx,ny,nz,periodic_x", [(63, 133, 80, 0), (96, 126, 96, 1), (160, 129, 64, 0)])
def test_seven_row_tiles(nx, ny, nz, periodic_x):
    """Grids whose planes the flux kernel takes seven rows at a time, with ragged last tiles; the FP64 parity bound."""
    eng, orc, f0 = _pair(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=1.1 * ny, zwidth=nz, periods_x=periodic_x,
                         ambient_fz=2e-5)
    eng.run(1, 2)
    assert rel_err(eng.get_state(), _oracle(orc, f0, 2)) <= TOL


@pytest.mark.parametrize("axis", ["x", "y", "z", None])
@pytest.mark.parametrize("mesh", ["uniform", "tanh"])
def test_force_axes_and_meshes(axis, mesh):
    kw = {"ambient_f" + axis: 3e-5} if axis else {}
    if mesh == "tanh":
        kw.update(mesh="tanh", mesh_alpha=0.85)
    eng, orc, f0 = _pair(nx=40, ny=9, nz=7, xwidth=40, ywidth=12, zwidth=10, periods_x=0, **kw)
    eng.run(1, 20)
    assert rel_err(eng.get_state(), _oracle(orc, f0, 20)) <= TOL


def _odd_states(nx, ny, nz):
    f = _state(nx, ny, nz, 4)
    dense = 3.0 * f                    # every cell out of range
    one = f.copy()
    one[nz // 2, ny // 2, nx // 2] *= 2.2  # one cell
    thin = 0.05 * f
    return {"dense": dense, "one cell": one, "thin": thin}


@pytest.mark.parametrize("which", ["dense", "one cell", "thin"])
@pytest.mark.parametrize("periodic_x", [0, 1])
def test_states_out_of_range_take_the_fp64_kernels(which, periodic_x):
    nx, ny, nz = 37, 10, 9
    kw = dict(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, periods_x=periodic_x)
    eng, orc, f0 = _pair(f0=_odd_states(nx, ny, nz)[which], **kw)
    eng.run(1, 18)  # graph-replayed and single steps
    got = eng.get_state()
    assert rel_err(got, _oracle(orc, f0, 18)) <= TOL
    # back in range: the next steps agree with the oracle again
    f1 = _state(nx, ny, nz, 9)
    eng.set_state(f1)
    eng.run(1, 2)
    assert rel_err(eng.get_state(), _oracle(orc, f1, 2)) <= TOL


def test_non_finite_cells_spread_as_in_fp64():
    nx, ny, nz = 20, 9, 8
    kw = dict(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, periods_x=1)
    f0 = _state(nx, ny, nz, 2)
    f0[4, 4, 10, 7] = np.nan
    a, _, _ = _pair(f0=f0, **kw)
    b, _, _ = _pair(f0=f0, **kw)
    b.device_ptr(pydugks.DG_BUF_FB)  # keeps f-bar-plus, and with it the step, in FP64
    a.run(1, 2)
    b.run(1, 2)
    x, y = a.get_state(), b.get_state()
    assert np.isnan(x).any() and np.array_equal(np.isnan(x), np.isnan(y))
    assert np.allclose(x, y, rtol=1e-14, atol=0, equal_nan=True)


@pytest.mark.parametrize("scale", [1.0, 3.0])  # the second: redone in FP64
def test_f_bar_plus_is_shown_in_fp64(scale):
    torch = pytest.importorskip("torch")
    nx, ny, nz = 37, 10, 9
    eng, orc, f0 = _pair(f0=scale * _state(37, 10, 9, 1), nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, periods_x=0, ambient_fz=1e-5)
    want = pyoracle.interior(orc.fbar(pyoracle.to_ghosted(f0)))
    eng.step(1)
    pitch = (nx + 2 + 15) // 16 * 16
    ps = (pitch * (ny + 2) * (nz + 2) + 31) // 32 * 32

    def interior():
        class Buf:
            __cuda_array_interface__ = {"shape": (19 * ps,), "typestr": "<f8", "strides": None, "version": 3,
                                        "data": (eng.device_ptr(pydugks.DG_BUF_FB), False)}
        eng.sync()
        t = torch.as_tensor(Buf(), device="cuda").view(19, ps)[:, :pitch * (ny + 2) * (nz + 2)]
        t = t.reshape(19, nz + 2, ny + 2, pitch)[:, 1:-1, 1:-1, 1:nx + 1]
        return t.permute(1, 2, 3, 0).cpu().numpy()

    assert rel_err(interior(), want) <= TOL           # of the fixed-point step
    f1 = eng.get_state()
    want = pyoracle.interior(orc.fbar(pyoracle.to_ghosted(f1)))
    eng.step(2)
    assert rel_err(interior(), want) <= TOL           # of the steps from here on
    assert rel_err(eng.get_state(), _oracle(orc, f0, 2)) <= TOL
