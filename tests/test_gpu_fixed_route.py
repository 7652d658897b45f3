"""Which kernels an FP64 step runs: the fixed-point ones with the tile rows that the other tests
name, on states in range to the end, and the FP64 ones, bit for bit, on states out of range.
A second engine that was asked for f-bar-plus steps with the FP64 kernels throughout."""
import numpy as np
import pytest

import pydugks
import test_gpu_fixed as tf
from graph_nodes import captured_kernels

pytestmark = pytest.mark.gpu


def _engines(f0=None, seed=1, **kw):
    cfg = pydugks.make_config(**dict(dict(CFL=0.6, visc=0.02, ambient_fz=0.0), **kw))
    a, b = pydugks.Engine(cfg), pydugks.Engine(cfg)
    b.device_ptr(pydugks.DG_BUF_FB)
    f0 = tf._state(a.nx, a.ny, a.nz, seed) if f0 is None else f0
    a.set_state(f0)
    b.set_state(f0)
    return a, b


def _rows(eng):
    """tile rows of the fixed-point flux kernel that a step launches, None if it launches another"""
    names = " ".join(n for n, _, _ in captured_kernels(eng, lambda: eng.step(1)))
    for r in (4, 7):
        if f"flux_fx_kernelILi{r}E" in names:
            return r
    return None


def _check(rows, n, **kw):
    a, b = _engines(**kw)
    assert _rows(a) == rows and _rows(b) is None
    a.run(1, n)
    b.run(1, n)
    # a step that is redone gives the FP64 kernels' bits (below)
    assert not np.array_equal(a.get_state(), b.get_state())


def _marks(f, name):
    return next(m.args[1] for m in f.pytestmark if m.name == "parametrize" and m.args[0] == name)


@pytest.mark.parametrize("nx,ny,nz", _marks(tf.test_edges_of_tiles, "nx,ny,nz"))
@pytest.mark.parametrize("periodic_x", [0, 1])
def test_edges_of_tiles_run_in_fixed_point(nx, ny, nz, periodic_x):
    _check(4, 3, nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, periods_x=periodic_x, ambient_fz=2e-5)


@pytest.mark.parametrize("nx,ny,nz", _marks(tf.test_edges_of_four_row_tiles, "nx,ny,nz"))
@pytest.mark.parametrize("periodic_x", [0, 1])
def test_four_row_tiles_are_chosen(nx, ny, nz, periodic_x):
    _check(4, 4, nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=1.3 * ny, zwidth=nz, periods_x=periodic_x, ambient_fy=2e-5)


@pytest.mark.parametrize("nx,ny,nz,periodic_x", _marks(tf.test_seven_row_tiles, "nx,ny,nz,periodic_x"))
def test_seven_row_tiles_are_chosen(nx, ny, nz, periodic_x):
    _check(7, 2, nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=1.1 * ny, zwidth=nz, periods_x=periodic_x, ambient_fz=2e-5)


@pytest.mark.parametrize("axis", ["x", "y", "z", None])
@pytest.mark.parametrize("mesh", ["uniform", "tanh"])
def test_force_axes_and_meshes_run_in_fixed_point(axis, mesh):
    kw = {"ambient_f" + axis: 3e-5} if axis else {}
    if mesh == "tanh":
        kw.update(mesh="tanh", mesh_alpha=0.85)
    _check(4, 20, nx=40, ny=9, nz=7, xwidth=40, ywidth=12, zwidth=10, periods_x=0, **kw)


@pytest.mark.parametrize("which", ["dense", "one cell", "thin"])
@pytest.mark.parametrize("periodic_x", [0, 1])
def test_states_out_of_range_give_the_fp64_kernels_bits(which, periodic_x):
    nx, ny, nz = 37, 10, 9
    a, b = _engines(f0=tf._odd_states(nx, ny, nz)[which], nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz,
                    periods_x=periodic_x)
    assert _rows(a) == 4
    a.step(1)
    b.step(1)
    assert np.array_equal(a.get_state(), b.get_state())


@pytest.mark.parametrize("kw", [dict(CFL=0.7), dict(recon="gradient"), dict(perturb=1), dict(ambient_fx=1e-5)],
                         ids=["dt/dx", "gradient", "perturb", "two axes"])
def test_other_parameters_keep_the_fp64_kernels(kw):
    kw = dict(dict(nx=32, ny=8, nz=6, xwidth=32, ywidth=8, zwidth=6, CFL=0.5, visc=0.02, ambient_fz=1e-5), **kw)
    eng = pydugks.Engine(pydugks.make_config(**kw))
    assert _rows(eng) is None
