"""dg_device_ptr(DG_BUF_FB) of an FP64 handle that steps in fixed point: a query that neither
waits nor needs the stream free, with f-bar-plus in FP64 from there on."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import pydugks
import pyoracle
from seeded import rel_err, seeded_state

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
TOL = 1e-12
N = (37, 10, 9)


def _pair(nx, ny, nz, **kw):
    cfg = pydugks.make_config(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, CFL=0.5, visc=0.02, **kw)
    eng, orc = pydugks.Engine(cfg), pyoracle.Oracle.from_config(cfg)
    f0 = seeded_state(nx, ny, nz, seed=4, umax=0.02, eps=0.005)
    eng.set_state(f0)
    return eng, orc, f0


def _fb(eng, ptr):
    """f-bar-plus at ptr, ghosts included, [k][j][i][p]"""
    nx, ny, nz = eng.nx, eng.ny, eng.nz
    pitch = (nx + 2 + 15) // 16 * 16
    ps = (pitch * (ny + 2) * (nz + 2) + 31) // 32 * 32

    class Buf:
        __cuda_array_interface__ = {"shape": (19 * ps,), "typestr": "<f8", "strides": None, "version": 3,
                                    "data": (ptr, False)}
    torch.cuda.synchronize()
    t = torch.as_tensor(Buf(), device="cuda").view(19, ps)[:, :pitch * (ny + 2) * (nz + 2)]
    return t.reshape(19, nz + 2, ny + 2, pitch)[..., :nx + 2].permute(1, 2, 3, 0).cpu().numpy()


def _capture(eng, call):
    g = torch.cuda.CUDAGraph()
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    out = []
    with torch.cuda.graph(g, stream=st):
        eng.set_stream(torch.cuda.current_stream().cuda_stream)
        out.append(call())
    eng.set_stream(0)
    return g, out[0]


@pytest.mark.parametrize("periodic_x", [0, 1])
@pytest.mark.parametrize("ny,nz", [(10, 9), (1, 3), (2, 1)])
def test_conversion_with_its_ghosts(periodic_x, ny, nz):
    eng, orc, f0 = _pair(37, ny, nz, periods_x=periodic_x, ambient_fz=1e-5)
    eng.step(1)
    got = _fb(eng, eng.device_ptr(pydugks.DG_BUF_FB))
    want = pyoracle.interior(orc.fbar(pyoracle.to_ghosted(f0)))
    # ghosts as the reference fills them: x, then y, then z
    w = np.zeros_like(got)
    w[1:-1, 1:-1, 1:-1] = want
    w[..., 0, :], w[..., -1, :] = ((w[..., -2, :], w[..., 1, :]) if periodic_x else
                                   (2 * w[..., 1, :] - w[..., 2, :], 2 * w[..., -2, :] - w[..., -3, :]))
    w[:, 0], w[:, -1] = w[:, -2], w[:, 1]
    w[0], w[-1] = w[-2], w[1]
    assert rel_err(got, w) <= TOL


def test_query_while_the_stream_is_captured():
    eng, orc, f0 = _pair(*N, periods_x=0, ambient_fz=1e-5)

    def call():
        eng.step(1)
        return eng.device_ptr(pydugks.DG_BUF_FB)
    g, ptr = _capture(eng, call)
    assert ptr
    for _ in range(2):  # the second replay steps in FP64
        f = eng.get_state()
        g.replay()
        got = _fb(eng, ptr)[1:-1, 1:-1, 1:-1]
        assert rel_err(got, pyoracle.interior(orc.fbar(pyoracle.to_ghosted(f)))) <= TOL
    h = pyoracle.to_ghosted(f0)
    orc.run(h, 1, 2)
    assert rel_err(eng.get_state(), pyoracle.interior(h)) <= TOL


def test_steps_captured_before_the_query_keep_fp64_after_it():
    eng, orc, f0 = _pair(*N, periods_x=0, ambient_fz=1e-5)
    g, _ = _capture(eng, lambda: eng.step(1))
    g.replay()
    torch.cuda.synchronize()
    ptr = eng.device_ptr(pydugks.DG_BUF_FB)
    assert rel_err(_fb(eng, ptr)[1:-1, 1:-1, 1:-1], pyoracle.interior(orc.fbar(pyoracle.to_ghosted(f0)))) <= TOL
    f1 = eng.get_state()
    g.replay()
    assert rel_err(_fb(eng, ptr)[1:-1, 1:-1, 1:-1], pyoracle.interior(orc.fbar(pyoracle.to_ghosted(f1)))) <= TOL


def test_query_does_not_wait_for_the_stream():
    eng, _, _ = _pair(128, 128, 64, periods_x=0)
    st = torch.cuda.Stream()
    eng.set_stream(st.cuda_stream)
    eng.run(1, 8)
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    eng.run(9, 400)  # some hundred milliseconds
    done.record(st)
    assert eng.device_ptr(pydugks.DG_BUF_FB)
    assert not done.query()
    torch.cuda.synchronize()


class _PoolProps(ctypes.Structure):  # CUmemPoolProps
    _fields_ = [("allocType", ctypes.c_int), ("handleTypes", ctypes.c_int), ("locType", ctypes.c_int),
                ("locId", ctypes.c_int), ("security", ctypes.c_void_p), ("maxSize", ctypes.c_size_t),
                ("usage", ctypes.c_ushort), ("reserved", ctypes.c_ubyte * 54)]


def _query_with_a_small_pool():
    eng, orc, f0 = _pair(64, 32, 32, periods_x=0)
    eng.step(1)
    eng.sync()
    cu = ctypes.CDLL("libcuda.so.1")
    props, pool = _PoolProps(allocType=1, locType=1, locId=0, maxSize=2 << 20), ctypes.c_void_p()
    assert cu.cuMemPoolCreate(ctypes.byref(pool), ctypes.byref(props)) == 0
    assert cu.cuDeviceSetMemPool(0, pool) == 0
    ptr = eng.device_ptr(pydugks.DG_BUF_FB)
    assert ptr
    want = pyoracle.interior(orc.fbar(pyoracle.to_ghosted(f0)))
    assert rel_err(_fb(eng, ptr)[1:-1, 1:-1, 1:-1], want) <= TOL


def test_query_without_device_memory_for_the_copy():
    """The device's stream-ordered pool limited to less than f-bar-plus (14 MB).  In a process of its
    own, which keeps that pool: once it was destroyed libcuda's cuStreamSynchronize crashed."""
    here = os.path.dirname(os.path.abspath(__file__))
    code = ("import conftest, test_gpu_fb_address as t; t._query_with_a_small_pool()")
    r = subprocess.run([sys.executable, "-c", code], cwd=here, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
