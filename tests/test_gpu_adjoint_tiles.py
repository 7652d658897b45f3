"""The adjoint step at the edges of its kernels' tiles (no counterpart in the reference).

The cell kernel runs the rows of a plane on into one another, 29 (walls) or 30 (periodic)
cells per warp, four adjacent rows per CTA; the FP32 face kernel takes 32 columns and 8
rows.  FP64: <J d, lam> against <d, J^T lam> as in test_gpu_adjoint.py, with J d from a
Richardson-extrapolated difference (rounding 1e-16/1e-4 per value, so 1e-9 of the sum at
random signs; bound 1e-7).  FP32: every value against the FP64 adjoint, some 100 operations
of 6e-8 each, so 1e-5 of the largest.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import pydugks  # noqa: E402
import dugks_autograd as da  # noqa: E402
from seeded import seeded_state, uniform_sym  # noqa: E402


def _adjoint(precision, shape, periodic, f, lam):
    nx, ny, nz = shape
    eng = pydugks.Engine(pydugks.make_config(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=1.5 * ny, zwidth=nz,
                                             periods_x=periodic, CFL=0.7, visc=0.02, ambient_fz=1e-5,
                                             precision=precision))
    dt = torch.float64 if precision == "fp64" else torch.float32
    ft = da.from_dump_order(eng, torch.from_numpy(f).cuda().to(dt))
    lt = da.from_dump_order(eng, torch.from_numpy(lam).cuda().to(dt))
    out = torch.zeros_like(lt)
    eng.set_stream(torch.cuda.current_stream().cuda_stream)
    eng.adjoint_step(1, ft.data_ptr(), lt.data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    return eng, da.to_dump_order(eng, out).double().cpu().numpy()


@pytest.mark.parametrize("periodic", (0, 1))
@pytest.mark.parametrize("shape", [(3, 1, 1), (27, 4, 2), (28, 5, 3), (29, 9, 2), (30, 8, 3), (31, 7, 2), (33, 16, 1),
                                   (57, 6, 2), (61, 3, 5), (96, 2, 3)])
def test_adjoint_at_tile_edges(shape, periodic):
    nx, ny, nz = shape
    f = seeded_state(nx, ny, nz, seed=4)
    d = uniform_sym(5, f.size, 7).reshape(f.shape) * 1e-2 * f
    lam = uniform_sym(6, f.size, 9).reshape(f.shape)
    eng, vjp = _adjoint("fp64", shape, periodic, f, lam)

    def cdiff(eps):
        s = []
        for g in (f + eps * d, f - eps * d):
            eng.set_state(g)
            eng.run(1, 1)
            s.append(eng.get_state())
        return (s[0] - s[1]) / (2 * eps)

    jvp = (4 * cdiff(5e-5) - cdiff(1e-4)) / 3
    lhs, rhs = float(np.sum(jvp * lam)), float(np.sum(d * vjp))
    scale = float(np.sqrt(np.sum((d * vjp) ** 2)))
    assert abs(lhs - rhs) <= 1e-7 * scale, (lhs, rhs, scale)
    _, v32 = _adjoint("fp32", shape, periodic, f, lam)
    assert np.max(np.abs(v32 - vjp)) <= 1e-5 * np.max(np.abs(vjp))
