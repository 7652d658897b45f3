"""The flux kernels of the float forms at the edges of their tiles (32 columns; 4 to 7 rows),
for both reconstructions (flux_tma_kernel, flux_sh_kernel), against the oracle."""
import numpy as np
import pytest

import pydugks
import pyoracle
from _cases import run_both
from seeded import rel_err, seeded_state

pytestmark = pytest.mark.gpu

# FP32: the bound of tests/test_gpu_parity.py; 16-bit: 3 storage quanta of the largest deviation
# from the rest equilibrium, as tests/test_gpu_mixed.py
QUANT = {"fp16": 2.0 ** -11, "bf16": 2.0 ** -8}


@pytest.mark.parametrize("nx,ny,nz", [(3, 4, 1), (31, 5, 9), (32, 8, 2), (33, 9, 5), (63, 7, 4), (64, 13, 3),
                                      (65, 15, 8), (97, 3, 17)])
@pytest.mark.parametrize("periodic_x", [0, 1])
@pytest.mark.parametrize("prec", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("recon", ["gradient", "trilinear"])
def test_edges_of_tiles(nx, ny, nz, periodic_x, prec, recon):
    cfg = pydugks.make_config(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=1.5 * ny, zwidth=2.0 * nz, periods_x=periodic_x,
                              CFL=0.5, visc=0.02, ambient_fx=1e-5 if periodic_x else 0.0, ambient_fy=2e-5,
                              ambient_fz=1e-5, precision=prec, recon=recon)
    eng = pydugks.Engine(cfg)
    orc = pyoracle.Oracle.from_config(cfg, dtype=np.float32 if prec == "fp32" else np.float64)
    eng.set_state(seeded_state(nx, ny, nz, seed=11))
    f0 = eng.get_state()  # the stored start
    got, want = run_both(eng, orc, f0, 1, 4)
    if prec == "fp32":
        tol = 2e-5
    else:
        w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
        tol = 3.0 * QUANT[prec] * max(1e-3, float(np.max(np.abs(f0 - w) / w)))
    assert rel_err(got, want) <= tol
