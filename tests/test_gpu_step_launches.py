"""What a step launches: no kernel that needs the whole GPU at once (a step runs on whatever
part of it is free)."""
import pytest

import pydugks
from graph_nodes import captured_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp16"])
def test_no_launch_is_cooperative(prec):
    cfg = pydugks.make_config(nx=40, ny=9, nz=7, xwidth=40, ywidth=9, zwidth=7, CFL=0.5, visc=0.02, precision=prec)
    eng = pydugks.Engine(cfg)
    kernels = captured_kernels(eng, lambda: eng.step(1))
    assert kernels and not any(coop for _, _, coop in kernels), kernels
