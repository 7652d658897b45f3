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


@pytest.mark.parametrize("prec,periodic_x,n", [("fp64", 0, 3), ("fp64", 1, 3), ("fp32", 0, 2), ("fp32", 1, 2),
                                               ("fp16", 0, 2), ("bf16", 1, 2)])
def test_launches_that_the_benchmark_reports(prec, periodic_x, n):
    """bench.py counts them; stage (a) of the 16-bit forms writes their ghosts with periodic x too."""
    import os
    import sys
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    import bench
    cfg = pydugks.make_config(nx=40, ny=9, nz=7, xwidth=40, ywidth=9, zwidth=7, CFL=0.5, visc=0.02, precision=prec,
                              periods_x=periodic_x)
    eng = pydugks.Engine(cfg)
    assert bench.count_launches(eng, 0) == n
    eng.step(1)
    eng.sync()
