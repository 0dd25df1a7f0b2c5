"""Batched FP32 problems whose sweep computes in FP64 (a Python literal is a double): they keep
the shared-memory kernel and its low tiles, with the bits of one call per problem per step."""
import numpy as np
import pytest

import xgrid
import workloads
from xgrid_gb300.codegen import CudaGenerator
from xgrid_gb300.config import get_config
from xgrid_gb300.operator import Operator


def damped(u: xgrid.grid[float, 2], a: float) -> None:
    u[0, 0] = 0.99 * (u[0, 0] + a * (u[0, 1] + u[0, -1] + u[1, 0] + u[-1, 0] - u[0, 0]))


def nine(u: xgrid.grid[float, 2], a: float) -> None:
    u[0, 0] = a * u[0, 0] + 0.07 * (u[0, 1] + u[-1, 0]) + 0.03 * (u[1, 1] + u[-1, -1])


@pytest.mark.parametrize("body,registers", [(damped, False), (nine, False), (workloads.convdiff2d.func, True)])
def test_kernel_by_arithmetic(body, registers):
    xgrid.init(precision="float", overstep="wrap")
    m = CudaGenerator(Operator(body, "kernel", body.__name__), get_config()).generate()
    assert m.batch and m.batch_registers == registers


@pytest.mark.gpu
@pytest.mark.parametrize("body", [damped, nine])
@pytest.mark.parametrize("temporal,steps", [((2, 16, 60), 7), ((4, 32, 56), 9), ((3, 58, 58), 4), (None, 6)])
def test_literals_equal_sequential_calls(cacheroot, body, temporal, steps):
    xgrid.init(precision="float", cacheroot=cacheroot, opt_level=3, overstep="wrap")
    kb, ks = (Operator(body, "kernel", body.__name__) for _ in range(2))

    def problems():
        rng = np.random.default_rng(4)
        out = []
        for shape in [(14, 131), (105, 58), (70, 64), (12, 12)]:
            g = xgrid.Grid(shape, float)
            g.now[...] = rng.random(shape).astype(np.float32)
            out.append((g, float(rng.uniform(0.01, 0.2))))
        return out
    a, b = problems(), problems()
    for _ in range(2):  # eager, then captured
        kb.batch(a, steps, temporal=temporal)
        for _ in range(steps):
            for args in b:
                ks(*args)
    for pa, pb in zip(a, b):
        for lvl in (0, 1):
            assert pa[0].read(lvl).tobytes() == pb[0].read(lvl).tobytes()
