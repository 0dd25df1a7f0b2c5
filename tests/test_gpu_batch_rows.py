"""Register-block kernel with 16 rows a warp (boxes of 65 to 128 rows) and 2 or 4 columns a
lane: the call runs on that kernel, and has the bits of one call per problem per step."""
import numpy as np
import pytest

import xgrid
import workloads
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu

SHAPES = [(14, 131), (105, 58), (200, 210), (116, 52), (57, 241), (12, 12)]  # every extent holds a halo of 12


def rows2d(u: xgrid.grid[float, 2], a: float) -> None:
    u[0, 0] = u[0, 0] + a * (u[-1, 0] - u[0, 0]) + a * (u[1, 0] - u[0, 0])


@pytest.mark.parametrize("program,nval,rx", [("convdiff2d", 5, 1), ("rows2d", 1, 0)])
@pytest.mark.parametrize("temporal,steps", [((12, 104, 104), 25), ((6, 116, 52), 13), ((4, 57, 120), 9), ((2, 61, 60), 5),
                                            ((8, 112, 40), 31), ((1 + 4, 118, 118), 11)])
def test_sixteen_rows_equal_sequential_calls(cacheroot, program, nval, rx, temporal, steps):
    xgrid.init(precision="float", cacheroot=cacheroot, opt_level=3, overstep="wrap")
    body = workloads.convdiff2d.func if program == "convdiff2d" else rows2d
    kb, ks = (Operator(body, "kernel", program) for _ in range(2))

    def problems():
        rng = np.random.default_rng(21)
        out = []
        for shape in SHAPES:
            g = xgrid.Grid(shape, float)
            g.now[...] = rng.random(shape).astype(np.float32)
            out.append((g, *(float(v) for v in rng.uniform(0.01, 0.2, nval))))
        return out
    a, b = problems(), problems()
    for _ in range(2):  # eager, then captured
        kb.batch(a, steps, temporal=temporal)
        for _ in range(steps):
            for args in b:
                ks(*args)
    T, ty, tx = temporal
    state = kb.native._batch
    assert all(entry[3] >= 0 for entry in state["desc"].values())  # work items of the temporal kernel
    assert 64 < ty + 2 * T <= 128 and tx + 2 * T * rx <= 128
    columns = 2 if tx + 2 * T * rx <= 64 else 4
    assert state["nblocks"][(256, T, ty, tx)][0] == 8 * 16 * 32 * columns * 4  # its staging buffer
    for pa, pb in zip(a, b):
        for lvl in (0, 1):
            assert pa[0].read(lvl).tobytes() == pb[0].read(lvl).tobytes()
