"""Register-block kernel of the batched path: tiles whose box (tile and halo) just fits
its 64 or 128 rows and columns, smaller and remainder tiles, one field and two with
diagonal loads, every depth's ring of levels -- the bits of one call per problem per step."""
import numpy as np
import pytest

import xgrid
import workloads
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


def coupled2d(u: xgrid.grid[float, 2], v: xgrid.grid[float, 2], a: float, b: float) -> None:
    u[0, 0] = u[0, 0] + a * (v[0, 1] - v[0, -1]) + b * (v[1, 1] - u[0, 0])
    v[0, 0] = v[0, 0] + b * (u[1, 0] - u[-1, 0]) + a * (u[-1, -1] - v[0, 0])


def rows2d(u: xgrid.grid[float, 2], a: float) -> None:
    u[0, 0] = u[0, 0] + a * (u[-1, 0] - u[0, 0]) + a * (u[1, 0] - u[0, 0])


@pytest.mark.parametrize("temporal,steps", [((6, 52, 116), 12), ((6, 52, 52), 13), ((2, 60, 124), 5), ((1, 30, 30), 3),
                                             ((8, 48, 112), 31), ((12, 104, 104), 25), ((3, 7, 59), 6), ((4, 56, 57), 9), ((5, 54, 1), 10)])
@pytest.mark.parametrize("program", ["convdiff2d", "coupled2d", "rows2d"])
def test_register_blocks_equal_sequential_calls(cacheroot, program, temporal, steps):
    xgrid.init(precision="float", cacheroot=cacheroot, opt_level=3, overstep="wrap")
    body, ngrid, nval = {"convdiff2d": (workloads.convdiff2d.func, 1, 5), "coupled2d": (coupled2d, 2, 2),
                         "rows2d": (rows2d, 1, 1)}[program]
    kb, ks = (Operator(body, "kernel", program) for _ in range(2))

    def problems():
        rng = np.random.default_rng(21)
        out = []
        for shape in [(8, 8), (9, 131), (64, 128), (52, 116), (105, 58), (53, 233)]:
            grids = [xgrid.Grid(shape, float) for _ in range(ngrid)]
            for g in grids:
                g.now[...] = rng.random(shape).astype(np.float32)
            out.append((*grids, *(float(v) for v in rng.uniform(0.01, 0.2, nval))))
        return out
    a, b = problems(), problems()
    for _ in range(2):  # eager, then captured
        kb.batch(a, steps, temporal=temporal)
        for _ in range(steps):
            for args in b:
                ks(*args)
    for pa, pb in zip(a, b):
        for i in range(ngrid):
            for lvl in (0, 1):
                assert pa[i].read(lvl).tobytes() == pb[i].read(lvl).tobytes()
