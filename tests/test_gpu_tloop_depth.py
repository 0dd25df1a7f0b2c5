"""Depth of the pressure loop's boxes by the grid's size (``loop_temporal`` left at
its default): every level of every grid has the bits of one launch per iteration,
on grids smaller than a box, of ragged sizes and over several waves of boxes, and
for iteration counts below the depth, at it and with remainders."""
import numpy as np
import pytest

import xgrid
import workloads
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision", [(9, "double"), (33, "double"), (65, "double"), (131, "double"), (257, "double"),
                                         (700, "double"), (1203, "double"), (201, "float")])
def test_cavity_bits(cacheroot, n, precision):
    out = []
    for kw in ({}, {"loop_temporal": 0}):
        xgrid.init(precision=precision, cacheroot=cacheroot, opt_level=3, **kw)
        k = Operator(workloads.cavity_kernel.func, "kernel", "cavity_kernel")
        g, cfg = workloads.cavity_setup(n, 5e-6, seed=n)
        for _ in range(3):
            k(g["b"], g["p"], g["u"], g["v"], cfg)
        out.append({c: (g[c].read(0).tobytes(), g[c].read(1).tobytes()) for c in "bpuv"})
    assert out[0] == out[1]


def walled(p: xgrid.grid[float, 2], f: xgrid.grid[float, 2], iters: int) -> None:
    for _ in range(0, iters):
        p[0, 0] = 0.25 * (p[1, 0][0] + p[-1, 0][0] + p[0, 1][0] + p[0, -1][0]) - f[0, 0][0]
        with xgrid.boundary(2):
            p[0, 0] = 0.5 * p[0, 1][0]


@pytest.mark.parametrize("shape,wall", [((150, 211), 0), ((47, 33), 0), ((600, 5), 0), ((5, 900), 0),
                                        ((150, 211), 40), ((64, 96), 17)])
def test_iteration_counts(cacheroot, shape, wall):
    """A wall column that reads its right neighbour: on the grid's left edge, and inside the grid."""
    rng = np.random.default_rng(8)
    p0, f0 = rng.random(shape), rng.random(shape)
    m = np.zeros(shape, np.int32)
    m[0, :] = m[-1, :] = m[:, 0] = m[:, -1] = 1
    m[1:-1, wall] = 2
    out = []
    for kw in ({}, {"loop_temporal": 0}):
        xgrid.init(precision="double", cacheroot=cacheroot, opt_level=3, **kw)
        k = Operator(walled, "kernel", "walled")
        p, f = xgrid.Grid(shape, float), xgrid.Grid(shape, float)
        p._extend_time(2)
        for lv in p._data:
            lv[...] = p0
        f.now[...] = f0
        p.boundary[...] = m
        for iters in (7, 2, 1, 3, 4, 5, 6, 13):
            k(p, f, iters)
        out.append(p.read(0).tobytes())
    assert out[0] == out[1]
