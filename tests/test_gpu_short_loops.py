"""In-place loops that one launch runs: boxes no deeper than the loop has iterations (a deeper
halo is only work), with the bits of one launch per iteration."""
import ctypes

import numpy as np
import pytest

import xgrid
from xgrid_gb300 import runtime
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


def relax(p: xgrid.grid[float, 2], f: xgrid.grid[float, 2], iters: int) -> None:
    for _ in range(0, iters):
        p[0, 0] = 0.25 * (p[1, 0][0] + p[-1, 0][0] + p[0, 1][0] + p[0, -1][0]) - f[0, 0][0]
        with xgrid.boundary(1):
            p[0, 0] = p[0, 1][0]


def _grids(n):
    rng = np.random.default_rng(n)
    p, f = xgrid.Grid((n, n), float), xgrid.Grid((n, n), float)
    p.now[...] = rng.random((n, n))
    f.now[...] = rng.random((n, n)) - 0.5
    p.boundary[:, 0] = 1
    p.boundary[0, :] = p.boundary[-1, :] = p.boundary[:, -1] = 2
    return p, f


def _depths(grid):
    """Depths of the boxes that the grid's mask has tables for."""
    built = runtime.load().xg_internal_boxes_built
    built.argtypes = [ctypes.c_void_p] + [ctypes.POINTER(ctypes.c_int32)] * 2 + [ctypes.c_int,
                                                                               ctypes.POINTER(ctypes.c_int32)]
    i3, value = ctypes.c_int32 * 3, (ctypes.c_int32 * 1)(1)
    return {d for d in range(1, 9) for w in (32, 64, 96, 128) for r in range(4, 65)
            if built(grid._mask, i3(1, r, w - 2 * d), i3(0, d, d), 1, value)}


@pytest.mark.parametrize("precision", ["double", "float"])
@pytest.mark.parametrize("n", [33, 257, 513])
@pytest.mark.parametrize("iters,depths", [(2, {2}), (3, {3}), (4, {4, 5, 6}), (50, {3, 4, 5, 6})])
def test_boxes_are_no_deeper_than_the_loop(cacheroot, precision, n, iters, depths):
    out = []
    for kw in ({}, {"loop_temporal": 0}):
        xgrid.init(precision=precision, cacheroot=cacheroot, opt_level=3, **kw)
        k = Operator(relax, "kernel", "relax")
        p, f = _grids(n)
        for _ in range(4):
            k(p, f, iters)
        if not kw:
            assert len(_depths(p)) == 1 and _depths(p) <= depths
        out.append(p.read(0).tobytes())
    assert out[0] == out[1]


@pytest.mark.parametrize("n,iters,direct", [(33, 1, False), (65, 3, False), (257, 2, False), (257, 3, False),
                                            (1025, 3, True), (1500, 2, True)])
def test_short_launches_replay_their_graph(cacheroot, n, iters, direct):
    """A short launch is cheaper as a graph replay, which issues no launch of its own; a long
    one is launched directly from the third call on."""
    xgrid.init(precision="double", cacheroot=cacheroot, opt_level=3)
    k = Operator(relax, "kernel", "relax")
    p, f = _grids(n)
    for _ in range(8):  # every rotation of the levels eager, then captured
        k(p, f, iters)
    lib = runtime.load()
    before = lib.xg_prof_launches()
    for _ in range(4):
        k(p, f, iters)
    assert lib.xg_prof_launches() - before == (4 if direct else 0)
