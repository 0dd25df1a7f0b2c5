"""One regular call is enough for later calls that may not build tables, whatever their
iteration counts: also where the mask allows the boxes of one count and not of the other
(a wall column inside the grid that reads its right neighbour, on an inner edge of either)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import xgrid
from xgrid_gb300 import device
from xgrid_gb300.operator import Operator
from test_gpu_tables_by_scalars import _noalloc

pytestmark = pytest.mark.gpu


def walled(p: xgrid.grid[float, 2], f: xgrid.grid[float, 2], iters: int) -> None:
    for _ in range(0, iters):
        p[0, 0] = 0.25 * (p[1, 0][0] + p[-1, 0][0] + p[0, 1][0] + p[0, -1][0]) - f[0, 0][0]
        with xgrid.boundary(2):
            p[0, 0] = 0.5 * p[0, 1][0]


def _grids(n, wall):
    rng = np.random.default_rng(n)
    p, f = xgrid.Grid((n, n), float), xgrid.Grid((n, n), float)
    p.now[...] = rng.random((n, n))
    f.now[...] = rng.random((n, n)) - 0.5
    p.boundary[0, :] = p.boundary[-1, :] = p.boundary[:, 0] = p.boundary[:, -1] = 1
    p.boundary[1:-1, wall] = 2
    return p, f


@pytest.mark.parametrize("first,later", [(1, 20), (2, 20), (20, 3), (20, 2)])
@pytest.mark.parametrize("wall", [22, 27, 31, 40])  # on an edge of depth 6, of depth 3, of neither, of depth 6
@pytest.mark.parametrize("how", ["noalloc", "captured"])
def test_later_iterations_need_no_new_tables(cacheroot, how, wall, first, later):
    n = 150
    xgrid.init(precision="double", cacheroot=cacheroot, opt_level=3)
    k = Operator(walled, "kernel", "walled")
    k.noalloc = True
    (pa, fa), (pb, fb) = _grids(n, wall), _grids(n, wall)
    k(pa, fa, first)
    k(pa, fa, later)
    k(pb, fb, first)
    if how == "noalloc":
        _noalloc(k, (pb, fb), [later])
    else:
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=device.stream()):
            k(pb, fb, later)
        graph.replay()
        torch.cuda.synchronize()
    assert pa.read(0).tobytes() == pb.read(0).tobytes()
