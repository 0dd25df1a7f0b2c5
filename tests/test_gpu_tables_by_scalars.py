"""One regular call builds every table that later calls on the same grids need, whatever
their scalars: a no-alloc call and a call captured by the caller give a regular call's bits
with scalars under which the pressure loop's boxes would have another shape (a power of two
costs no FP64 operation in a product, and the shape follows the operation count)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import xgrid
from xgrid_gb300 import device, runtime
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


def relax(p: xgrid.grid[float, 2], f: xgrid.grid[float, 2], iters: int, h2: float) -> None:
    for _ in range(0, iters):
        p[0, 0] = 0.25 * (p[1, 0][0] + p[-1, 0][0] + p[0, 1][0] + p[0, -1][0] - h2 * f[0, 0][0])
        with xgrid.boundary(1):
            p[0, 0] = p[0, 1][0]
        with xgrid.boundary(2):
            p[0, 0] = 0.5


def _grids(n):
    rng = np.random.default_rng(n)
    p, f = xgrid.Grid((n, n), float), xgrid.Grid((n, n), float)
    p.now[...] = rng.random((n, n))
    f.now[...] = rng.random((n, n)) - 0.5
    p.boundary[:, 0] = 1
    p.boundary[0, :] = p.boundary[-1, :] = p.boundary[:, -1] = 2
    return p, f


def _noalloc(k, grids, values):
    nk = k.native
    fn = nk.lib.entry(f"xg_kernel_{nk.module.name}_noalloc")
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.POINTER(runtime.XGGrid), ctypes.c_int, ctypes.c_void_p, ctypes.c_size_t,
                   ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p]
    for g in grids:
        g._op_invoke(nk.depth, True)
        g._sync_device(False)
    device.stream().synchronize()
    arr = (runtime.XGGrid * len(grids))(*[g.serialize() for g in grids])
    packed = nk.pack(values)
    rc = fn(arr, len(grids), ctypes.addressof(packed), ctypes.sizeof(packed), None, 0, device.stream_handle())
    device.stream().synchronize()
    assert rc == 0, runtime.last_error()
    for g, st in zip(grids, arr):
        g._adopt(st)


@pytest.mark.parametrize("first,later", [((7, 0.01), (7, 0.25)), ((7, 0.25), (7, 0.01)), ((1, 0.25), (9, 0.3)),
                                         ((20, 0.01), (2, 0.25))])
@pytest.mark.parametrize("n", [257, 449])
@pytest.mark.parametrize("how", ["noalloc", "captured"])
def test_later_scalars_need_no_new_tables(cacheroot, how, n, first, later):
    xgrid.init(precision="double", cacheroot=cacheroot, opt_level=3)
    k = Operator(relax, "kernel", "relax")
    k.noalloc = True
    (pa, fa), (pb, fb) = _grids(n), _grids(n)
    k(pa, fa, *first)
    k(pa, fa, *later)
    k(pb, fb, *first)
    if how == "noalloc":
        _noalloc(k, (pb, fb), list(later))
    else:
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=device.stream()):
            k(pb, fb, *later)
        graph.replay()
        torch.cuda.synchronize()
    assert pa.read(0).tobytes() == pb.read(0).tobytes()
