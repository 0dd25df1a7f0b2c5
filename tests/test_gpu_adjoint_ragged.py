"""Adjoint step on the staged z-walk at the edges of its block: rows that are not
16-byte aligned, aligned rows with a narrow last block, single columns and rows
beyond a block, fewer planes than a chunk.  Gradients against the register
z-walk, to the rounding of the two kernels' contractions over the steps."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import xgrid
import workloads
from xgrid_gb300 import adjoint
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,dtype,tol", [("float", np.float32, 1e-5), ("double", np.float64, 1e-13)])
@pytest.mark.parametrize("shape", [(3, 9, 33), (9, 8, 129), (17, 7, 128), (40, 33, 127), (16, 9, 132), (70, 3, 5),
                                   (24, 65, 260)])
def test_edges_of_the_staged_block(cacheroot, precision, dtype, tol, shape):
    xgrid.init(precision=precision, cacheroot=cacheroot, opt_level=3, overstep="wrap")
    rng = np.random.default_rng(sum(shape))
    u0 = torch.tensor(rng.random(shape).astype(dtype), device="cuda")
    kap = torch.tensor(rng.uniform(0.01, 0.1, shape).astype(dtype), device="cuda")
    grads = []
    for staged in (True, False):
        ro = adjoint.Rollout(Operator(workloads.diffuse3d.func, "kernel", "diffuse3d"), 5)
        ro.set_zstage(staged)
        a = u0.clone().requires_grad_(True)
        b = kap.clone().requires_grad_(True)
        ((ro(a, {"k": b}, (0.5,))) ** 2).mean().backward()
        grads.append((a.grad.clone(), b.grad.clone()))
    for g, r in zip(*grads):
        assert float((g - r).abs().max() / r.abs().max()) < tol
