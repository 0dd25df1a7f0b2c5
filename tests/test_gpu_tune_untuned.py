"""Tuning against the launch rules: the untuned dispatch (strips here) is one of the tuner's
candidates, a tuning that it wins leaves the group untuned, in this process and from the
cache, and a set tiling can be taken back.  Same bits either way."""
import os

import numpy as np
import pytest

import xgrid
from xgrid_gb300 import autotune
from xgrid_gb300.codegen import DEFAULT_TILING
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


def transport(u: xgrid.grid[float, 2], a: float, b: float) -> None:
    u[0, 0] = a * u[0, 0] + b * (u[0, -1] + u[-1, 0])


@pytest.mark.parametrize("strips_win", [True, False])
def test_untuned_dispatch_is_a_candidate(cacheroot, monkeypatch, strips_win):
    shape = (1500, 1501)
    xgrid.init(precision="float", cacheroot=cacheroot, opt_level=3, overstep="wrap")
    monkeypatch.setattr(autotune, "CACHE_FILE", "autotune_untuned.json")
    path = os.path.join(cacheroot, "autotune_untuned.json")
    if os.path.exists(path):
        os.remove(path)
    k = Operator(transport, "kernel", "transport")
    u = xgrid.Grid(shape, float)
    u.now[...] = np.random.default_rng(4).random(shape)
    k(u, 0.5, 0.25)
    nk = k.native

    def on_strips():
        before = nk.zstage_launches()
        k(u, 0.5, 0.25)
        return nk.zstage_launches() > before

    def timed(fn):  # a clock under which strips win, or lose
        before = nk.zstage_launches()
        fn()
        return 1.0 if (nk.zstage_launches() > before) == strips_win else 2.0
    monkeypatch.setattr(autotune, "_time", timed)
    try:
        assert on_strips()
        chosen = autotune.tune(k, u, 0.5, 0.25)
        assert on_strips() == strips_win
        if strips_win:
            assert chosen == {0: DEFAULT_TILING[2]}
        nk.set_tiling(0, (1, 16, 64, 32, 8, 1))
        assert not on_strips()
        assert autotune.tune(k, u, 0.5, 0.25) == chosen  # from the cache
        assert on_strips() == strips_win
        tuned = u.read(0)
    finally:
        nk.set_tiling(0, None)
    assert on_strips()
    v = xgrid.Grid(shape, float)
    v.now[...] = np.random.default_rng(4).random(shape)
    for _ in range(5):  # the calls above that were not the tuner's own
        k(v, 0.5, 0.25)
    assert v.read(0).tobytes() == tuned.tobytes()
