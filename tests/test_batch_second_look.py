"""The batched tuner times its nearest candidates again over more steps: a short call is bound
by the host, and its noise must not pick the candidate.  Timer and kernel replaced, on the CPU."""
import types

import pytest

import xgrid
from xgrid_gb300 import autotune


class Kernel:
    module = types.SimpleNamespace(name="k", batch_registers=True)

    def split(self, args):
        return [types.SimpleNamespace(shape=(64, 64))], []

    def batch(self, problems, steps, temporal=None):
        self.ran = steps, temporal


@pytest.mark.parametrize("best", [(8, 48, 48), (12, 40, 40), (2, 60, 60)])
@pytest.mark.parametrize("lucky", [(6, 52, 52), (12, 104, 40)])
def test_noise_of_short_calls_does_not_pick(monkeypatch, tmp_path, best, lucky):
    xgrid.init(precision="float", cacheroot=str(tmp_path), overstep="wrap")
    k = Kernel()

    def timed(fn):  # us a step: 1.5 the best, 1.8 the others; a call of n steps takes 80 us of the host
        fn()
        steps, c = k.ran
        ms = max(steps * (1.5 if c[:3] == best else 1.8), 80) * 1e-3
        return ms * (0.97 if c[:3] == lucky and steps == autotune.TUNE_STEPS else 1.0)
    stored = {}
    monkeypatch.setattr(autotune, "_time", timed)
    monkeypatch.setattr(autotune, "_key", lambda *a: "key")
    monkeypatch.setattr(autotune, "_load", lambda root: {})
    monkeypatch.setattr(autotune, "_store", lambda root, key, value: stored.update({key: value}))
    monkeypatch.setattr(autotune, "Snapshot", lambda grids: types.SimpleNamespace(restore=lambda: None))
    assert autotune.tune_batch(k, [()])[:3] == best
    assert tuple(stored["key"][:3]) == best
