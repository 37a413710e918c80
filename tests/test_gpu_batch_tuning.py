"""autotune_threads times what Batch.solve runs, the batched PCG, and no other
plan of the factor."""

import numpy as np
import pytest

from rchol_gb300 import _lib, batch, generators

pytestmark = pytest.mark.gpu


class Spy:
    def __init__(self, lib):
        self._lib, self.calls = lib, []

    def __getattr__(self, name):
        self.calls.append(name)
        return getattr(self._lib, name)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_tuning_times_the_solve(cuda, R, monkeypatch, precision):
    spy = Spy(_lib.lib())
    monkeypatch.setattr(_lib, "lib", lambda: spy)
    rng = np.random.default_rng(1)
    mats = [generators.grid_2d_weighted(int(a), int(b), "lognormal", sigma=0.5, rng=rng)
            for a, b in rng.integers(20, 60, size=(4, 2))]
    best, timings = batch.autotune_threads(mats, candidates=(1, 2), sample=3, reps=2, precision=precision)
    assert set(timings) == {1, 2} and best in timings
    assert spy.calls.count("rchol_gpu_pcg_batch_d") == 2 * 3  # a warm-up and two timed ones each
    assert not {"rchol_gpu_precond_d", "rchol_gpu_trsv_d"} & set(spy.calls)
