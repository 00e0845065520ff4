"""Grids of the four-launch stage (N <= 128) have one launch shape: sns_autotune keeps it, writes
it to the cache and reads it back, and a batch that asks for tuning steps as one that does not."""
import numpy as np
import pytest

from spectral_solver_b200 import Batch, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 64, 128])
@pytest.mark.parametrize("precision", [0, 1])
def test_the_shape_stays(n, precision, tmp_path):
    cache = str(tmp_path / "shapes.txt")
    with Solver(n, precision=precision) as s:
        before = s.launch_config()
        for _ in range(2):
            cfg = s.autotune(1, cache)
            assert s.launch_config() == before
            assert cfg == dict(tma_grid=before["tma_grid"], xpass_grid=before["xpass_grid"], p5_grid=before["p5_grid"])
    assert len(open(cache).read().splitlines()) == 1


def test_batch_with_tuning(tmp_path):
    specs = [dict(n=n, nu=1e-2, seed=n, pert_amp=0.01, pert_kmax=2, precision=1, dt=1e-3) for n in (16, 32, 128)]
    states = []
    for trials in (0, 1):
        with Batch(specs, autotune_trials=trials, autotune_cache=str(tmp_path / "b.txt")) as b:
            b.step(3)
            states.append([b.solver(i).get_state() for i in range(len(specs))])
    for one, two in zip(*states):
        assert all(np.array_equal(a, c) for a, c in zip(one, two))
