"""Training runs that follow one another on one trainer: parameters set by the caller
start a run with cleared Adam moments, whatever ran before, and each run returns its
own losses."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import glisser_gb300 as G  # noqa: E402
from glisser_gb300 import learned as L  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def native():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    G.build()
    G.lib()


def trainer():
    rng = np.random.default_rng(2)
    n = 4096
    tr = L.Trainer(n, seed=9)
    feat = np.stack([rng.uniform(-10, 0, n), rng.uniform(-1, 1, n), rng.uniform(0, 2, n)], 1).astype(np.float32)
    tr.add_samples(feat, rng.normal(0.0, 0.03, n).astype(np.float32))
    tr.fit_norm()
    return tr


def test_set_parameters_start_a_fresh_run():
    a = trainer()
    p = a.params.copy()
    want_losses = a.train(20, batch=256, lr=1e-2, seed=5)
    want = a.params.copy()
    for _ in range(10):
        a.params = p
        losses = a.train(20, batch=256, lr=1e-2, seed=5)
        assert np.array_equal(losses, want_losses) and np.array_equal(a.params, want)


def test_losses_of_runs_of_different_lengths():
    # the trainer's loss buffer grows with the longest run and is used again
    a = trainer()
    p = a.params.copy()
    for steps in (1, 50, 3, 50, 49):
        a.params = p
        got = a.train(steps, batch=256, lr=1e-2, seed=steps)
        b = trainer()
        b.params = p
        assert np.array_equal(got, b.train(steps, batch=256, lr=1e-2, seed=steps))
