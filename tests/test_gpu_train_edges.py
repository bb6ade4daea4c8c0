"""The training kernels at the edges of their tiles (128 samples a CTA) and of the
update kernel's groups of partials (64 CTAs), against the float64 oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import glisser_gb300 as G  # noqa: E402
from glisser_gb300 import learned as L  # noqa: E402
from oracle import mlp_oracle as M  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def native():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    G.build()
    G.lib()


def trainer():
    rng = np.random.default_rng(4)
    tr = L.Trainer(1024, seed=9)
    tr.norm = dict(in_mean=[-6.5, 0.0, 1.1], in_scale=[0.45, 2.2, 1.7], x_lo=[-30, -5, -1], x_hi=[5, 5, 5],
                   out_mean=0.002, out_scale=0.015)
    p = M.init_params(9)
    p[M.OFF_B1:M.OFF_W2] = rng.normal(0, 0.2, 32)
    p[M.OFF_B2:M.OFF_W3] = rng.normal(0, 0.2, 32)
    tr.params = p
    return tr, p


@pytest.mark.parametrize("n", [1, 127, 128, 129, 63 * 128, 64 * 128, 65 * 128 + 1, 130 * 128])
def test_gradients_at_tile_edges(n):
    tr, p = trainer()
    rng = np.random.default_rng(n)
    feat = np.stack([rng.uniform(-10, 0, n), rng.uniform(-1, 1, n), rng.uniform(0, 2, n)], 1).astype(np.float32)
    target = rng.normal(0.0, 0.03, n).astype(np.float32)
    got, loss = tr.gradients(feat, target)
    want_loss, want = M.loss_and_grad(p, tr.norm, feat.astype(np.float64), target.astype(np.float64))
    # the bounds of the 1,000-sample comparison: FP32 sums and the fast exponential
    assert abs(loss - want_loss) <= 1e-5 * want_loss
    for a, b in ((M.OFF_W1, M.OFF_B1), (M.OFF_B1, M.OFF_W2), (M.OFF_W2, M.OFF_B2), (M.OFF_B2, M.OFF_W3),
                 (M.OFF_W3, M.OFF_B3), (M.OFF_B3, M.NPARAM)):
        assert np.linalg.norm(got[a:b] - want[a:b]) / np.linalg.norm(want[a:b]) < 1e-4, (a, b)


def test_every_steps_loss_is_returned():
    tr, _ = trainer()
    rng = np.random.default_rng(2)
    n = 1000
    feat = np.stack([rng.uniform(-10, 0, n), rng.uniform(-1, 1, n), rng.uniform(0, 2, n)], 1).astype(np.float32)
    tr.add_samples(feat, rng.normal(0.0, 0.03, n).astype(np.float32))
    tr.fit_norm()
    before = tr.params
    losses = tr.train(37, batch=256, lr=1e-3, seed=5)
    assert losses.shape == (37,) and np.all(np.isfinite(losses)) and np.all(losses > 0)
    assert len(np.unique(losses)) == 37 and not np.array_equal(before, tr.params)
    assert tr.train(0, batch=256).size == 0
