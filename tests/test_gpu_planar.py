"""Swarms in a plane: the third component is zero at every step, a value that the
float-float conversions treat apart.  Against long double, with both kicks, and
with a third component so small that it takes the conversions' rare branch."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import glisser_gb300 as G  # noqa: E402
from test_gpu_smallstep import N, block  # noqa: E402
from test_smallstep_host import DT, MU, drift_long_double, states  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def native():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    G.build()
    G.lib()


@pytest.mark.parametrize("kick", [G.KICK_FLOAT_FLOAT, G.KICK_FP64])
@pytest.mark.parametrize("z", [0.0, 1e-25])
@pytest.mark.parametrize("hi", [0.9e-3, 8e-3])
def test_planar_block(hi, z, kick):
    rng = np.random.default_rng(41)
    rv = states(np.exp(rng.uniform(np.log(1e-6), np.log(hi), N)), np.full(N, 0.2), 42)
    # turned into the plane: the same distances, speeds and angles between r and v
    r, v = rv[:, :3], rv[:, 3:]
    r0, v0 = np.linalg.norm(r, axis=1), np.linalg.norm(v, axis=1)
    c = (r * v).sum(1) / (r0 * v0)
    th, s = rng.uniform(0, 2 * np.pi, N), np.sqrt(1 - c * c)
    flat = np.zeros((N, 6))
    flat[:, 0], flat[:, 1] = r0 * np.cos(th), r0 * np.sin(th)
    flat[:, 3] = v0 * (c * np.cos(th) - s * np.sin(th))
    flat[:, 4] = v0 * (c * np.sin(th) + s * np.cos(th))
    flat[:, 2], flat[:, 5] = z, -z
    steps = 8
    got, _ = block(flat, steps, kick)
    want = flat.astype(np.longdouble)
    for _ in range(steps):
        want = np.concatenate(drift_long_double(want, DT, MU), 1)
    # as in the block test of the tiers: a few 2^-53 a step, carried along
    tol = 1.2e-15 * steps * (1 + 4 * np.sqrt(hi) * steps)
    for k in (slice(0, 3), slice(3, 6)):
        err = np.linalg.norm((got[:, k] - want[:, k]).astype(np.float64), axis=1)
        err /= np.linalg.norm(want[:, k].astype(np.float64), axis=1)
        assert err.max() < tol, (err.max(), tol)
    if z == 0.0:
        assert not got[:, 2].any() and not got[:, 5].any()
