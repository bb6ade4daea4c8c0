"""The time-block kernel's choice between the small-step and the general drift
(tau^2 = dt^2 mu / r^3 around 1e-3): blocks without planets, so that a step is
one drift, against the long-double drift; and each particle's result
independent of the particles that share its warp."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import glisser_gb300 as G  # noqa: E402
from test_smallstep_host import DT, MU, drift_long_double, states  # noqa: E402

N = 1000        # fifteen full CTAs of the single-system kernel and a part of one


@pytest.fixture(scope="module", autouse=True)
def native():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    G.build()
    G.lib()


def block(rv, steps, kick):
    from gpu_util import DevHandoff, DevParticles, DevPlanetBlock, timeblock
    n = len(rv)
    p = DevParticles(rv[:, :3], rv[:, 3:], np.zeros((n, 3)), np.zeros(n), np.arange(n))
    b = DevPlanetBlock(np.zeros((steps, 3)), np.zeros((steps, 0, 3)), [MU], [0], [0.1])
    ho = timeblock(p, b, DT, 1e6, handoff=DevHandoff(n), kick=kick)
    h = p.host()
    assert not h["flags"].any() and ho["evals"] >= n * steps
    return np.concatenate([h["r"], h["v"]], 1), ho


@pytest.mark.parametrize("kick", [G.KICK_FLOAT_FLOAT, G.KICK_FP64])
@pytest.mark.parametrize("steps", [1, 2, 33])
@pytest.mark.parametrize("lo,hi", [(1e-6, 0.9e-3), (0.9e-3, 1.1e-3), (1e-5, 8e-3)])
def test_block_of_drifts(lo, hi, steps, kick):
    rng = np.random.default_rng(11)
    rv = states(np.exp(rng.uniform(np.log(lo), np.log(hi), N)), rng.uniform(0, 0.6, N), 12)
    got, ho = block(rv, steps, kick)
    assert steps > 2 or ho["wide"] == 0      # later some reach a pericentre beyond the series domain
    want = rv.astype(np.longdouble)
    for _ in range(steps):
        want = np.concatenate(drift_long_double(want, DT, MU), 1)
    # a few 2^-53 a step in position and velocity, carried along: an error in the
    # velocity moves the position by tau a step, one in the energy shears it
    tau = np.sqrt(hi) * 4           # the pericentre of the same orbit is nearer
    tol = 1.2e-15 * steps * (1 + tau * steps)
    for s in (slice(0, 3), slice(3, 6)):
        d = (got[:, s] - want[:, s]).astype(np.float64)
        err = np.linalg.norm(d, axis=1) / np.linalg.norm(want[:, s].astype(np.float64), axis=1)
        assert err.max() < tol, (err.max(), tol)


@pytest.mark.parametrize("steps", [1, 2])
def test_block_of_drifts_at_the_medium_bound(steps):
    # tau^2 around 1e-2, where the float-float solution gives way to the general one
    rng = np.random.default_rng(15)
    rv = states(np.exp(rng.uniform(np.log(0.8e-2), np.log(1.2e-2), N)), rng.uniform(0, 0.6, N), 16)
    got, _ = block(rv, steps, G.KICK_FLOAT_FLOAT)
    want = rv.astype(np.longdouble)
    for _ in range(steps):
        want = np.concatenate(drift_long_double(want, DT, MU), 1)
    tol = 1.2e-15 * steps * (1 + 4 * np.sqrt(1.2e-2) * steps)      # as above
    for s in (slice(0, 3), slice(3, 6)):
        d = (got[:, s] - want[:, s]).astype(np.float64)
        err = np.linalg.norm(d, axis=1) / np.linalg.norm(want[:, s].astype(np.float64), axis=1)
        assert err.max() < tol, (err.max(), tol)


def test_a_particles_path_is_its_own():
    rng = np.random.default_rng(13)
    rv = states(np.exp(rng.uniform(np.log(1e-4), np.log(5e-3), N)), np.full(N, 0.05), 14)
    order = rng.permutation(N)
    a, _ = block(rv, 8, G.KICK_FLOAT_FLOAT)
    b, _ = block(rv[order], 8, G.KICK_FLOAT_FLOAT)
    # nearly circular: tau^2 stays on its side of the bound (e 0.05: within 18 %)
    small = DT * DT * MU / np.linalg.norm(rv[:, :3], axis=1) ** 3 < 0.8e-3
    assert small.sum() > 300 and np.array_equal(a[order][small[order]], b[small[order]])
