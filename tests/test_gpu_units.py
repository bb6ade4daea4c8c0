"""Blocks in other units of length and time, where the float-float drift's ranges
do not hold and the general drift runs at every step: the same swarm with giant
planets in au and days, kilometres and seconds, metres and years, centimetres and
seconds.  States agree to the rounding each carries, flags are the same, with both
kicks and with the classic starter (whose steps are all general in any units)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import glisser_gb300 as G  # noqa: E402

GM, DT, STEPS, N = 2.959122e-4, 100.0, 33, 500
AU_KM, DAY_S, YEAR_D = 1.495978707e8, 86400.0, 365.25
UNITS = {"km,s": (AU_KM, DAY_S), "m,yr": (1e3 * AU_KM, 1 / YEAR_D), "cm,s": (1e5 * AU_KM, DAY_S)}


@pytest.fixture(scope="module", autouse=True)
def native():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    G.build()
    G.lib()


def run(length, time, kick, starter):
    from gpu_util import DevHandoff, DevParticles, DevPlanetBlock, timeblock
    rng = np.random.default_rng(6)
    el = np.stack([rng.uniform(8, 60, N), rng.uniform(0, 0.3, N), rng.uniform(0, 0.3, N),
                   *rng.uniform(0, 2 * np.pi, (3, N))], 1)
    r, v = G.elements_to_cartesian(GM, el)
    m = np.array([GM, 9.55e-4 * GM, 2.86e-4 * GM])
    pos = np.array([[5.2, 0.3, 0.1], [-7.0, 6.0, -0.2]])
    # a few particles inside an encounter radius, beyond the limit, inside the Sun's
    r[0], r[1], r[2] = pos[0] + 0.05, (90.0, 0, 0), (0.2, 0.1, 0.0)
    v[0] = v[2] = 0.0
    h0 = -(m[1:, None] * pos / np.linalg.norm(pos, axis=1)[:, None] ** 3).sum(0)
    vel, acc = length / time, length / time ** 2
    p = DevParticles(r * length, v * vel, np.zeros((N, 3)), np.zeros(N), np.arange(N))
    b = DevPlanetBlock(np.tile(h0 * acc, (STEPS, 1)), np.tile(pos * length, (STEPS, 1, 1)),
                       m * length ** 3 / time ** 2, [0, 5, 6], np.array([0.5, 1.0, 0.8]) * length)
    timeblock(p, b, DT * time, 80.0 * length, handoff=DevHandoff(N), kick=kick, starter=starter,
              encounters=G.ENCOUNTERS_KILL)
    h = p.host()
    return h["r"] / length, h["v"] / vel, h["a"] / acc, h["flags"], h["dti"]


@pytest.mark.parametrize("starter", [G.STARTER_SERIES, G.STARTER_CLASSIC])
@pytest.mark.parametrize("kick", [G.KICK_FLOAT_FLOAT, G.KICK_FP64])
@pytest.mark.parametrize("unit", list(UNITS))
def test_same_block_in_other_units(unit, kick, starter):
    want = run(1.0, 1.0, kick, starter)
    got = run(*UNITS[unit], kick, starter)
    assert np.array_equal(got[3], want[3]) and np.array_equal(got[4], want[4])
    assert (want[3] == 0).sum() > 400 and (want[3] != 0).sum() >= 3
    ok = want[3] == 0
    # a few 2^-53 a step in each, carried along (33 steps of at most tau = 0.5 at the
    # innermost pericentres); the planets' pull, below 1e-3 of the Sun's, to 1e-13 of its
    # own size, in units where the pull's two forms (float-float, FP64 beyond its
    # range) differ by that
    tol = 2 * 1.2e-15 * STEPS * (1 + 0.5 * STEPS) + 1e-3 * 1e-13 * STEPS ** 2 * 0.25
    for a, b in zip(got[:2], want[:2]):
        err = np.linalg.norm(a[ok] - b[ok], axis=1) / np.linalg.norm(b[ok], axis=1)
        assert err.max() < tol, (err.max(), tol)
    err = np.linalg.norm(got[2][ok] - want[2][ok], axis=1) / np.linalg.norm(want[2][ok], axis=1)
    assert err.max() < 1e-11           # the planets' accelerations nearly cancel against h0 far out


@pytest.mark.parametrize("kick", [G.KICK_FLOAT_FLOAT, G.KICK_FP64])
def test_classic_starter_against_the_series(kick):
    want, got = run(1.0, 1.0, kick, G.STARTER_SERIES), run(1.0, 1.0, kick, G.STARTER_CLASSIC)
    assert np.array_equal(got[3], want[3])
    ok = want[3] == 0
    tol = 2 * 1.2e-15 * STEPS * (1 + 0.5 * STEPS)
    for a, b in zip(got[:2], want[:2]):
        err = np.linalg.norm(a[ok] - b[ok], axis=1) / np.linalg.norm(b[ok], axis=1)
        assert err.max() < tol, (err.max(), tol)
