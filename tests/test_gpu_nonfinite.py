"""Particles and planet logs that hold NaN, an infinity or a value beyond a
float's range, at steps short enough for the small-step drift: the particle is
flagged at its first step as the FP64 drift flags it (outer limit, not converged,
unbound), its neighbours' results stay bit for bit what they are without it, and a
planet position that is not finite leaves no particle unflagged."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import glisser_gb300 as G  # noqa: E402

MU = 2.959122e-4
N, STEPS = 200, 6
# beyond the outer limit; where |r|^2 overflows, 1/|r| = 0 and the energy is that
# of an unbound orbit (0x08)
FAR = [2.0 ** 127, -1e40, 2.0 ** 216, 3e77, 1e150, np.inf, -np.inf, -1e300]
FAR_FLAGS = [0x02] * 5 + [0x08] * 3


@pytest.fixture(scope="module", autouse=True)
def native():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    G.build()
    G.lib()


def swarm():
    rng = np.random.default_rng(4)
    el = np.stack([rng.uniform(40, 50, N), rng.uniform(0, 0.1, N), rng.uniform(0, 0.1, N),
                   *rng.uniform(0, 2 * np.pi, (3, N))], 1)
    return G.elements_to_cartesian(MU, el)


def block(r, v, dt, kick, planet=(30.0, 1.0, 0.1), starter=G.STARTER_SERIES):
    from gpu_util import DevHandoff, DevParticles, DevPlanetBlock, timeblock
    p = DevParticles(r, v, np.zeros((N, 3)), np.zeros(N), np.arange(N))
    b = DevPlanetBlock(np.zeros((STEPS, 3)), np.tile(planet, (STEPS, 1, 1)), [MU, 5e-5 * MU], [0, 4], [0.5, 0.5])
    timeblock(p, b, dt, 300.0, handoff=DevHandoff(N), kick=kick, starter=starter, encounters=G.ENCOUNTERS_KILL)
    return p.host()


@pytest.mark.parametrize("kick", [G.KICK_FLOAT_FLOAT, G.KICK_FP64])
@pytest.mark.parametrize("dt", [1.0, 2.0, 180.0])
def test_bad_particles_are_flagged_and_alone(dt, kick):
    r, v = swarm()
    good = block(r, v, dt, kick)
    assert not good["flags"].any()
    bad = np.zeros(N, bool)
    r2, v2 = r.copy(), v.copy()
    for k, x in enumerate(FAR):
        r2[3 * k, k % 3] = x
    at = 3 * len(FAR)
    for k in range(3):
        r2[at + 3 * k, k] = np.nan
        v2[at + 3 * k + 1, k] = np.nan
        v2[at + 3 * k + 2, k] = (np.inf, -1e40, 1e300)[k]
    bad[:at:3] = True
    bad[at:at + 9] = True
    got = block(r2, v2, dt, kick)
    assert np.array_equal(got["flags"][:at:3], FAR_FLAGS)
    assert np.all(got["flags"][at:at + 9] != 0) and np.all(got["flags"][at:at + 9:3] & 0x04)
    assert np.all(got["dti"][bad] == 1)
    for key in ("r", "v", "a", "flags", "dti"):
        assert np.array_equal(got[key][~bad], good[key][~bad]), key
    # the general drift alone (the classic starter's) sets the same flags
    assert np.array_equal(block(r2, v2, dt, kick, starter=G.STARTER_CLASSIC)["flags"], got["flags"])


@pytest.mark.parametrize("kick", [G.KICK_FLOAT_FLOAT, G.KICK_FP64])
@pytest.mark.parametrize("planet", [(np.nan, 1.0, 0.1), (30.0, 1.0, np.nan)])
def test_planet_position_that_is_not_a_number(planet, kick):
    r, v = swarm()
    assert block(r, v, 1.0, kick, planet)["flags"].all()
