"""The device planet integrator against a numpy restatement with converged
Kepler solutions (the host integrator's iteration stops 1e-14 rad short, a part
in 1e12 of a small step) over the planet counts that choose its kernel (a lane per vector component up to five planets, a lane per
planet beyond) and steps on both sides of the drift's choice (universal
variables for modest steps, the eccentric-anomaly iteration for wide ones)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import glisser_gb300 as G  # noqa: E402
from perf.cases import _planet_wh  # noqa: E402

GM = 2.959122e-4
STEPS, BLOCKS = 33, 3


@pytest.fixture(scope="module", autouse=True)
def native():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    G.build()
    G.lib()


def system(rng, planets, e_max):
    a = 5.2 * 1.5 ** np.arange(planets)
    m = np.concatenate([[GM], GM * 10 ** rng.uniform(-6, -4, planets)])
    pr, pv = [np.zeros(3)], [np.zeros(3)]
    for j in range(planets):
        el = [[a[j], rng.uniform(0, e_max), rng.uniform(0, 0.05), *rng.uniform(0, 2 * np.pi, 3)]]
        r, v = G.elements_to_cartesian(m[0] + m[j + 1], el)
        pr.append(r[0])
        pv.append(v[0])
    r, v = G.elements_to_cartesian(m[0], np.stack([rng.uniform(40, 50, 5) * 1.5 ** max(0, planets - 4),
                                                   np.zeros(5), np.zeros(5), *rng.uniform(0, 6, (3, 5))], 1))
    return m, np.array(pr), np.array(pv), r, v


def run(syst, dt, device):
    ens = G.Ensemble("Time-Step %r\nTime-Block-Size %d\nFinal-Time 1e30\nCull-Radius 0.5\nOuter-Limit 1e6\n"
                     "Encounter-RH-Factor 3\nInput-File x\nOutput-Folder x\n" % (dt, STEPS), len(syst))
    for s, (m, pr, pv, r, v) in enumerate(syst):
        ens.set_system(s, m, pr, pv, r, v)
    ens.set_device_planets(device)
    ens.init()
    for _ in range(BLOCKS):
        ens.step()
    return ens


# the innermost planet's step: 20 d, 0.03 rad; 180 d, 0.26 rad; 400 d, 0.58 rad, past
# the universal-variable drift's bound (0.5 rad); 1,000 d, 1.45 rad
@pytest.mark.parametrize("dt", [20.0, 180.0, 400.0, 1000.0])
@pytest.mark.parametrize("planets,e_max", [(1, 0.05), (2, 0.3), (3, 0.05), (4, 0.05), (4, 0.6), (5, 0.1), (6, 0.05),
                                           (11, 0.02)])
def test_device_planets(planets, e_max, dt):
    rng = np.random.default_rng(100 * planets)
    syst = [system(rng, planets, e_max) for _ in range(3)]
    dev, host = run(syst, dt, True), run(syst, dt, False)
    # an ulp or two per drift, carried through the orbit's shear: 99 steps of up
    # to 1.45 rad, magnified by 1 / (1 - e)^2 at pericentre and by close approaches
    # of eccentric planets
    tol = 99 * 1e-15 * (1 + 99 * dt * np.sqrt(GM / 5.2 ** 3)) * (1 - e_max) ** -2 * (100 if e_max > 0.2 else 1)
    for s in range(len(syst)):
        m, pr, pv = syst[s][:3]
        want = _planet_wh(m[None], pr[None], pv[None], dt, STEPS * BLOCKS)[0][-1, 0, 1:]
        err = np.linalg.norm(dev.planets(s)["r"][1:] - want, axis=1) / np.linalg.norm(want, axis=1)
        assert err.max() < tol, (err.max(), tol)
        pa, pb = dev.particles(s), host.particles(s)
        assert np.array_equal(pa["flags"], pb["flags"])
