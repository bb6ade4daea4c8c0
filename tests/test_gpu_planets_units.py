"""The device planet integrator in other units of length and time: the same system
in au and days, in metres and years and in centimetres and years, where G Msun is
beyond a float's range.  The positions agree to the rounding that each carries."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import glisser_gb300 as G  # noqa: E402

GM = 2.959122e-4
DT, STEPS, BLOCKS = 180.0, 33, 3
AU_M, YEAR_D = 1.495978707e11, 365.25


@pytest.fixture(scope="module", autouse=True)
def native():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    G.build()
    G.lib()


def positions(planets, length, time):
    rng = np.random.default_rng(planets)
    a = 5.2 * 1.5 ** np.arange(planets)
    m = np.concatenate([[GM], GM * 10 ** rng.uniform(-6, -4, planets)])
    pr, pv = [np.zeros(3)], [np.zeros(3)]
    for j in range(planets):
        el = [[a[j], rng.uniform(0, 0.1), rng.uniform(0, 0.05), *rng.uniform(0, 2 * np.pi, 3)]]
        r, v = G.elements_to_cartesian(m[0] + m[j + 1], el)
        pr.append(r[0])
        pv.append(v[0])
    r, v = G.elements_to_cartesian(GM, [[100.0, 0.0, 0.0, 1.0, 2.0, 3.0]])
    ens = G.Ensemble("Time-Step %r\nTime-Block-Size %d\nFinal-Time 1e30\nCull-Radius %r\nOuter-Limit %r\n"
                     "Input-File x\nOutput-Folder x\n" % (DT * time, STEPS, 0.5 * length, 1e6 * length), 1)
    ens.set_system(0, m * length ** 3 / time ** 2, np.array(pr) * length, np.array(pv) * (length / time), r * length,
                   v * (length / time))
    ens.set_device_planets(True)
    ens.init()
    for _ in range(BLOCKS):
        ens.step()
    return ens.planets(0)["r"][1:] / length


@pytest.mark.parametrize("length", [AU_M, 100 * AU_M])
@pytest.mark.parametrize("planets", [1, 4, 6])
def test_same_orbits_in_other_units(planets, length):
    want, got = positions(planets, 1.0, 1.0), positions(planets, length, 1 / YEAR_D)
    # an ulp or two a drift in each, carried through the orbit's shear over 99 steps
    tol = 2 * 99e-15 * (1 + 99 * DT * np.sqrt(GM / 5.2 ** 3)) * (1 - 0.1) ** -2
    err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert np.isfinite(got).all() and err.max() < tol, (err, tol)
