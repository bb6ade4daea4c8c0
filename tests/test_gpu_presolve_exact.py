"""Drifts that the FP32 pre-solve starts (tau^2 of 0.01 and more), one step each
against a long-double Kepler solution, with each particle's own bound: where the
Stumpff argument stays below 4.5 (the series to x^11, no quartering) a drift lands at
FP64 rounding times the orbit's own conditioning."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import glisser_gb300 as G  # noqa: E402
from glisser_gb300 import learned as L  # noqa: E402

LD = np.longdouble
MU, DT = 2.959122e-4, 180.0


@pytest.fixture(scope="module", autouse=True)
def native():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    G.build()
    G.lib()


def exact(r, v):
    """r', v' and the step's eccentric anomaly dE, all in long double."""
    r, v, mu, dt = r.astype(LD), v.astype(LD), LD(MU), LD(DT)
    r0 = np.sqrt((r * r).sum(1))
    u = (r * v).sum(1)
    a = 1 / (2 / r0 - (v * v).sum(1) / mu)
    n = np.sqrt(mu / a ** 3)
    ec, es = 1 - r0 / a, u / (n * a * a)
    dm = n * dt
    de = dm + 0
    for _ in range(60):
        f = de - ec * np.sin(de) + es * (1 - np.cos(de)) - dm
        fp = 1 - ec * np.cos(de) + es * np.sin(de)
        de = de - np.clip(f / fp, -0.5, 0.5)
    s, h = np.sin(de), np.sin(de / 2)
    c1 = -2 * h * h                      # cos(de) - 1
    fp = 1 - ec * (1 + c1) + es * s
    f, g = 1 + a * c1 / r0, dt + (s - de) / n
    fd, gd = -n * s * a / (r0 * fp), 1 + c1 / fp
    return f[:, None] * r + g[:, None] * v, fd[:, None] * r + gd[:, None] * v, de.astype(np.float64)


@pytest.mark.parametrize("starter", [G.STARTER_SERIES, G.STARTER_CLASSIC])
@pytest.mark.parametrize("lo,hi", [(0.12, 0.5), (0.5, 1.0), (1.0, 2.0), (2.0, 7.9), (8.1, 40.0)])
def test_wide_drift_lands_at_its_conditioning(lo, hi, starter):
    n = 4096
    rng = np.random.default_rng(61)
    dM = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    a = np.cbrt(MU * (DT / dM) ** 2)
    e = rng.uniform(0, 0.7, n)
    el = np.stack([a, e, rng.uniform(0, 1, n), *rng.uniform(0, 2 * np.pi, (3, n))], 1)
    r, v = G.elements_to_cartesian(MU, el)
    got = L.drift_states(r, v, DT, MU, starter)
    assert not got[3].any()
    want = exact(r, v)
    # a rounding of the state moves 1/a by (2a / r0) of it and the mean anomaly of the
    # step by 3/2 dM of that; a step off in M by d lands off by d sqrt((1+e)/(1-e)^3) of
    # |r'| at most (of |v'|: once more 1 / (1 - e)).  Eight roundings of each kind, and
    # each quartering of x = dE^2 from 4.5 on doubles the Stumpff functions' error; the
    # first of them goes from 4.5 to below 0.1, three at once
    x = want[2] ** 2
    q = np.where(x < 4.4, 0, np.ceil(np.log(np.maximum(x, 0.1) / 0.1) / np.log(4)))
    cond = 1 + 3 * dM / (1 - e) * np.sqrt((1 + e) / (1 - e) ** 3)
    bound = 8 * 2.0 ** -53 * cond * 4 ** q
    for k, extra in ((0, 1.0), (1, 1 / (1 - e))):
        err = np.linalg.norm((got[k] - want[k]).astype(np.float64), axis=1)
        err /= np.linalg.norm(want[k].astype(np.float64), axis=1)
        assert np.all(err <= bound * extra), (err / (bound * extra)).max()
