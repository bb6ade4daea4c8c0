"""Drifts at the edges of the Stumpff evaluation's ranges (series to x^6 below
|x| = 0.1, to x^11 below 4.5, quartered beyond; x = alpha s^2, about the square of
the step's eccentric anomaly), elliptic and hyperbolic, against long double."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import glisser_gb300 as G  # noqa: E402

LD = np.longdouble


@pytest.fixture(scope="module", autouse=True)
def native():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    G.build()
    G.lib()


def g_long_double(s, alpha):
    """G1, G2, G3 by their series (to x^24: |x| <= 20)."""
    s, alpha = s.astype(LD), alpha.astype(LD)
    x = alpha * s * s
    c2, c3 = np.zeros_like(x), np.zeros_like(x)
    t2, t3 = np.full_like(x, LD(1) / 2), np.full_like(x, LD(1) / 6)
    for k in range(40):
        c2, c3 = c2 + t2, c3 + t3
        t2, t3 = -t2 * x / ((2 * k + 3) * (2 * k + 4)), -t3 * x / ((2 * k + 4) * (2 * k + 5))
    g3 = s * s * s * c3
    return s - alpha * g3, s * s * c2, g3


@pytest.mark.parametrize("lo,hi", [(2e-3, 0.1), (0.099, 0.101), (0.1, 1.0), (1.0, 4.49), (4.4, 4.6), (4.51, 9.0)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_g_functions(lo, hi, sign):
    n = 4096
    rng = np.random.default_rng(3)
    s = np.exp(rng.uniform(-3, 3, n))
    alpha = sign * rng.uniform(lo, hi, n) / (s * s)
    _, g1, g2, g3 = G.drift_math_check(np.ones(n), s, alpha, np.ones(n, np.float32))
    for got, want, scale in zip((g1, g2, g3), g_long_double(s, alpha), (s, s * s / 2, s ** 3 / 6)):
        # Horner and three products in units of 2^-53 of the leading term, times the
        # terms' sum of magnitudes over it (cosh of the half anomaly: 1.6 at |x| = 4.5);
        # beyond 4.5 each of the three quarterings doubles what it finds
        bound = 2.0 ** -53 * (8 if hi < 4.4 else 64) * np.cosh(np.sqrt(hi) / 2)
        err = np.abs((got - want) / np.maximum(np.abs(want), scale)).astype(np.float64)
        assert err.max() < bound, (err.max(), bound)
