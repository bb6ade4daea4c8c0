"""Values that a float-float cannot hold -- NaN, the infinities, magnitudes of
2^127 and more -- through the small-step arithmetic (smallstep.cuh) compiled for
the host: the conversions must not turn them into ordinary numbers, and no tier of
the float-float drift may take a state that holds one, at any step."""
import ctypes as C

import numpy as np
import pytest

from test_smallstep_host import lib, ptr, split, states  # noqa: F401

DAY, YEAR = 2.959122e-4, 4 * np.pi ** 2          # G Msun in au^3 / d^2 and au^3 / yr^2
BAD = [np.nan, -np.nan, np.inf, -np.inf, 2.0 ** 127, 2.0 ** 128, -1e40, 2.0 ** 216, 2.0 ** 256, -3e77, 1e154, 1e300]


def test_split_of_what_a_float_cannot_hold(lib):  # noqa: F811
    hi, lo = split(lib, np.array([np.nan, -np.nan]))
    assert np.isnan(hi).all() and np.isnan(lo).all()
    big = np.array([np.inf, 2.0 ** 128, 1e40, 2.0 ** 256, 3e77, 1e300])
    for sign in (1.0, -1.0):
        hi, lo = split(lib, sign * big)
        assert np.array_equal(hi, np.full(len(big), sign * np.inf, np.float32)) and not lo.any()
    # the last values below 2^127 and the binade above it, still a float's
    d = np.array([np.nextafter(2.0 ** 127, 0), 2.0 ** 127, 1.7 * 2.0 ** 127])
    hi, lo = split(lib, d)
    assert np.all(np.abs(d.astype(np.longdouble) - hi.astype(np.longdouble) - lo.astype(np.longdouble)) <=
                  2.0 ** -47 * d)


def test_widening_keeps_nan_and_infinity(lib):  # noqa: F811
    hi = np.float32([np.nan, np.nan, 1.0, np.inf, -np.inf])
    lo = np.float32([np.nan, 0.0, 2.0 ** -30, 0.0, 0.0])
    got = np.zeros(5)
    lib.widen(5, ptr(hi), ptr(lo), ptr(got))
    assert np.isnan(got[:2]).all() and got[2] == 1 + 2.0 ** -30 and got[3] == np.inf and got[4] == -np.inf


@pytest.mark.parametrize("dt,mu,r", [(1.0, DAY, 50.0), (2.0, DAY, 5.0), (180.0, DAY, 50.0), (0.005, YEAR, 1.0),
                                     (0.2, YEAR, 30.0)])
def test_no_tier_takes_such_a_state(lib, dt, mu, r):  # noqa: F811
    base = states(np.full(len(BAD), 1e-4), np.full(len(BAD), 0.1), 1)
    # the same orbits at this distance and speed: tau^2 stays below the tiers' bounds
    scale = r / np.linalg.norm(base[:, :3], axis=1)
    base[:, :3] *= scale[:, None]
    base[:, 3:] *= (0.9 * np.sqrt(mu / r) / np.linalg.norm(base[:, 3:], axis=1))[:, None]
    ok = np.zeros(len(BAD), np.int32)
    lib.drift(len(BAD), C.c_double(dt), C.c_double(mu), ptr(base.copy()), ptr(ok))
    assert ok.all()                  # without the bad value every one is a small step
    for col in range(6):
        rv = base.copy()
        rv[:, col] = BAD
        before = rv.copy()
        for step in range(3):
            lib.drift(len(BAD), C.c_double(dt), C.c_double(mu), ptr(rv), ptr(ok))
            assert not ok.any(), (col, step, np.array(BAD)[ok != 0])
        assert np.array_equal(rv, before, equal_nan=True)
        tier, g = np.full(len(BAD), -1, np.int32), np.zeros((len(BAD), 3))
        lib.gfuns_medium(len(BAD), C.c_double(dt), C.c_double(mu), ptr(rv), ptr(tier), ptr(g))
        assert not tier.any(), (col, tier)
