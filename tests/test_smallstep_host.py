"""The small-step drift's device arithmetic (smallstep.cuh) compiled for the
host and compared with long double: the float-float conversions at their
edges, the reciprocals, and whole drifts over the domain and at its bounds."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LD = np.longdouble
MU, DT = 2.959122e-4, 180.0
TAU2_MAX = 1e-3


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("host") / "smallstep.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "tests", "host_cuda"), "-I" + os.path.join(ROOT, "glisser_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "host_cuda", "smallstep_check.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def split(lib, d):
    hi, lo = np.zeros(len(d), np.float32), np.zeros(len(d), np.float32)
    lib.split(len(d), ptr(d), ptr(hi), ptr(lo))
    return hi, lo


def test_split_of_a_double(lib):
    rng = np.random.default_rng(1)
    d = np.ldexp(1 + rng.random(200_000), rng.integers(-70, 126, 200_000)) * rng.choice([-1.0, 1.0], 200_000)
    edge = np.array([1.0, -1.0, 2.0, 1 - 2.0 ** -53, 1 + 2.0 ** -52, 1 + 2.0 ** -24, 1 + 2.0 ** -24 + 2.0 ** -52,
                     2 - 2.0 ** -24, 2 - 2.0 ** -25, 2 - 2.0 ** -52, 2.0 ** -70, 3 * 2.0 ** -71])
    d = np.concatenate([d, edge, -edge])
    hi, lo = split(lib, d)
    err = np.abs(d.astype(LD) - hi.astype(LD) - lo.astype(LD))
    assert np.all(err <= 2.0 ** -49 * np.abs(d))
    # zero stays zero; below 2^-70 the other split's bound, down to its own range
    hi, lo = split(lib, np.array([0.0, -0.0]))
    assert not hi.any() and not lo.any()
    d = np.ldexp(1 + rng.random(1000), rng.integers(-95, -70, 1000))
    hi, lo = split(lib, d)
    assert np.all(np.abs(d.astype(LD) - hi.astype(LD) - lo.astype(LD)) <= 2.0 ** -47 * d)


def test_float_float_widened_to_double(lib):
    rng = np.random.default_rng(2)
    n = 200_000
    hi = (np.ldexp(1 + rng.random(n), rng.integers(-75, 60, n)) * rng.choice([-1.0, 1.0], n)).astype(np.float32)
    hi[:2000] = np.ldexp(1.0, rng.integers(-75, 60, 2000))       # powers of two: the binade below
    hi[2000:4000] = np.nextafter(hi[:2000], np.float32(0))       # and the last float before one
    ulp = np.spacing(np.abs(hi)).astype(np.float64)
    lo = (ulp * rng.uniform(-0.25, 0.25, n)).astype(np.float32)
    hi = np.concatenate([hi, np.float32([0.0, -0.0, 1e-30, 1.0])])
    lo = np.concatenate([lo, np.float32([0.0, 0.0, 1e-38, -2.0 ** -26])])
    got = np.zeros(len(hi))
    lib.widen(len(hi), ptr(hi), ptr(lo), ptr(got))
    exact = hi.astype(LD) + lo.astype(LD)
    assert np.all(np.abs(got - exact) <= 2.0 ** -46 * np.abs(exact))
    assert got[n] == 0 and got[n + 1] == 0


def test_reciprocals(lib):
    rng = np.random.default_rng(3)
    n = 100_000
    x = np.ldexp(1 + rng.random(n), rng.integers(-40, 44, n))
    f = [np.zeros(n, np.float32) for _ in range(4)]
    lib.inverses(n, ptr(x), *[ptr(a) for a in f])
    s = (f[0].astype(LD) + f[1]) * np.sqrt(x.astype(LD)) - 1
    r = (f[2].astype(LD) + f[3]) * x.astype(LD) - 1
    # three roundings of 2^-24 numbers and the split of x: 2^-46; no bias above 2^-52
    for e in (s, r):
        assert np.abs(e).max() < 2.0 ** -46 and abs(e.mean()) < 2.0 ** -52


def states(tau2, e, seed, sign=1.0):
    """States at tau^2 = dt^2 mu / r^3 on orbits of eccentricity e."""
    rng = np.random.default_rng(seed)
    n = len(tau2)
    r = np.cbrt(DT * DT * MU / tau2)
    a = r / rng.uniform(1 - 0.999 * e, 1 + 0.999 * e)
    cE = np.clip(np.where(e > 0, (1 - r / a) / np.maximum(e, 1e-12), rng.uniform(-1, 1, n)), -1, 1)
    M = np.arccos(cE) * rng.choice([-1.0, 1.0], n)
    q, w = np.sqrt(1 - e * e), np.sqrt(MU / a ** 3)
    x, y = a * (cE - e), a * q * np.sin(M)
    d = w / (1 - e * cE)
    vx, vy = -a * np.sin(M) * d, a * q * cE * d * sign
    th, inc = rng.uniform(0, 2 * np.pi, n), rng.uniform(0, 1, n)
    c, s, ci, si = np.cos(th), np.sin(th), np.cos(inc), np.sin(inc)
    return np.stack([x * c - y * s, (x * s + y * c) * ci, (x * s + y * c) * si,
                     vx * c - vy * s, (vx * s + vy * c) * ci, (vx * s + vy * c) * si], 1)


def drift_long_double(rv, dt, mu):
    r, v = rv[:, :3].astype(LD), rv[:, 3:].astype(LD)
    dt, mu = LD(dt), LD(mu)
    r0 = np.sqrt((r * r).sum(1))
    u = (r * v).sum(1)
    al = 2 * mu / r0 - (v * v).sum(1)
    s = dt / r0
    for _ in range(8):
        x = al * s * s
        c2, c3 = LD(0), LD(0)
        f2, f3 = LD(1) / 2, LD(1) / 6
        for k in range(10):
            c2, c3 = c2 + f2, c3 + f3
            f2, f3 = -f2 * x / ((2 * k + 3) * (2 * k + 4)), -f3 * x / ((2 * k + 4) * (2 * k + 5))
        g2, g3 = s * s * c2, s * s * s * c3
        g0, g1 = 1 - al * g2, s - al * g3
        s = s - (r0 * g1 + u * g2 + mu * g3 - dt) / (r0 * g0 + u * g1 + mu * g2)
    f, g = (-mu / r0 * g2)[:, None], (dt - mu * g3)[:, None]
    nr = r + (f * r + g * v)
    n0 = np.sqrt((nr * nr).sum(1))
    return nr, v + ((-mu * g1 / (r0 * n0))[:, None] * r + (-mu * g2 / n0)[:, None] * v)


@pytest.mark.parametrize("lo,hi", [(1e-8, 1e-6), (1e-6, 1e-4), (1e-4, 0.9999e-3)])
@pytest.mark.parametrize("kind", ["spread", "circular", "retrograde", "planar", "eccentric"])
def test_drift_against_long_double(lib, lo, hi, kind):
    n = 4000
    rng = np.random.default_rng(7)
    e = {"circular": np.zeros(n), "eccentric": rng.uniform(0.9, 0.99, n)}.get(kind, rng.uniform(0, 0.9, n))
    rv = states(np.exp(rng.uniform(np.log(lo), np.log(hi), n)), e, 8, -1.0 if kind == "retrograde" else 1.0)
    if kind == "planar":
        rv[:, 2] = rv[:, 5] = 0.0
    want_r, want_v = drift_long_double(rv, DT, MU)
    v0 = np.linalg.norm(rv[:, 3:], axis=1)
    r0 = np.linalg.norm(rv[:, :3], axis=1)
    ok = np.zeros(n, np.int32)
    lib.drift(n, C.c_double(DT), C.c_double(MU), ptr(rv), ptr(ok))
    # every state of a planar cut of an inclined orbit may change its tau^2, not its bounds
    assert ok.mean() > (0.5 if kind == "planar" else 0.999)
    keep = ok == 1
    er = np.sqrt(((rv[:, :3] - want_r) ** 2).sum(1)) / r0
    ev = np.sqrt(((rv[:, 3:] - want_v) ** 2).sum(1)) / v0
    # one FP64 rounding per component (2^-53 of |r|) and a correction of at most
    # tau^2 / 2 < 5e-4 known to 2^-40; the velocity's correction is of the size
    # tau v_circ, known to 2^-45
    kick = np.sqrt(MU / r0 ** 3) * DT * np.sqrt(MU / r0) / v0
    assert np.all(er[keep] <= 2.0 ** -53 * np.sqrt(3) + 5e-4 * 2.0 ** -40)
    assert np.all(ev[keep] <= 2.0 ** -53 * np.sqrt(3) + (2.0 ** -45 * kick)[keep])
    if kind == "planar":
        assert not rv[:, 2].any() and not rv[:, 5].any()


def test_drift_leaves_what_is_outside_its_domain(lib):
    n = 500
    e = np.full(n, 0.3)
    wide = states(np.full(n, 1.001 * TAU2_MAX), e, 1)
    tiny = states(np.full(n, 1e-10), e, 2)
    fast = states(np.full(n, 1e-4), e, 3)
    fast[:, 3:] *= 1.5 * np.sqrt(2 * MU / np.linalg.norm(fast[:, :3], axis=1) / (fast[:, 3:] ** 2).sum(1))[:, None]
    bad = states(np.full(n, 1e-4), e, 4)
    bad[:, 0] = np.nan
    for rv in (wide, tiny, fast, bad):
        before = rv.copy()
        ok = np.zeros(n, np.int32)
        lib.drift(n, C.c_double(DT), C.c_double(MU), ptr(rv), ptr(ok))
        assert not ok.any() and np.array_equal(rv, before, equal_nan=True)


def gfuns_long_double(rv, dt, mu):
    r, v = rv[:, :3].astype(LD), rv[:, 3:].astype(LD)
    dt, mu = LD(dt), LD(mu)
    r0 = np.sqrt((r * r).sum(1))
    u = (r * v).sum(1)
    al = 2 * mu / r0 - (v * v).sum(1)
    s = dt / r0
    for _ in range(10):
        x = al * s * s
        c2, c3 = LD(0), LD(0)
        f2, f3 = LD(1) / 2, LD(1) / 6
        for k in range(12):
            c2, c3 = c2 + f2, c3 + f3
            f2, f3 = -f2 * x / ((2 * k + 3) * (2 * k + 4)), -f3 * x / ((2 * k + 4) * (2 * k + 5))
        g2, g3 = s * s * c2, s * s * s * c3
        g0, g1 = 1 - al * g2, s - al * g3
        s = s - (r0 * g1 + u * g2 + mu * g3 - dt) / (r0 * g0 + u * g1 + mu * g2)
    return g1, g2, g3


@pytest.mark.parametrize("lo,hi", [(1.0001e-3, 2e-3), (2e-3, 5e-3), (5e-3, 0.9999e-2)])
@pytest.mark.parametrize("kind", ["spread", "circular", "retrograde", "eccentric"])
def test_medium_solution_against_long_double(lib, lo, hi, kind):
    n = 4000
    rng = np.random.default_rng(17)
    e = {"circular": np.zeros(n), "eccentric": rng.uniform(0.9, 0.99, n)}.get(kind, rng.uniform(0, 0.9, n))
    rv = states(np.exp(rng.uniform(np.log(lo), np.log(hi), n)), e, 18, -1.0 if kind == "retrograde" else 1.0)
    tier, g = np.zeros(n, np.int32), np.zeros((n, 3))
    lib.gfuns_medium(n, C.c_double(DT), C.c_double(MU), ptr(rv), ptr(tier), ptr(g))
    assert (tier == 2).all()
    want = gfuns_long_double(rv, DT, MU)
    r0 = np.linalg.norm(rv[:, :3], axis=1)
    v0 = np.linalg.norm(rv[:, 3:], axis=1)
    # what the G-functions carry into the state: mu G2 / r0 into r, mu G3 into the
    # time step, mu G1 / r0^2 and mu G2 / r0 into v; each may add a quarter of the
    # state's own FP64 rounding: 2^-55 of |r0| and 2^-53 of the velocity's scale
    vs = np.maximum(v0, np.sqrt(MU / r0))
    d1, d2, d3 = (np.abs(g[:, k] - want[k]) for k in range(3))
    assert np.all(MU * d2 / r0 <= 2.0 ** -55)
    assert np.all(MU * d3 * v0 / r0 <= 2.0 ** -55)
    assert np.all(MU * d1 / r0 <= 2.0 ** -53 * vs)
    assert np.all(MU * d2 / r0 * v0 <= 2.0 ** -53 * vs)


def test_medium_solution_leaves_the_rest(lib):
    n = 500
    e = np.full(n, 0.3)
    below, above = states(np.full(n, 0.999e-3), e, 21), states(np.full(n, 1.001e-2), e, 22)
    fast = states(np.full(n, 5e-3), e, 23)
    fast[:, 3:] *= 1.5 * np.sqrt(2 * MU / np.linalg.norm(fast[:, :3], axis=1) / (fast[:, 3:] ** 2).sum(1))[:, None]
    for rv, want in ((below, 1), (above, 0), (fast, 0)):
        tier, g = np.full(n, -1, np.int32), np.zeros((n, 3))
        lib.gfuns_medium(n, C.c_double(DT), C.c_double(MU), ptr(rv), ptr(tier), ptr(g))
        assert (tier == want).all() and not g.any()


@pytest.mark.parametrize("e_max", [0.0, 0.6, 0.99])
def test_drift_far_out_against_long_double(lib, e_max):
    # the lower end of the domain, tau^2 down to 2^-33: every correction is below
    # tau^2, so one FP64 rounding a component and 2^-40 of the correction remain
    n = 4000
    rng = np.random.default_rng(31)
    rv = states(np.exp(rng.uniform(np.log(1.2e-10), np.log(1e-8), n)), rng.uniform(0, e_max, n), 32)
    want_r, want_v = drift_long_double(rv, DT, MU)
    v0, r0 = np.linalg.norm(rv[:, 3:], axis=1), np.linalg.norm(rv[:, :3], axis=1)
    ok = np.zeros(n, np.int32)
    lib.drift(n, C.c_double(DT), C.c_double(MU), ptr(rv), ptr(ok))
    assert ok.mean() > 0.99
    k = ok == 1
    er = np.sqrt(((rv[:, :3] - want_r) ** 2).sum(1)) / r0
    ev = np.sqrt(((rv[:, 3:] - want_v) ** 2).sum(1)) / v0
    kick = np.sqrt(MU / r0 ** 3) * DT * np.sqrt(MU / r0) / v0
    assert np.all(er[k] <= 2.0 ** -53 * np.sqrt(3) + 1e-8 * 2.0 ** -40)
    assert np.all(ev[k] <= 2.0 ** -53 * np.sqrt(3) + (2.0 ** -45 * kick)[k])
