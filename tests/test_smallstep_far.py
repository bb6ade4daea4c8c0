"""The small-step drift at steps that are a tiny part of the dynamical time (tau^2 from
1e-8 down to 1e-30: small steps, far particles), compiled for the host with the
kernels' lower bound and compared with long double, also at the corners of the
ranges of mu dt^2 / 2 (2^-40..2^30), dt (2^-24..2^24) and |r|^2 (2^-40..2^44)
within which the kernels use it."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from test_smallstep_host import DT, MU, ROOT, drift_long_double, ptr, states


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("host") / "far.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "tests", "host_cuda"), "-I" + os.path.join(ROOT, "glisser_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "host_cuda", "far_check.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def check(lib, rv, dt, mu, planar=False):
    n = len(rv)
    want_r, want_v = drift_long_double(rv, dt, mu)
    r0, v0 = np.linalg.norm(rv[:, :3], axis=1), np.linalg.norm(rv[:, 3:], axis=1)
    ok = np.zeros(n, np.int32)
    lib.drift_far(n, C.c_double(dt), C.c_double(mu), ptr(rv), ptr(ok))
    assert ok.mean() > (0.5 if planar else 0.99)
    k = ok == 1
    er = np.sqrt(((rv[:, :3] - want_r) ** 2).sum(1)) / r0
    ev = np.sqrt(((rv[:, 3:] - want_v) ** 2).sum(1)) / v0
    # one FP64 rounding a component; a position correction below tau^2 |r| known to
    # 2^-40 and a velocity correction of mu dt / r^2 known to 2^-45
    tau2 = dt * dt * mu / r0 ** 3
    assert np.all(er[k] <= (2.0 ** -53 * np.sqrt(3) + 2.0 ** -40 * tau2)[k])
    assert np.all(ev[k] <= (2.0 ** -53 * np.sqrt(3) + 2.0 ** -45 * mu * dt / (r0 * r0) / v0)[k])


@pytest.mark.parametrize("lo,hi", [(1e-12, 1e-8), (1e-20, 1e-12)])
@pytest.mark.parametrize("e_max", [0.0, 0.6, 0.99])
@pytest.mark.parametrize("planar", [False, True])
def test_far_drift_against_long_double(lib, lo, hi, e_max, planar):
    n = 4000
    rng = np.random.default_rng(51)
    rv = states(np.exp(rng.uniform(np.log(lo), np.log(hi), n)), rng.uniform(0, e_max, n), 52)
    scale = 1.0
    if lo < 1e-15:                      # the same tau^2 at a shorter step: |r| stays below 2^22
        scale = 1e-3
    dt = DT * scale
    rv[:, :3] *= scale ** (2 / 3)
    rv[:, 3:] *= scale ** (-1 / 3)
    if planar:
        rv[:, 2] = rv[:, 5] = 0.0
    check(lib, rv, dt, MU, planar)


@pytest.mark.parametrize("muh,dt", [(2.0 ** -39.9, 2.0 ** -23.9), (2.0 ** -39.9, 2.0 ** 23.9), (2.0 ** -39.9, 1.0),
                                    (2.0 ** 29.9, 2.0 ** -23.9), (2.0 ** 29.9, 2.0 ** 23.9), (2.0 ** 29.9, 1.0)])
def test_corners_of_the_ranges(lib, muh, dt):
    mu = 2 * muh / (dt * dt)
    n = 2000
    rng = np.random.default_rng(53)
    # distances up to the range's end and down to tau^2 = 9e-4
    lo, hi = max((2 * muh / 9e-4) ** (1 / 3), 2.0 ** -19.5), 2.0 ** 21.9
    r = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    base = states(DT * DT * MU / r ** 3, rng.uniform(0, 0.6, n), 54)     # |r| = r about MU
    base[:, 3:] *= np.sqrt(mu / MU)
    check(lib, base, dt, mu)
