"""The small-step drift's constants mu dt^2 / 2 and mu dt of the central mass,
compiled for the host: a constant's error is the same at every step of a run, so it
must be a rounding (to either side), not a truncation."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LD = np.longdouble


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("host") / "constants.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "tests", "host_cuda"), "-I" + os.path.join(ROOT, "glisser_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "host_cuda", "constants_check.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def test_sun_constants_are_rounded(lib):
    rng = np.random.default_rng(1)
    n = 100_000
    mu = np.concatenate([[2.9591220828559e-4, 2.959122e-4, 4 * np.pi ** 2], np.exp(rng.uniform(-9, 4, n))])
    dt = np.concatenate([[50.0, 180.0, 0.2], np.exp(rng.uniform(-5, 6, n))])
    a, b = np.zeros((n + 3, 2), np.float32), np.zeros((n + 3, 2), np.float32)
    p = [x.ctypes.data_as(C.c_void_p) for x in (mu, dt, a, b)]
    lib.sun_constants(n + 3, *p)
    for got, want in ((a, mu.astype(LD) * dt * dt / 2), (b, mu.astype(LD) * dt)):
        err = ((got[:, 0].astype(LD) + got[:, 1] - want) / want).astype(np.float64)
        # the float-float holds 49 bits (lo to nearest: 2^-49 of the whole at most), the
        # product in FP64 one or two roundings of 2^-53
        assert np.abs(err).max() <= 2.0 ** -49 + 2 * 2.0 ** -53
        # no side is preferred: the mean of n errors spread over +-2^-49 stays within
        # four of its standard deviations
        assert abs(err.mean()) <= 4 * 2.0 ** -49 / np.sqrt(3 * n)
