"""The float64 quotient from a reciprocal (csrc/quotient.cuh), compiled for the
host, against the division it stands for: equal bit for bit, also where an
operand is infinite, not a number or zero (up to the sign of a zero)."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "mirgecom_b200", "csrc")
SOURCE = """
#define __host__
#define __device__
#define __forceinline__ inline
#include "quotient.cuh"
extern "C" void quotients(long n, const double* x, const double* y, double* out) {
  for (long i = 0; i < n; ++i) out[i] = mgc::quotient(x[i], y[i], 1.0 / y[i]);
}
"""


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotient")
    src, lib = str(d / "quotient.cpp"), str(d / "quotient.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    CSRC, "-o", lib, src], check=True)
    fn = ctypes.CDLL(lib).quotients
    fn.restype = None
    fn.argtypes = [ctypes.c_long] + [np.ctypeslib.ndpointer(np.float64, flags="C")] * 3

    def run(x, y):
        out = np.empty_like(x)
        fn(len(x), np.ascontiguousarray(x), np.ascontiguousarray(y), out)
        return out
    return run


def _equal(got, x, y):
    with np.errstate(all="ignore"):
        want = x / y
    assert np.array_equal(got, want, equal_nan=True)


def test_special_operands(quotients):
    v = np.array([0.0, 1.0, 1.2, 3.0, 1e-3, 7e5, 1e-280, 1e280, np.inf])
    v = np.concatenate([v, -v, [np.nan]])
    x, y = (a.ravel().copy() for a in np.meshgrid(v, v))
    # quotients of finite operands within the normal range (their mantissas are
    # covered below)
    with np.errstate(all="ignore"):
        r = np.abs(x / y)
    ok = ~np.isfinite(x) | ~np.isfinite(y) | (y == 0) | (x == 0) | ((r > 1e-270) & (r < 1e300))
    _equal(quotients(x, y)[ok], x[ok], y[ok])


@pytest.mark.parametrize("near_two", [False, True])
def test_random_operands(quotients, near_two):
    """*near_two*: mantissas within 4096 units of 2, where the reciprocal is
    least accurate against the quotient's last place."""
    g = np.random.default_rng(7)
    n = 1 << 20
    if near_two:
        y = np.nextafter(2.0, 0.0) - g.integers(0, 4096, n) * 2.0 ** -52
        x = y - g.integers(0, 4096, n) * 2.0 ** -52
    else:
        x = g.uniform(1.0, 2.0, n) * 2.0 ** g.integers(-400, 400, n)
        y = g.uniform(1.0, 2.0, n) * 2.0 ** g.integers(-60, 60, n)
    _equal(quotients(x, y), x, y)
