"""The quick phase of crmath.cuh's log (Ziv's rounding test around one double
and its tail), compiled for the host: every value it settles is the correctly
rounded logarithm -- the accurate double-double phase's value on a million
arguments, and the exact value rounded (60 digits) wherever the two differ -- and
it leaves only a few in a thousand to the accurate phase."""
import ctypes
import os
import subprocess
import tempfile
from decimal import Decimal, getcontext

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mckl_b200", "csrc")
SRC = r"""
#include "crmath.cuh"
extern "C" void acc(long n, const double *x, double *y) { for (long i = 0; i < n; ++i) y[i] = mckl_b200::dd::log_dd(x[i]); }
extern "C" void both(long n, const double *x, double *y) { for (long i = 0; i < n; ++i) y[i] = mckl_b200::dd::log(x[i]); }
extern "C" void quick(long n, const double *x, double *y, unsigned char *ok) {
    for (long i = 0; i < n; ++i) { y[i] = 0; ok[i] = mckl_b200::dd::log_quick(x[i], y + i); }
}
"""


@pytest.fixture(scope="module")
def lib():
    d = tempfile.mkdtemp()
    src, so = os.path.join(d, "lq.cpp"), os.path.join(d, "liblq.so")
    with open(src, "w") as f:
        f.write(SRC)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, src, "-o", so],
                       capture_output=True, text=True)
    if r.returncode != 0:
        pytest.skip("host compiler unavailable: " + r.stderr[:200])
    return ctypes.CDLL(so)


def call(fn, x, *more):
    y = np.empty_like(x)
    fn(ctypes.c_long(len(x)), *[a.ctypes.data_as(ctypes.c_void_p) for a in (x, y) + more])
    return y


def test_log_quick_is_correctly_rounded(lib):
    rng = np.random.default_rng(21)
    u = (rng.integers(0, 2**32, 500000).astype(np.float64) + 0.5) * 2.0**-32
    xs = np.ascontiguousarray(np.concatenate([
        u, np.exp(rng.uniform(-708, 709, 200000)),                      # the whole normal range
        1.0 + rng.integers(-2**30, 2**30, 200000) * 2.0**-52,           # around 1: the sum cancels
        (1.0 + rng.integers(0, 129, 100000) / 128.0) * (1 + rng.integers(-8, 9, 100000) * 2.0**-52),  # table edges
        np.ldexp(1.0 + rng.random(50000) * 2.0**-30, rng.integers(-1021, 1023, 50000)),
    ]))
    xs = xs[xs >= 2.2250738585072014e-308]
    ok = np.zeros(len(xs), dtype=np.uint8)
    q = call(lib.quick, xs, ok)
    a = call(lib.acc, xs)
    taken = ok == 1
    differ = np.flatnonzero(taken & (q.view(np.int64) != a.view(np.int64)))
    assert len(differ) <= 20
    getcontext().prec = 60
    for i in differ:  # the accurate phase is off in a few cases per million
        assert q[i] == float(Decimal(float(xs[i])).ln()), xs[i]
    n = 500000
    assert taken[:n].mean() >= 0.995, taken[:n].mean()


def test_log_special_values(lib):
    xs = np.array([0.0, -0.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, 2.2250738585072009e-308, 1.0, 1.7976931348623157e308])
    got, want = call(lib.both, xs), call(lib.acc, xs)
    assert np.array_equal(got.view(np.int64)[~np.isnan(got)], want.view(np.int64)[~np.isnan(want)])
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = np.zeros(len(xs), dtype=np.uint8)
    call(lib.quick, xs, ok)
    assert not ok[:8].any()  # zero, negative, infinite, NaN and subnormal arguments
