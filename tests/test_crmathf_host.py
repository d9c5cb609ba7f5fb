"""The float log, exp, sin and cos of crmathf.cuh, compiled for the host from
the same source: every value that the short evaluations settle is the float
nearest to the double library function's value (the C library's here), and they
leave less than one argument in 10,000 of their ranges."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mckl_b200", "csrc")
SRC = r"""
#include "crmathf.cuh"
using namespace mckl_b200::dd;
extern "C" void f_log(long n, const float *x, float *y, char *ok) { for (long i = 0; i < n; ++i) ok[i] = log_float(x[i], y + i); }
extern "C" void f_exp(long n, const float *x, float *y, char *ok) { for (long i = 0; i < n; ++i) ok[i] = exp_float(x[i], y + i); }
extern "C" void f_sin(long n, const float *x, float *y, char *ok) { float c; for (long i = 0; i < n; ++i) ok[i] = sincos_float(x[i], y + i, &c); }
extern "C" void f_cos(long n, const float *x, float *y, char *ok) { float s; for (long i = 0; i < n; ++i) ok[i] = sincos_float(x[i], &s, y + i); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("crmathf")
    src, so = str(d / "f.cpp"), str(d / "libf.so")
    with open(src, "w") as f:
        f.write(SRC)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, src,
                        "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[:500]
    return ctypes.CDLL(so)


def args(name):
    rng = np.random.default_rng(3)
    u = (rng.integers(0, 2**32, 400000).astype(np.float64) + 0.5) * 2.0**-32
    near1 = (1.0 + np.arange(-40000, 40000) * 2.0**-24).astype(np.float32)
    if name == "log":
        bits = rng.integers(0x00800000, 0x7F800000, 400000, dtype=np.uint32)
        return np.concatenate([u.astype(np.float32), near1, bits.view(np.float32),
                               np.float32([2.0**-24, 2.0**-126, 1.0, 3.4e38])])
    if name == "exp":
        return np.concatenate([rng.uniform(-86.9, 86.9, 400000), -rng.exponential(1, 200000),
                               rng.uniform(-1e-3, 1e-3, 100000), [0.0, 1e-30]]).astype(np.float32)
    grid = (np.arange(-9, 10)[:, None] * (np.pi / 4) + np.arange(-300, 300) * 2.0**-22).ravel()
    return np.concatenate([2 * np.pi * u, rng.uniform(-16, 16, 300000), grid[np.abs(grid) > 1e-12],
                           rng.uniform(1e-9, 1e-3, 50000)]).astype(np.float32)


@pytest.mark.parametrize("name", ["log", "exp", "sin", "cos"])
def test_float_functions(lib, name):
    x = np.ascontiguousarray(args(name))
    y, ok = np.zeros_like(x), np.zeros(len(x), dtype=np.int8)
    p = ctypes.c_void_p
    getattr(lib, "f_" + name)(ctypes.c_long(len(x)), x.ctypes.data_as(p), y.ctypes.data_as(p), ok.ctypes.data_as(p))
    want = getattr(np, name)(x.astype(np.float64)).astype(np.float32)
    t = ok != 0
    assert t.mean() > 0.9999, t.mean()
    assert np.array_equal(y[t].view(np.uint32), want[t].view(np.uint32))


def test_float_functions_leave_special_arguments(lib):
    bad = {"log": [0.0, -0.0, -1.0, np.inf, -np.inf, np.nan, 1e-39], "exp": [87.0, -87.0, np.inf, -np.inf, np.nan],
           "sin": [0.0, -0.0, 16.0, -16.0, np.inf, np.nan, 1e-30], "cos": [0.0, -0.0, 16.0, np.inf, np.nan]}
    p = ctypes.c_void_p
    for name, v in bad.items():
        x = np.array(v, dtype=np.float32)
        y, ok = np.zeros_like(x), np.ones(len(x), dtype=np.int8)
        getattr(lib, "f_" + name)(ctypes.c_long(len(x)), x.ctypes.data_as(p), y.ctypes.data_as(p),
                                  ok.ctypes.data_as(p))
        assert not ok.any(), (name, ok)
