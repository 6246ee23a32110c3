"""The FP64 exp, log and reciprocal of csrc/vert_math.cuh, compiled as plain
C++: their error against long double over the arguments the stages meet and
the whole range, and the values at the ends."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include "vert_math.cuh"
extern "C" void rcp(const double* x, double* y, long n) { for (long i = 0; i < n; ++i) y[i] = gv::rcp_nr(x[i]); }
#include <cmath>
// results, and the error in units of the last place against long double
extern "C" void elog(const double* x, double* y, double* u, long n) {
  for (long i = 0; i < n; ++i) {
    double a[3] = {x[i], 2.0, x[i]}, b[3];
    gv::log_n(a, b);
    y[i] = b[0];
    const long double w = logl((long double)x[i]);
    u[i] = (b[0] == b[2]) ? (double)(fabsl(b[0] - w) / (std::nextafter(std::fabs((double)w), INFINITY) - std::fabs((double)w))) : 99;
  }
}
extern "C" void eexp(const double* x, double* y, double* u, long n) {
  for (long i = 0; i < n; ++i) {
    double a[3] = {x[i], 0.5, x[i]}, b[3];
    gv::exp_n(a, b);
    y[i] = b[0];
    const long double w = expl((long double)x[i]);
    u[i] = (b[0] == b[2]) ? (double)(fabsl(b[0] - w) / (std::nextafter((double)w, INFINITY) - (double)w)) : 99;
  }
}
"""


@pytest.fixture(scope="module")
def mathlib(tmp_path_factory):
    import ctypes
    d = tmp_path_factory.mktemp("math")
    src, so = d / "m.cpp", d / "m.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-x", "c++",
                    "-I" + os.path.join(ROOT, "gitm_b200", "csrc"), str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


def _apply(f, x):
    import ctypes
    x = np.ascontiguousarray(x, dtype=np.float64)
    y = np.empty_like(x)
    f(x.ctypes.data_as(ctypes.c_void_p), y.ctypes.data_as(ctypes.c_void_p), ctypes.c_long(x.size))
    return y


@pytest.mark.parametrize("lo,hi", [(-1020, -900), (-130, 130), (0, 1), (900, 1020)])
def test_rcp_nr(mathlib, lo, hi):
    rng = np.random.default_rng(abs(lo) + hi)
    x = np.ldexp(rng.uniform(1.0, 2.0, 20000), rng.integers(lo, hi, 20000)) * rng.choice([-1.0, 1.0], 20000)
    x[:2] = np.ldexp(1.0, [lo, hi])
    y = _apply(mathlib.rcp, x)
    want = 1.0 / x
    # two Newton-Raphson steps leave the rounding of the last one: within one unit in the last place
    assert (np.abs(y - want) <= np.spacing(np.abs(want))).all()


@pytest.mark.parametrize("x", [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324])
def test_rcp_nr_outside_its_range_is_not_finite(mathlib, x):
    assert not np.isfinite(_apply(mathlib.rcp, [x]))[0]


def _apply2(f, x):
    import ctypes
    x = np.ascontiguousarray(x, dtype=np.float64)
    y, u = np.empty_like(x), np.empty_like(x)
    f(*[a.ctypes.data_as(ctypes.c_void_p) for a in (x, y, u)], ctypes.c_long(x.size))
    return y, u


@pytest.mark.parametrize("lo,hi", [(-1.0, 1.0), (-45.0, 45.0), (-707.9, 707.9)])
def test_exp_n(mathlib, lo, hi):
    _, ulp = _apply2(mathlib.eexp, np.random.default_rng(1).uniform(lo, hi, 200000))
    assert ulp.max() <= 1.0  # CUDA's bound for its own exp


@pytest.mark.parametrize("lo,hi", [(-0.7, 0.7), (3.0, 9.0), (-60.0, 60.0), (-708.0, 709.0)])
def test_log_n(mathlib, lo, hi):
    _, ulp = _apply2(mathlib.elog, np.exp(np.random.default_rng(2).uniform(lo, hi, 200000)))
    assert ulp.max() <= 1.0  # CUDA's bound for its own log


def test_ends(mathlib):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 709.7, 709.8, -745.1, -746.0, 1e308, -1e308, 708.0, -708.0])
    with np.errstate(all="ignore"):
        np.testing.assert_allclose(_apply2(mathlib.eexp, x)[0], np.exp(x), rtol=3e-16, atol=5e-324)
        x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, -1.0, 5e-324, 1e-310, 2.3e-308, 1.7e308, 1.0])
        np.testing.assert_allclose(_apply2(mathlib.elog, x)[0], np.log(x), rtol=3e-16)
