"""The limiter of csrc/vert_math.cuh, compiled as plain C++, against the
branches of the reference (ModLimiter.f90:16-36): every pair of zeros,
subnormals, ordinary and extreme values, infinities and NaN of either sign, and
random pairs, bit for bit (of a zero, the value)."""
import ctypes
import itertools
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include "vert_math.cuh"
extern "C" void both(const double* u, const double* d, double beta, double* got, double* want, long n) {
  for (long i = 0; i < n; ++i) {
    got[i] = gv::limiter_mc(u[i], d[i], beta);
    const double a = beta * u[i], b = beta * d[i], c = (u[i] + d[i]) * 0.5;
    want[i] = 0.0;
    if (u[i] > 0.0) {
      if (d[i] > 0.0) want[i] = std::fmin(std::fmin(a, b), c);
    } else if (d[i] < 0.0) {
      want[i] = std::fmax(std::fmax(a, b), c);  // a NaN among the three is passed over
    }
  }
}
"""


@pytest.fixture(scope="module")
def both(tmp_path_factory):
    d = tmp_path_factory.mktemp("limiter")
    src, so = d / "l.cpp", d / "l.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "gitm_b200", "csrc"), "-x", "c++", str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so)).both


@pytest.mark.parametrize("beta", [1.0, 1.3, 1.5, 2.0])
def test_limiter(both, beta):
    v = [0.0, 5e-324, 1e-310, 2.3e-308, 1e-200, 1e-3, 1.0, 1.0 + 2 ** -52, 1.5, 2.0, 7.0, 1e200, 8.9e307, 1.7e308, np.inf, np.nan]
    v = np.array(v + [-x for x in v])
    pairs = np.array(list(itertools.product(v, v)))
    rng = np.random.default_rng(1)
    r = rng.normal(size=(20000, 2)) * 10.0 ** rng.uniform(-6, 6, (20000, 1))
    r[::3, 1] = r[::3, 0] * rng.uniform(0.3, 3.0, r[::3].shape[0])
    x = np.concatenate([pairs, r])
    u, d = np.ascontiguousarray(x[:, 0]), np.ascontiguousarray(x[:, 1])
    got, want = np.empty_like(u), np.empty_like(u)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    both(p(u), p(d), ctypes.c_double(beta), p(got), p(want), ctypes.c_long(u.size))
    np.testing.assert_array_equal(got, want)
