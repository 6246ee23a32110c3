"""The FP64 helpers of csrc/vert_math.cuh, compiled as plain C++: their error
against the correctly rounded value over the exponents the stages meet and
the ends of the stated range."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include "vert_math.cuh"
extern "C" void rcp(const double* x, double* y, long n) { for (long i = 0; i < n; ++i) y[i] = gv::rcp_nr(x[i]); }
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
