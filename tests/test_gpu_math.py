"""The FP64 exp, log and reciprocal of csrc/vert_math.cuh as the device runs
them (run on a B200): the batches by lane and by warp, compiled here into a
kernel of their own, against 80-bit results over the arguments the stages meet,
the whole range and the values at its ends.  Each has to be within one unit in
the last place, the bound of CUDA's own functions."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from gitm_b200 import build

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include "vert_math.cuh"
// one argument a thread, n a multiple of 32; a batch holds the thread's argument and ordinary ones beside it
template <int WHAT>
__global__ void run(const double* x, double* y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double v = x[i];
  if (WHAT == 4) {
    y[i] = gv::rcp_nr(v);
  } else {
    const double a[3] = {v, 0.5, v};
    double b[3];
    if (WHAT == 0) gv::exp_n(a, b);
    if (WHAT == 1) gv::exp_n<3, true>(a, b);
    if (WHAT == 2) gv::log_n(a, b);
    if (WHAT == 3) gv::log_n<3, true>(a, b);
    y[i] = (__double_as_longlong(b[0]) == __double_as_longlong(b[2])) ? b[0] : __longlong_as_double(0x7ff8dead00000000ll);
  }
}
extern "C" int device_run(int what, const double* x, double* y, int n) {
  double *dx = nullptr, *dy = nullptr;
  cudaMalloc(&dx, n * sizeof(double));
  cudaMalloc(&dy, n * sizeof(double));
  cudaMemcpy(dx, x, n * sizeof(double), cudaMemcpyHostToDevice);
  const int grid = (n + 127) / 128;
  if (what == 0) run<0><<<grid, 128>>>(dx, dy, n);
  if (what == 1) run<1><<<grid, 128>>>(dx, dy, n);
  if (what == 2) run<2><<<grid, 128>>>(dx, dy, n);
  if (what == 3) run<3><<<grid, 128>>>(dx, dy, n);
  if (what == 4) run<4><<<grid, 128>>>(dx, dy, n);
  const int e = int(cudaMemcpy(y, dy, n * sizeof(double), cudaMemcpyDeviceToHost));
  cudaFree(dx);
  cudaFree(dy);
  return e;
}
"""
EXP, EXP_WARP, LOG, LOG_WARP, RCP = range(5)


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    d = tmp_path_factory.mktemp("math")
    src, so = d / "m.cu", d / "m.so"
    src.write_text(SOURCE)
    flags = [f for f in build.NVCC_FLAGS if f != "-lineinfo"]
    subprocess.run([build.nvcc(), *flags, "-shared", "-I" + os.path.join(ROOT, "gitm_b200", "csrc"), str(src), "-o", str(so)],
                   check=True)
    lib = ctypes.CDLL(str(so))

    def run(what, x):
        x = np.ascontiguousarray(np.resize(x, (len(x) + 31) // 32 * 32), dtype=np.float64)
        y = np.empty_like(x)
        p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        assert lib.device_run(what, p(x), p(y), x.size) == 0
        return x, y

    return run


def _ulp(y, want):
    w = np.abs(want.astype(np.float64))
    return np.abs(y.astype(np.longdouble) - want) / np.spacing(w).astype(np.longdouble)


@pytest.mark.parametrize("what", [EXP, EXP_WARP])
@pytest.mark.parametrize("lo,hi", [(-1.0, 1.0), (-45.0, 45.0), (-707.9, 707.9), (-708.3, 709.7)])
def test_exp(device, what, lo, hi):
    x, y = device(what, np.random.default_rng(1).uniform(lo, hi, 200000))
    assert _ulp(y, np.exp(x.astype(np.longdouble))).max() <= 1.0


@pytest.mark.parametrize("what", [LOG, LOG_WARP])
@pytest.mark.parametrize("lo,hi", [(-0.7, 0.7), (3.0, 9.0), (-60.0, 60.0), (-708.0, 709.0)])
def test_log(device, what, lo, hi):
    x, y = device(what, np.exp(np.random.default_rng(2).uniform(lo, hi, 200000)))
    assert _ulp(y, np.log(x.astype(np.longdouble))).max() <= 1.0


@pytest.mark.parametrize("lo,hi", [(-1020, -900), (-130, 130), (0, 1), (900, 1020)])
def test_rcp(device, lo, hi):
    rng = np.random.default_rng(abs(lo) + hi)
    v = np.ldexp(rng.uniform(1.0, 2.0, 200000), rng.integers(lo, hi, 200000)) * rng.choice([-1.0, 1.0], 200000)
    x, y = device(RCP, v)
    assert _ulp(y, 1 / x.astype(np.longdouble)).max() <= 1.0


def test_ends(device):
    with np.errstate(all="ignore"):
        v = [0.0, -0.0, np.inf, -np.inf, np.nan, 709.7, 709.8, -745.1, -746.0, 1e308, -1e308, 708.0, -708.0]
        for what in (EXP, EXP_WARP):
            x, y = device(what, np.array(v))
            np.testing.assert_allclose(y, np.exp(x), rtol=3e-16, atol=5e-324)
        v = [0.0, -0.0, np.inf, -np.inf, np.nan, -1.0, 5e-324, 1e-310, 2.3e-308, 1.7e308, 1.0]
        for what in (LOG, LOG_WARP):
            x, y = device(what, np.array(v))
            np.testing.assert_allclose(y, np.log(x), rtol=3e-16)
    x, y = device(RCP, np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324]))
    assert not np.isfinite(y).any()
