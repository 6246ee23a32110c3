"""What one call has answered with an error, or found not finished, does not
come back as the error of the next (run on a B200)."""
import ctypes as C

import numpy as np
import pytest

from gitm_b200 import abi, synthetic
from gitm_b200 import vertical as V
from gitm_b200._lib import lib
from tests.test_gpu_fortran import fortran_arrays
from tests.test_gpu_parity import STATE, gpu_advance
from tests.test_gpu_refused import N, N_ALTS, fortran_call

pytestmark = pytest.mark.gpu


def refused_allocation(ctx, dm):
    """A plan of more columns than there is memory for status words."""
    b = dm.batch()
    b.n_cols = 1 << 38
    h = C.c_void_p()
    assert lib().gitm_vert_plan_create(ctx.handle, (abi.GitmColumnBatch * 1)(b), 1, C.byref(h)) == abi.ERR_CUDA


def unfinished_wait(ctx, dm):
    """A wait that gives up: 32 resident steps of 20,000 columns just issued."""
    import torch
    long = V.device_member(synthetic.make_member(20000, 50, seed=4))
    plan = V.Plan(ctx, [long])
    plan.set_config(threads=512, steps_per_launch=32)
    torch.cuda.synchronize()
    plan.advance(2.0, 32)
    assert plan.wait(0.0) is False
    unfinished_wait.plan = plan  # still running


@pytest.mark.parametrize("first", [refused_allocation, unfinished_wait])
@pytest.mark.parametrize("then", ["plan", "fortran", "cfl"])
def test_next_call(first, then):
    p = abi.default_params(compute_coefficients=0)
    m = synthetic.make_member(N, N_ALTS, seed=3)
    ctx = V.VerticalContext(p)
    dm = V.device_member(m)
    first(ctx, dm)
    if then == "plan":
        V.advance_vertical_all(ctx, [dm], 2.0)
        want, _ = gpu_advance(m, p, 2.0)
        for k in STATE:
            np.testing.assert_array_equal(dm.to_numpy()[k], want[k], err_msg=k)
    elif then == "fortran":
        rc, _ = fortran_call(ctx, fortran_arrays(m, 1), 1)
        assert rc == abi.OK, ctx.last_error()
    else:
        assert 0.0 < V.calc_timestep_vertical(ctx, [dm]) < 1e30
    ctx.close()
