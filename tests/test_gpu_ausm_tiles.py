"""The AUSM 384-thread shape, whose stage runs in whole warps with its values
in tensor memory, at tiles of one to six columns (the last warp with idle
lanes, warps without cells) and tiles with a remainder, against the CPU oracle
at the tolerances of test_gpu_ausm.py."""
import numpy as np
import pytest

from gitm_b200 import abi, synthetic
from tests.parity import assert_state_close
from tests.test_gpu_parity import STATE, gpu_advance, ref_advance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cols", [1, 2, 5, 6, 7, 13])
@pytest.mark.parametrize("steps", [1, 3])
def test_ausm_tile_sizes(oracle_lib, n_cols, steps):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = abi.default_params(solver=abi.SOLVER_AUSM)
    m = synthetic.make_member(n_cols, 50, seed=400 + n_cols)
    ref, st_ref = ref_advance(oracle_lib, m, p, 2.0, steps)
    out, st = gpu_advance(m, p, 2.0, steps, config=dict(threads=384, steps_per_launch=steps))
    np.testing.assert_array_equal(st, st_ref)
    assert_state_close(out, ref, STATE, rtol=1e-10 if steps == 1 else 1e-9)
