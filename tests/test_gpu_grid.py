"""The grid-coefficient kernel (csrc/vert_grid.cu): an altitude grid per
column with the same altitudes gives the bits of the shared grid, from host
and from device memory, and columns with grids of their own match the oracle
(which forms the coefficients in the reference's order)."""
import numpy as np
import pytest

from gitm_b200 import abi, synthetic
from tests.parity import assert_state_close
from tests.test_gpu_parity import STATE, gpu_advance, ref_advance

pytestmark = pytest.mark.gpu
GRID = ("altitude", "gravity", "dalt_c", "inv_r")


@pytest.mark.parametrize("solver", [abi.SOLVER_RUSANOV, abi.SOLVER_AUSM])
@pytest.mark.parametrize("n_alts,n_cols", [(8, 1), (50, 3), (50, 129), (100, 5)])
def test_grid_per_column(oracle_lib, n_alts, n_cols, solver):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gitm_b200 import vertical as V
    p = abi.default_params(solver=solver)
    m = synthetic.make_member(n_cols, n_alts, seed=90 + n_alts)
    shared, _ = gpu_advance(m, p, 2.0, config=dict(threads=128))
    c = m.copy()
    for k in GRID:
        setattr(c, k, np.ascontiguousarray(np.repeat(getattr(m, k)[:, None], n_cols, axis=1)))
    own, _ = gpu_advance(c, p, 2.0, config=dict(threads=128))
    h = c.copy()
    ctx = V.VerticalContext(p)
    V.advance_vertical_all_host(ctx, [h], 2.0)
    ctx.close()
    for k in STATE:
        np.testing.assert_array_equal(own[k], shared[k], err_msg=k)
        np.testing.assert_array_equal(getattr(h, k), shared[k], err_msg=k)
    # a grid of its own for every column
    for j in range(n_cols):
        alt = m.altitude * (1.0 + 1.0e-3 * j / n_cols)
        c.altitude[:, j] = alt
        for k, v in zip(("dalt_c", "inv_r", "gravity"), synthetic.grid_geometry(alt)):
            getattr(c, k)[:, j] = v
    ref, st_ref = ref_advance(oracle_lib, c, p, 2.0)
    out, st = gpu_advance(c, p, 2.0, config=dict(threads=128))
    np.testing.assert_array_equal(st, st_ref)
    assert_state_close(out, ref, STATE)
