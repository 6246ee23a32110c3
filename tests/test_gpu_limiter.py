"""A NaN among the slopes goes the way of the reference's comparisons (run on
a B200): bad values next to a column's ends set the status the oracle sets, in
both solvers and every shape of the limiter's callers."""
import numpy as np
import pytest

from gitm_b200 import abi, synthetic
from tests.test_gpu_parity import gpu_advance, ref_advance

pytestmark = pytest.mark.gpu

# (field, value, cell index) planted in a column each
LOWER = [("ndensity_s", np.nan, 0), ("ndensity_s", np.inf, 0), ("ndensity_s", -np.inf, 0), ("ndensity_s", 0.0, 1),
         ("temperature", 0.0, 1), ("temperature", 1e-300, 1)]
UPPER = [("ndensity_s", np.nan, 52), ("ndensity_s", np.nan, 53)]


@pytest.mark.parametrize("solver,threads,plant", [
    (abi.SOLVER_RUSANOV, 512, LOWER), (abi.SOLVER_RUSANOV, 256, LOWER), (abi.SOLVER_RUSANOV, 128, LOWER),
    (abi.SOLVER_AUSM, 384, UPPER), (abi.SOLVER_AUSM, 256, UPPER)])
def test_status_of_bad_ends(oracle_lib, solver, threads, plant):
    p = abi.default_params(solver=solver)
    m = synthetic.make_member(3 * len(plant), 50, seed=3)
    for c, (field, value, g) in enumerate(plant):
        getattr(m, field)[0, g, 3 * c] = value
    _, want = ref_advance(oracle_lib, m, p, 2.0)
    _, got = gpu_advance(m, p, 2.0, config=dict(threads=threads))
    np.testing.assert_array_equal(got, want)
    assert (want[::3] != 0).all() and (want[1::3] == 0).all() and (want[2::3] == 0).all()
