"""A species of extreme density in one cell (run on a B200): 1e170 to 1e300,
where the symmetric friction matrix's products of two densities are no numbers
any more.  The AUSM solver takes it as the reference does, against the oracle
(the reference's Rusanov solver does not)."""
import numpy as np
import pytest

from gitm_b200 import abi, synthetic
from tests.parity import assert_state_close
from tests.test_gpu_parity import STATE, gpu_advance, ref_advance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [384, 256, 128])
@pytest.mark.parametrize("friction", [1, 0], ids=["friction", "no_friction"])
@pytest.mark.parametrize("density", [1e150, 1e170, 1e230, 1e300], ids=str)
def test_ausm(oracle_lib, density, friction, threads):
    p = abi.default_params(solver=abi.SOLVER_AUSM, use_neutral_friction=friction)
    m = synthetic.make_member(24, 50, seed=3)
    cells = (25, 50, 51)
    for c, g in enumerate(cells):
        m.ndensity_s[0, g, 8 * c] = density
    ref, st_ref = ref_advance(oracle_lib, m, p, 2.0)
    assert (st_ref == 0).all() and all(np.isfinite(ref[k]).all() for k in STATE)
    out, st = gpu_advance(m, p, 2.0, config=dict(threads=threads))
    np.testing.assert_array_equal(st, st_ref)
    assert_state_close(out, ref, STATE)
