"""The coefficients a step writes back with compute_coefficients = 1 (run on a
B200): TempUnit is MeanMajorMass times 1 / k to the bit, as calc_rates forms it
from the mass itself, in every shape, after one step and after several."""
import numpy as np
import pytest

from gitm_b200 import abi, synthetic
from gitm_b200 import vertical as V

pytestmark = pytest.mark.gpu
KB = 1.3807e-23


@pytest.mark.parametrize("threads", [512, 256, 128])
@pytest.mark.parametrize("n_alts,steps,spl", [(50, 1, 1), (50, 3, 3), (30, 4, 2), (100, 2, 2)])
def test_mean_major_mass(threads, n_alts, steps, spl):
    m = synthetic.make_member(40, n_alts, seed=55)
    ctx = V.VerticalContext(abi.default_params())
    dm = V.device_member(m)
    for k in ("mean_major_mass", "temp_unit", "gamma"):
        dm.tensors[k].fill_(np.nan)
    plan = V.Plan(ctx, [dm])
    plan.set_config(threads=threads, steps_per_launch=spl)
    plan.advance(2.0, steps)
    plan.check()
    out = {k: dm.tensors[k].cpu().numpy() for k in ("mean_major_mass", "temp_unit", "gamma")}
    plan.close()
    ctx.close()
    assert np.isfinite(out["gamma"]).all()
    np.testing.assert_array_equal(out["temp_unit"], out["mean_major_mass"] * (1.0 / KB))
