"""The 512-thread shape (csrc/vert_tile.cuh) against the CPU oracle at the
sizes where its task lists, runs and lane groups have their edges, and on the
branches it splits over lanes.

Tolerances: tests/parity.py's 1e-10 for one step; 1e-9 over resident steps,
which keep LogNS where separate steps take log(exp(.)).
"""
import numpy as np
import pytest

from gitm_b200 import abi, synthetic
from tests.parity import assert_state_close
from tests.test_gpu_parity import STATE, gpu_advance, ref_advance

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


# nAlts: the smallest and largest, odd and even, one and several slope runs; columns: 1, tiles with remainders of
# the lane groups (2 and 3 columns), the full tile and one column more
@pytest.mark.parametrize("n_alts,n_cols", [(8, 64), (8, 65), (9, 1), (21, 25), (37, 14), (50, 1), (50, 2), (50, 10),
                                           (50, 11), (50, 23), (64, 8), (75, 7), (100, 5), (127, 4), (128, 9)])
@pytest.mark.parametrize("steps", [1, 3])
def test_sizes(oracle_lib, n_alts, n_cols, steps):
    p = abi.default_params()
    m = synthetic.make_member(n_cols, n_alts, seed=200 + n_alts + n_cols, with_heating=True)
    ref, st_ref = ref_advance(oracle_lib, m, p, 2.0, steps)
    out, st = gpu_advance(m, p, 2.0, steps, config=dict(threads=512, steps_per_launch=steps))
    np.testing.assert_array_equal(st, st_ref)
    assert_state_close(out, ref, STATE, rtol=1e-10 if steps == 1 else 1e-9)


VARIANTS = {
    "log_ions": dict(use_improved_ion_advection=0),
    "no_ion_advection": dict(use_ion_advection=0),
    "msis_damping": dict(use_msis_bcs=1, use_damping=1),
    "no_friction": dict(use_neutral_friction=0),
    "given_coefficients": dict(compute_coefficients=0),
    "eddy": dict(compute_eddy=1),
    "low_clamp": dict(max_vertical_velocity=1.0, beta_limiter=1.3),
}


@pytest.mark.parametrize("name", sorted(VARIANTS))
def test_variants(oracle_lib, name):
    p = abi.default_params(**VARIANTS[name])
    steps = 1 if name == "given_coefficients" else 2
    m = synthetic.make_member(23, 50, seed=31, with_lbc=True)
    ref, st_ref = ref_advance(oracle_lib, m, p, 2.0, steps)
    out, st = gpu_advance(m, p, 2.0, steps, config=dict(threads=512, steps_per_launch=steps))
    np.testing.assert_array_equal(st, st_ref)
    names = STATE + (("eddy",) if name == "eddy" else ()) + synthetic.Member.COEFFS
    assert_state_close(out, ref, names, rtol=1e-10 if steps == 1 else 1e-9)


@pytest.mark.parametrize("cells,ion", [((48,), 0), ((46,), 1), ((47, 48), 5), ((45, 46), 0)])
def test_negative_ions_near_the_top(oracle_lib, cells, ion):
    """The repair of set_vertical_bcs.Earth.f90:608-649 changes cells whose slopes other tasks have taken."""
    p = abi.default_params()
    m = synthetic.make_member(13, 50, seed=72)
    for i in cells:
        m.idensity_s[ion, i + 1, 7] = -5.0
    ref, st_ref = ref_advance(oracle_lib, m, p, 2.0)
    out, st = gpu_advance(m, p, 2.0, config=dict(threads=512))
    np.testing.assert_array_equal(st, st_ref)
    keep = np.arange(13) != 7 if st_ref[7] else slice(None)
    assert_state_close({k: out[k][..., keep] for k in STATE}, {k: ref[k][..., keep] for k in STATE}, STATE)


@pytest.mark.parametrize("plant,bit", [("temperature", abi.ST_LU_SINGULAR | abi.ST_NONFINITE),
                                       ("ndensity_s", abi.ST_NEG_DENSITY)])
def test_bad_column_stays_alone(oracle_lib, plant, bit):
    p = abi.default_params()
    m = synthetic.make_member(13, 50, seed=73)
    getattr(m, plant)[0, 26, 4] = np.nan if plant == "temperature" else 0.0
    ref, st_ref = ref_advance(oracle_lib, m, p, 2.0)
    out, st = gpu_advance(m, p, 2.0, config=dict(threads=512))
    # a column with a density <= 0 is not stored; its stages still run and may set other bits
    assert st[4] & bit == bit and st_ref[4] & bit == bit and (np.delete(st, 4) == 0).all()
    if plant == "temperature":
        assert st[4] == st_ref[4]
    keep = np.arange(13) != 4
    assert_state_close({k: out[k][..., keep] for k in STATE}, {k: ref[k][..., keep] for k in STATE}, STATE)
