"""Lanes of a warp that part ways ahead of its tensor-memory accesses (run on
a B200): a column whose values leave the ranges of the batched exponentials
and logarithms, damping's own exponential and division, eddy diffusion in some
cells of a warp only, columns that the adjoint skips.  The columns beside the
odd one have the bits they have without it."""
import numpy as np
import pytest
import torch

from gitm_b200 import abi, synthetic
from tests.test_gpu_adjoint import _gpu_vjp, _ybar
from tests.test_gpu_parity import STATE, gpu_advance

pytestmark = pytest.mark.gpu

N_COLS, N_ALTS = 13, 50
ODD = {
    "nan_temperature": lambda m, c: m.temperature.__setitem__((0, 26, c), np.nan),
    "negative_temperature": lambda m, c: m.temperature.__setitem__((0, 31, c), -1.0),
    "inf_wind": lambda m, c: m.vert_vel.__setitem__((1, 12, c), np.inf),
    "huge_density": lambda m, c: m.ndensity_s.__setitem__((2, 40, c), 1e306),
    "zero_density": lambda m, c: m.ndensity_s.__setitem__((5, 9, c), 0.0),
}


@pytest.mark.parametrize("solver,threads,over", [
    (abi.SOLVER_AUSM, 384, {}), (abi.SOLVER_AUSM, 384, dict(use_neutral_friction=0)),
    (abi.SOLVER_RUSANOV, 512, {}), (abi.SOLVER_RUSANOV, 512, dict(use_damping=1))],
    ids=["ausm", "ausm_no_friction", "rusanov", "rusanov_damping"])
@pytest.mark.parametrize("odd", list(ODD))
@pytest.mark.parametrize("bad", [4, 12])
def test_step(solver, threads, over, odd, bad):
    p = abi.default_params(solver=solver, **over)
    m = synthetic.make_member(N_COLS, N_ALTS, seed=91)
    assert 0 < (m.eddy > 0.0).sum() < m.eddy.size
    cfg = dict(threads=threads, steps_per_launch=2)
    want, st = gpu_advance(m, p, 2.0, 2, config=cfg)
    assert (st == 0).all()
    ODD[odd](m, bad)
    out, st = gpu_advance(m, p, 2.0, 2, config=cfg)
    keep = np.arange(N_COLS) != bad
    assert st[bad] != 0 and (st[keep] == 0).all()
    for k in STATE:
        np.testing.assert_array_equal(out[k][..., keep], want[k][..., keep], err_msg=k)


@pytest.mark.parametrize("odd", list(ODD))
@pytest.mark.parametrize("n_alts,bad", [(50, 4), (50, 12), (30, 5)])
def test_adjoint(odd, n_alts, bad):
    p = abi.default_params()
    m = synthetic.make_member(N_COLS, n_alts, seed=92, with_heating=True)
    y = _ybar(m, torch.Generator().manual_seed(3), torch.device("cuda"))
    want, st = _gpu_vjp(m, p, 2.0, y)
    assert st == (0, 0)
    m2 = m.copy()
    if n_alts < 50:
        m2.temperature[0, 12, bad] = np.nan
    else:
        ODD[odd](m2, bad)
    got, _ = _gpu_vjp(m2, p, 2.0, y)
    keep = torch.arange(N_COLS) != bad
    for k, w in want.items():
        assert torch.equal(got[k].cpu()[..., keep], w.cpu()[..., keep]), k
