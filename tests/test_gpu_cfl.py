"""gitm_vert_cfl_dt where its kernel's blocks of 32 columns and its rows of
every 8th altitude have their edges: column counts about 32, few and many
altitudes, and the fastest cell of the batch in each part of a column, against
the CPU oracle at the tolerance of test_gpu_parity.py."""
import pytest

from gitm_b200 import abi, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cols,n_alts,col,alt", [(1, 20, 0, 1), (31, 20, 30, 20), (32, 50, 31, 7), (33, 50, 32, 8),
                                                   (65, 64, 40, 9), (300, 100, 299, 100), (64, 50, 5, 0),
                                                   (64, 50, 5, 51)])
def test_cfl_fastest_cell(oracle_lib, n_cols, n_alts, col, alt):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gitm_b200 import vertical as V
    p = abi.default_params()
    m = synthetic.make_member(n_cols, n_alts, seed=n_cols + n_alts)
    m.vert_vel[n_alts % 6, alt + 1, col] = -9.0e3  # cell alt; 0 and nAlts + 1 do not count
    want = oracle_lib.cfl_dt(m, p, 0.75)
    ctx = V.VerticalContext(p)
    got = V.calc_timestep_vertical(ctx, [V.device_member(m)], cfl=0.75)
    ctx.close()
    assert got == pytest.approx(want, rel=1e-14)
