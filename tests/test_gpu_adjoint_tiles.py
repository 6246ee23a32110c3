"""The adjoint kernel where its tiles have their edges: 4, 3, 2 and 1 columns
per CTA at the altitude counts on both sides of each change, a last tile with
fewer columns (one half of a warp idle in the boundary tasks), the ends of a
column in one task (9) and in two (10), against autograd at the tolerance of
test_gpu_adjoint.py."""
import pytest
import torch

from gitm_b200 import abi, synthetic
from tests.test_gpu_adjoint import _gpu_vjp, _rel, _torch_vjp, _ybar

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_alts,n_cols", [(9, 7), (10, 5), (32, 7), (33, 7), (42, 5), (43, 5), (50, 1), (64, 3),
                                           (65, 3), (127, 2)])
def test_adjoint_tile_edges(n_alts, n_cols):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = abi.default_params()
    m = synthetic.make_member(n_cols, n_alts, seed=300 + n_alts)
    y = _ybar(m, torch.Generator().manual_seed(n_alts), torch.device("cuda"))
    want = _torch_vjp(m, p, 2.0, y, torch.device("cuda"))
    got, status = _gpu_vjp(m, p, 2.0, y)
    assert status == (0, 0)
    for k, w in want.items():
        g = got[k]
        if k == "idensity_s":
            g, w = g[:9], w[:9]
        assert _rel(g, w) < 1e-9, (k, _rel(g, w))
