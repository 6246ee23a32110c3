"""gitm_hz_advance at the block shapes where its kernel's threads, lines and
shared-memory plan have their edges (one cell, one line, thin blocks whose
slopes go in batches and whose Orig stays in registers, the largest blocks of
each thread count), against the CPU oracle at the tolerance of
test_gpu_horizontal.py."""
import pytest

from gitm_b200 import abi
from gitm_b200 import horizontal as H
from tests.test_gpu_horizontal import _compare, _ref, _run, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_lons,n_lats", [(1, 1), (1, 9), (9, 1), (2, 2), (8, 12), (12, 8), (97, 1), (13, 13), (16, 12),
                                           (12, 16), (16, 16), (2, 128), (128, 2), (1, 150)])
def test_block_shapes(ctx, oracle_lib, n_lons, n_lats):  # noqa: F811
    p = abi.default_hz_params()
    blocks = H.synthetic_blocks(n_lons, n_lats, 8, 2, 1, seed=n_lons + 300 * n_lats)
    _compare(_run(ctx, blocks, p, dt=0.05), _ref(oracle_lib, blocks, p, dt=0.05))
