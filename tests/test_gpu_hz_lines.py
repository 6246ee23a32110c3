"""The horizontal advance on blocks with long lines, whose slopes several
threads share: lines on both sides of the length where sharing begins, last
parts of one cell and of all, in either direction, against the oracle."""
import pytest

from gitm_b200 import abi
from gitm_b200 import horizontal as H
from tests.test_gpu_horizontal import _compare, _ref, _run, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nl,nt", [(24, 3), (25, 3), (3, 24), (3, 25), (28, 8), (29, 2), (33, 7), (2, 34), (38, 1), (1, 39),
                                   (6, 42), (63, 4), (4, 64), (85, 3), (128, 2), (2, 123)])
def test_long_lines(ctx, oracle_lib, nl, nt):  # noqa: F811
    p = abi.default_hz_params()
    blocks = H.synthetic_blocks(nl, nt, 8, 2, 1, seed=nl + 300 * nt)
    _compare(_run(ctx, blocks, p, dt=0.05), _ref(oracle_lib, blocks, p, dt=0.05))
