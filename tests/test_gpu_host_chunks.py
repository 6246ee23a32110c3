"""The host-pointer call over few and many chunks of columns and several
members (run on a B200): bit for bit the device form with the launch shape the
host form uses, whichever way the chunks' copies follow one another."""
import numpy as np
import pytest

from gitm_b200 import abi, synthetic
from gitm_b200 import vertical as V
from tests.test_gpu_parity import STATE, gpu_advance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [((900, 30),), ((3072, 30),), ((3073, 30),), ((4200, 50),), ((1500, 30), (1100, 50)),
                                   ((20, 8), (1030, 64), (2500, 30)), ((17000, 20),)], ids=str)
def test_chunks(shape):
    p = abi.default_params()
    ms = [synthetic.make_member(n, a, seed=40 + i) for i, (n, a) in enumerate(shape)]
    want = [gpu_advance(m, p, 2.0, config=dict(threads=128, steps_per_launch=1))[0] for m in ms]
    ctx = V.VerticalContext(p)
    for _ in range(2):  # the plan of the first call serves the second
        hs = [m.copy() for m in ms]
        for h in hs:
            h.log_ns, h.ndensity = np.zeros_like(h.ndensity_s), np.zeros_like(h.rho)
        V.advance_vertical_all_host(ctx, hs, 2.0)
        for h, w in zip(hs, want):
            for k in STATE:
                np.testing.assert_array_equal(getattr(h, k), w[k], err_msg=k)
    ctx.close()


@pytest.mark.parametrize("n", [32768, 32784])  # chunks of 2,048 and 2,049 columns: either order of the copies
def test_long_rows(n):
    p = abi.default_params()
    m = synthetic.make_member(n, 8, seed=47)
    want = gpu_advance(m, p, 2.0, config=dict(threads=128, steps_per_launch=1))[0]
    ctx = V.VerticalContext(p)
    h = m.copy()
    V.advance_vertical_all_host(ctx, [h], 2.0)
    for k in STATE:
        np.testing.assert_array_equal(getattr(h, k), want[k], err_msg=k)
    ctx.close()
