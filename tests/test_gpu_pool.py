"""Plans take their device memory from their context's pool: a plan that is
destroyed while its launches run, on another stream, gives nothing back that
they still use, and plans of other sizes, solvers and threads that follow get
the results of fresh ones."""
import threading

import numpy as np
import pytest

from gitm_b200 import abi, synthetic
from tests.test_gpu_parity import STATE, gpu_advance

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def test_destroyed_in_flight(torch_cuda):
    from gitm_b200 import vertical as V
    p = abi.default_params()
    long, short = synthetic.make_member(6000, 50, seed=1), synthetic.make_member(500, 30, seed=2)
    want_long, _ = gpu_advance(long, p, 2.0, 8, config=dict(threads=512, steps_per_launch=4))
    want_short, _ = gpu_advance(short, p, 2.0, 1)
    ctx = V.VerticalContext(p)
    side = torch_cuda.cuda.Stream()
    for _ in range(3):
        a, b = V.device_member(long), V.device_member(short)
        torch_cuda.cuda.synchronize()
        plan = V.Plan(ctx, [a])
        plan.set_config(threads=512, steps_per_launch=4)
        plan.advance(2.0, 8, stream=side)
        plan.close()  # while the launches run
        V.advance_vertical_all(ctx, [b], 2.0)
        torch_cuda.cuda.synchronize()
        for k in STATE:
            np.testing.assert_array_equal(a.to_numpy()[k], want_long[k], err_msg=k)
            np.testing.assert_array_equal(b.to_numpy()[k], want_short[k], err_msg=k)
    # a plan may outlive its context
    plan = V.Plan(ctx, [V.device_member(short)])
    ctx.close()
    plan.close()


def test_threads(torch_cuda):
    from gitm_b200 import vertical as V
    p = abi.default_params()
    ms = [synthetic.make_member(n, a, seed=n) for n, a in ((300, 50), (41, 20), (1000, 64), (7, 100))]
    want = [gpu_advance(m, p, 2.0, 1)[0] for m in ms]
    errors = []

    def work(m, w):
        try:
            ctx = V.VerticalContext(p)
            for _ in range(5):
                d = V.device_member(m)
                V.advance_vertical_all(ctx, [d], 2.0)
                got = d.to_numpy()
                for k in STATE:
                    np.testing.assert_array_equal(got[k], w[k], err_msg=k)
            ctx.close()
        except Exception as e:  # reported by the main thread
            errors.append(e)

    ts = [threading.Thread(target=work, args=x) for x in zip(ms, want)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
