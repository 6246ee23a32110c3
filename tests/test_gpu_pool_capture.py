"""A plan that is destroyed while a stream is being captured (run on a B200):
the device cannot be waited for then, so the plan's memory must not go to the
next plan while the launches of the first still use it."""
import numpy as np
import pytest

from gitm_b200 import abi, synthetic
from gitm_b200 import vertical as V
from tests.test_gpu_parity import STATE, gpu_advance

pytestmark = pytest.mark.gpu


def test_destroyed_during_a_capture():
    import torch
    from cuda.bindings import runtime as rt
    p = abi.default_params()
    long, short = synthetic.make_member(30000, 50, seed=1), synthetic.make_member(500, 30, seed=2)
    cfg = dict(threads=512, steps_per_launch=4)
    want_long, _ = gpu_advance(long, p, 2.0, 32, config=cfg)
    want_short, _ = gpu_advance(short, p, 2.0, 1)
    ctx = V.VerticalContext(p)
    side = torch.cuda.Stream()
    err, captured = rt.cudaStreamCreateWithFlags(rt.cudaStreamNonBlocking)
    assert err == rt.cudaError_t.cudaSuccess
    for _ in range(3):
        a = V.device_member(long)
        b = [V.device_member(short) for _ in range(4)]
        torch.cuda.synchronize()
        plan = V.Plan(ctx, [a])
        plan.set_config(**cfg)
        plan.advance(2.0, 32, stream=side)
        mode = rt.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed
        assert rt.cudaStreamBeginCapture(captured, mode)[0] == rt.cudaError_t.cudaSuccess
        plan.close()  # while its launches run
        rt.cudaStreamEndCapture(captured)  # the wait in close() has ended the capture
        rt.cudaGetLastError()
        for d in b:
            V.advance_vertical_all(ctx, [d], 2.0)
        torch.cuda.synchronize()
        for k in STATE:
            np.testing.assert_array_equal(a.to_numpy()[k], want_long[k], err_msg=k)
            for d in b:
                np.testing.assert_array_equal(d.to_numpy()[k], want_short[k], err_msg=k)
    ctx.close()
    rt.cudaStreamDestroy(captured)


def test_one_context_in_several_threads():
    """Plans of one context created, run and destroyed by several threads."""
    import threading

    import torch
    p = abi.default_params()
    ms = [synthetic.make_member(n, a, seed=n) for n, a in ((300, 50), (41, 20), (1000, 64), (7, 100))]
    want = [gpu_advance(m, p, 2.0, 1)[0] for m in ms]
    ctx = V.VerticalContext(p)
    errors = []

    def work(m, w):
        try:
            stream = torch.cuda.Stream()
            for _ in range(8):
                d = V.device_member(m)
                torch.cuda.synchronize()
                plan = V.Plan(ctx, [d])
                plan.advance(2.0, 1, stream=stream)
                plan.check()
                plan.close()
                got = d.to_numpy()
                for k in STATE:
                    np.testing.assert_array_equal(got[k], w[k], err_msg=k)
        except Exception as e:  # reported by the main thread
            errors.append(e)

    ts = [threading.Thread(target=work, args=x) for x in zip(ms, want)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    ctx.close()
    assert not errors, errors
