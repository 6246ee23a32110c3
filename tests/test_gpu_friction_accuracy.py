"""The friction solve against one in 80 bits (run on a B200).  Where friction
is strong the species' common velocity hangs on the diagonal's surplus over
the couplings, which a diagonal held as one number loses: the step's winds
have to be nearer to the 80-bit solution than those of a 64-bit LU of the
matrix by a factor of two (measured before at 20 altitudes: 0.15 of its error;
an elimination that subtracts from the diagonal 0.84)."""
import numpy as np
import pytest
import torch

from gitm_b200 import abi, synthetic
from tests import torch_step as TS
from tests.test_gpu_parity import gpu_advance

pytestmark = pytest.mark.gpu


def solve_80bit(a, b):
    """a v = b for rows 1 + sum_j c_ij on the diagonal, -c_ij beside it: the
    diagonal from its parts, all in long double."""
    a, b = (x.detach().cpu().numpy().astype(np.longdouble) for x in (a, b))
    n = a.shape[-1]
    for r in range(n):
        a[..., r, r] = 0
        a[..., r, r] = 1 - a[..., r, :].sum(-1)
    for p in range(n):
        for r in range(p + 1, n):
            f = a[..., r, p] / a[..., p, p]
            a[..., r, p:] -= f[..., None] * a[..., p, p:]
            b[..., r] -= f * b[..., p]
    for r in reversed(range(n)):
        b[..., r] = (b[..., r] - (a[..., r, r + 1:] * b[..., r + 1:]).sum(-1)) / a[..., r, r]
    return torch.from_numpy(b.astype(np.float64))


@pytest.mark.parametrize("threads", [512, 256])
def test_friction_accuracy(monkeypatch, threads):
    p = abi.default_params()
    m = synthetic.make_member(200, 20, seed=61)
    out, st = gpu_advance(m, p, 2.0, config=dict(threads=threads))
    assert (st == 0).all()
    lu = TS.to_member_arrays(TS.step(*TS.from_member(m), p, 2.0))["vert_vel"]
    monkeypatch.setattr(torch.linalg, "solve", solve_80bit)
    want = TS.to_member_arrays(TS.step(*TS.from_member(m), p, 2.0))["vert_vel"]
    err = [np.linalg.norm(x - want) / np.linalg.norm(want) for x in (out["vert_vel"], lu)]
    assert err[0] < 0.5 * err[1], err
