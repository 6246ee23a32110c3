"""The adjoint without saved states over more than one chunk of columns, and
over members of different altitude counts (run on a B200): bit for bit the one
that reads the states the caller saved, the members' arrays untouched; and the
chunks' buffer is not taken for callers that bring their own states."""
import pytest
import torch

from gitm_b200 import abi, synthetic
from gitm_b200 import vertical as V
from tests.test_gpu_adjoint import _ybar

pytestmark = pytest.mark.gpu
BARS = ("ndensity_s", "idensity_s", "rho", "temperature", "velocity", "vert_vel", "log_ns", "ndensity", "eddy",
        "heating_scale")


@pytest.mark.parametrize("shape", [((6100, 50),), ((3100, 50), (1, 50), (700, 30)), ((130, 8), (3001, 64))], ids=str)
def test_chunks(shape):
    p = abi.default_params()
    ms = [synthetic.make_member(n, a, seed=70 + i, with_heating=True) for i, (n, a) in enumerate(shape)]
    ctx = V.VerticalContext(p)
    dms = [V.device_member(m) for m in ms]
    plan = V.Plan(ctx, dms)
    dev = torch.device("cuda")
    ys = [_ybar(m, torch.Generator().manual_seed(9), dev) for m in ms]

    def bars():
        out = []
        for dm, y in zip(dms, ys):
            b = {k: v.clone() for k, v in y.items()}
            b["eddy"] = torch.zeros_like(dm.tensors["eddy"])
            b["heating_scale"] = torch.zeros(dm.n_cols, dtype=torch.float64, device=dev)
            out.append(b)
        return out

    before = [{k: v.clone() for k, v in dm.tensors.items() if v is not None} for dm in dms]
    got = bars()
    plan.adjoint(got, 2.0)
    torch.cuda.synchronize()
    for dm, b in zip(dms, before):
        for k, v in b.items():
            assert torch.equal(dm.tensors[k], v), k
    states = torch.empty(plan.saved_state_doubles(), dtype=torch.float64, device=dev)
    plan.advance_saving(2.0, states)
    for dm, b in zip(dms, before):
        for k, v in b.items():
            dm.tensors[k].copy_(v)
    want = bars()
    plan.adjoint(want, 2.0, saved=states)
    plan.check()
    for g, w in zip(got, want):
        for k in BARS:
            assert torch.equal(g[k], w[k]), k
            assert bool(torch.isfinite(g[k]).all()) and float(g[k].abs().max()) > 0.0, k
    plan.close()
    ctx.close()


def test_buffer_only_without_saved_states():
    """2,592 columns of 50 altitudes: 137 MB of stage states for a call
    without saved ones, nothing of that size for one with them."""
    p = abi.default_params()
    m = synthetic.make_member(2592, 50, seed=77)
    ctx = V.VerticalContext(p)
    dm = V.device_member(m)
    plan = V.Plan(ctx, [dm])
    dev = torch.device("cuda")
    y = _ybar(m, torch.Generator().manual_seed(9), dev)
    states = torch.empty(plan.saved_state_doubles(), dtype=torch.float64, device=dev)
    y["eddy"] = torch.zeros_like(dm.tensors["eddy"])
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    plan.advance_saving(2.0, states)
    plan.adjoint([{k: v for k, v in y.items()}], 2.0, saved=states)
    torch.cuda.synchronize()
    with_states = free - torch.cuda.mem_get_info()[0]
    plan.adjoint([{k: v for k, v in y.items()}], 2.0)
    torch.cuda.synchronize()
    without = free - torch.cuda.mem_get_info()[0]
    plan.close()
    ctx.close()
    assert with_states < 16 << 20 and without - with_states > 128 << 20, (with_states, without)
