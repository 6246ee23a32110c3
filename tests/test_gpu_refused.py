"""A column that a step refuses (a density that is not positive) in the calls
that stage their arrays (run on a B200): the state it came with is kept, and
LogNS and NDensity, which the step does not form for it, come back as zeros
whatever the staging memory held before."""
import ctypes as C

import numpy as np
import pytest

from gitm_b200 import _lib, abi, synthetic
from gitm_b200 import vertical as V
from tests.test_gpu_fortran import NLAT, NLON, fortran_arrays, state_struct

pytestmark = pytest.mark.gpu

N, N_ALTS = NLON * NLAT, 30
BAD = 31  # column (i, j) = (4, 3)


def fortran_call(ctx, f, on_device):
    """One step of one block; returns the code and the arrays after it."""
    import torch
    held = {k: torch.from_numpy(v).cuda() for k, v in f.items()} if on_device else f

    def getptr(name):
        a = held[name]
        strides = list(a.stride()) if on_device else [s // 8 for s in a.strides]
        if name in ("mean_major_mass", "temp_unit"):
            strides[3] = 0
        return (a.data_ptr() if on_device else a.ctypes.data), strides

    st = state_struct(N_ALTS, 1, getptr)
    rc = _lib.lib().gitm_vert_advance_fortran(ctx.handle, C.byref(st), 1, 1, 2.0, on_device)
    if on_device:
        torch.cuda.synchronize()
        return rc, {k: v.cpu().numpy() for k, v in held.items()}
    return rc, f


@pytest.mark.parametrize("on_device", [1, 0], ids=["device", "host"])
def test_fortran_arrays(on_device):
    ctx = V.VerticalContext(abi.default_params(compute_coefficients=0))
    good = fortran_arrays(synthetic.make_member(N, N_ALTS, seed=11), 1)
    rc, _ = fortran_call(ctx, good, on_device)  # leaves its LogNS and NDensity in the staging memory
    assert rc == abi.OK, ctx.last_error()
    m = synthetic.make_member(N, N_ALTS, seed=12)
    m.ndensity_s[2, 20, BAD] = 0.0
    f = fortran_arrays(m, 1)
    before = {k: v.copy() for k, v in f.items()}
    rc, out = fortran_call(ctx, f, on_device)
    ctx.close()
    assert rc == abi.ERR_COLUMN
    li, lj = BAD % NLON + 2, BAD // NLON + 2
    for k in ("ndensity_s", "idensity_s", "rho", "temperature", "velocity", "vertical_velocity"):
        np.testing.assert_array_equal(out[k][li, lj], before[k][li, lj], err_msg=k)
    for k in ("log_ns", "ndensity"):
        np.testing.assert_array_equal(out[k][li, lj], np.zeros_like(out[k][li, lj]), err_msg=k)
        assert (out[k][li - 1, lj] != before[k][li - 1, lj]).all()  # a column that was advanced


def test_host_pointers():
    """The host-pointer call, whose coefficients come from the step: the
    refused column, and cMax's outermost cells, which the step does not form."""
    ctx = V.VerticalContext(abi.default_params())

    def member(seed):
        m = synthetic.make_member(1500, N_ALTS, seed=seed)  # two chunks of columns
        m.log_ns, m.ndensity = np.full_like(m.ndensity_s, 7.0), np.full_like(m.rho, 7.0)
        m.cmax[:, [0, -1]] = 7.0
        return m

    V.advance_vertical_all_host(ctx, [member(13)], 2.0)
    m = member(14)
    bad = 1100
    m.ndensity_s[2, 20, bad] = 0.0
    before = m.copy()
    with pytest.raises(V.GitmStop):
        V.advance_vertical_all_host(ctx, [m], 2.0)
    ctx.close()
    for k in synthetic.Member.STATE:
        np.testing.assert_array_equal(getattr(m, k)[..., bad], getattr(before, k)[..., bad], err_msg=k)
    for k in ("log_ns", "ndensity"):
        a = getattr(m, k)
        assert (a[..., bad] == 0.0).all() and (a[..., bad - 1] != 7.0).all(), k
    np.testing.assert_array_equal(m.cmax[:, [0, -1]], before.cmax[:, [0, -1]])
    assert (m.cmax[:, 1:-1, :bad] > 0.0).all()
