"""Altitude grids that the coefficient kernel does not read where they stand
(run on a B200): an empty member without grids is refused as an error of the
call, one with grids is taken, and a grid at an address that is no multiple of
8 gives the bits of an aligned one."""
import ctypes as C

import numpy as np
import pytest
import torch

from gitm_b200 import abi, synthetic
from gitm_b200 import vertical as V
from gitm_b200._lib import lib
from tests.test_gpu_parity import STATE, gpu_advance

pytestmark = pytest.mark.gpu
GRID = ("altitude", "gravity", "dalt_c", "inv_r")


def test_empty_member():
    p = abi.default_params()
    m = synthetic.make_member(20, 50, seed=5)
    want, _ = gpu_advance(m, p, 2.0)
    ctx = V.VerticalContext(p)
    dm = V.device_member(m)
    empty = abi.GitmColumnBatch()
    empty.n_alts, empty.n_cols = 50, 0
    h = C.c_void_p()
    arr = (abi.GitmColumnBatch * 2)(dm.batch(), empty)
    assert lib().gitm_vert_plan_create(ctx.handle, arr, 2, C.byref(h)) == abi.ERR_CUDA
    for k in GRID:
        setattr(empty, k, abi.dptr(dm.tensors[k].data_ptr()))
    arr = (abi.GitmColumnBatch * 2)(dm.batch(), empty)
    assert lib().gitm_vert_plan_create(ctx.handle, arr, 2, C.byref(h)) == abi.OK
    assert lib().gitm_vert_plan_advance(h, 2.0, 1, None) == abi.OK
    lib().gitm_vert_plan_destroy(h)
    ctx.close()
    for k in STATE:
        np.testing.assert_array_equal(dm.to_numpy()[k], want[k], err_msg=k)


def test_unaligned_grid():
    p = abi.default_params()
    m = synthetic.make_member(20, 50, seed=6)
    want, _ = gpu_advance(m, p, 2.0)
    ctx = V.VerticalContext(p)
    dm = V.device_member(m)
    b = dm.batch()
    held = []
    for k in GRID:
        raw = torch.zeros(8 * 54 + 8, dtype=torch.uint8, device="cuda")
        raw[4:4 + 8 * 54] = torch.from_numpy(np.ascontiguousarray(getattr(m, k)).view(np.uint8)).cuda()
        held.append(raw)
        setattr(b, k, abi.dptr(raw.data_ptr() + 4))
    torch.cuda.synchronize()
    assert lib().gitm_vert_advance_native(ctx.handle, (abi.GitmColumnBatch * 1)(b), 1, 2.0, 1) == abi.OK
    ctx.close()
    for k in STATE:
        np.testing.assert_array_equal(dm.to_numpy()[k], want[k], err_msg=k)
