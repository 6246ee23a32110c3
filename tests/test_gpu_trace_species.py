"""A species of hardly any density (run on a B200): the friction solve scales
the rows of its matrix by the species' mass densities, which for a density
below 1e-282 are no normal numbers any more.  The step takes such a column as
the reference does, against the oracle."""
import numpy as np
import pytest

from gitm_b200 import abi, synthetic
from tests.parity import assert_state_close
from tests.test_gpu_parity import STATE, gpu_advance, ref_advance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [512, 256, 128])
@pytest.mark.parametrize("scale", [1e-250, 1e-295, 1e-300], ids=str)
def test_trace_species(oracle_lib, scale, threads):
    p = abi.default_params()
    m = synthetic.make_member(24, 50, seed=81)
    for s, bad in ((3, 4), (5, 11)):  # N and He: their densities come to scale * (1e5 .. 1e13)
        m.ndensity_s[s, :, bad] *= scale
    ref, st_ref = ref_advance(oracle_lib, m, p, 2.0)
    assert (st_ref == 0).all() and all(np.isfinite(ref[k]).all() for k in STATE)
    out, st = gpu_advance(m, p, 2.0, config=dict(threads=threads))
    np.testing.assert_array_equal(st, st_ref)
    assert_state_close(out, ref, STATE)


@pytest.mark.parametrize("threads", [384, 256])
@pytest.mark.parametrize("scale", [1e-292, 1e-302], ids=str)
def test_trace_species_ausm(oracle_lib, scale, threads):
    """At 1e-302 the species' mass densities are subnormal, for the reference
    too (1e6 to 1e8 times the smallest of them, so of 6 to 8 digits): its own
    winds are compared to 1e-5."""
    p = abi.default_params(solver=abi.SOLVER_AUSM)
    m = synthetic.make_member(24, 50, seed=82)
    m.ndensity_s[5, :, 11] *= scale
    ref, st_ref = ref_advance(oracle_lib, m, p, 2.0)
    assert (st_ref == 0).all() and all(np.isfinite(ref[k]).all() for k in STATE)
    out, st = gpu_advance(m, p, 2.0, config=dict(threads=threads))
    np.testing.assert_array_equal(st, st_ref)
    if scale < 1e-300:
        np.testing.assert_allclose(out["vert_vel"][5, :, 11], ref["vert_vel"][5, :, 11], rtol=1e-5, atol=1e-5)
        out["vert_vel"][5, :, 11] = ref["vert_vel"][5, :, 11]
    assert_state_close(out, ref, STATE)


def test_trace_species_adjoint():
    """Against autograd through the transcription.  The species' own density
    adjoint is compared as that of its logarithm."""
    import torch
    from tests.test_gpu_adjoint import _gpu_vjp, _rel, _torch_vjp, _ybar
    p = abi.default_params()
    m = synthetic.make_member(6, 50, seed=83)
    m.ndensity_s[5, :, 3] *= 1e-295
    y = _ybar(m, torch.Generator().manual_seed(4), torch.device("cuda"))
    want = _torch_vjp(m, p, 2.0, y, torch.device("cuda"))
    got, status = _gpu_vjp(m, p, 2.0, y)
    assert status == (0, 0)
    nd = torch.from_numpy(m.ndensity_s)
    for k in ("vert_vel", "temperature", "velocity", "rho", "eddy"):
        assert _rel(got[k], want[k]) < 1e-9, (k, _rel(got[k], want[k]))
    for s in range(6):
        g, w = got["ndensity_s"][s].cpu() * nd[s], want["ndensity_s"][s].cpu() * nd[s]
        assert _rel(g, w) < 1e-9, (s, _rel(g, w))
