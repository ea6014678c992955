"""BP adjoints of detectors coarser than the image: channels from about six pixels wide, where
the kernel's form for wide strips begins, to 10^6 images wide (a source far beyond the object)."""
from __future__ import annotations

import numpy as np
import pytest

from fanbeamctrecon_tensorflowop_gb300.geometry import angle, fan_param16

pytestmark = pytest.mark.gpu


# a boundary between two channels passes through the axis (shift 1/2), or next to it
@pytest.mark.parametrize("sid,dcol,shift", [(2e4, 0.0031, 0.0), (2e4, 0.0033, 0.0),
                                            (2e4, 0.005, 0.0), (2e4, 0.0175, 0.5),
                                            (2e4, 0.0181, 0.5003), (2e4, 0.05, 0.5),
                                            (1e6, 0.01, 0.5), (1e6, 0.01, 0.5003),
                                            (1e8, 0.01, 0.5), (1e10, 0.05, 0.5)])
@pytest.mark.parametrize("n,ny,nb", [(24, None, 1), (17, 33, 4), (20, None, 7), (31, 12, 16)])
def test_bp_adjoint_of_wide_channels(cuda, orc, sid, dcol, shift, n, ny, nb):
    """The column fractions carry ~1e-7 and the sums 2^-24 per add: 2e-6 of the result."""
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import FanPlan
    p = fan_param16(sdd=2 * sid, sid=sid, n_views=11, n_cols=6, n=n, ny=ny, pixel_mm=358.4 / n,
                    dcol_rad=dcol, shift=shift)
    a = angle(11, 0.13)
    plan = FanPlan(p, a, device=cuda)
    g = orc.decode(p)
    x = np.random.default_rng(n).random((nb, g.ny, g.nx), dtype=np.float32)
    xt = torch.from_numpy(x).to(cuda)
    got = plan.bp_adjoint(xt)
    ref = orc.bp_fan_transpose(g, a, x)
    assert np.linalg.norm(got.cpu().numpy() - ref) <= 2e-6 * np.linalg.norm(ref)
    assert torch.equal(plan.bp_adjoint(xt[-1:])[0], got[-1])


@pytest.mark.parametrize("n_cols,dcol,sid", [(96, 4.0 / 949.0, 541.0), (12, 0.08, 541.0),
                                             (6, 0.01, 1e6)])
def test_debug_build_finds_every_index_in_range(cuda, n_cols, dcol, sid):
    """The index-checking library on narrow, wide and very wide strips: no flag, equal results."""
    import torch
    from test_gpu_debug_build import _plan, _run
    from fanbeamctrecon_tensorflowop_gb300 import FanPlan, _lib
    p = fan_param16(sdd=2 * sid, sid=sid, n_views=37, n_cols=n_cols, n=45, ny=38,
                    pixel_mm=358.4 / 45, dcol_rad=dcol, shift=0.5)
    a = angle(37, 0.13)
    dlib = _lib.load_debug()
    h, ref = _plan(dlib, p, a), FanPlan(p, a, device=cuda)
    for nb in (1, 3, 7, 20):
        x = torch.rand((nb, *ref.image_shape), device=cuda)
        got = _run(dlib, h, "ct_bp_fan_adjoint", None, x, (nb, *ref.sino_shape), cuda)
        torch.testing.assert_close(got, ref.bp_adjoint(x), rtol=1e-5, atol=1e-4)
        assert dlib.ct_plan_check(h) == 0, dlib.ct_last_error()
    assert dlib.ct_plan_destroy(h) == 0
