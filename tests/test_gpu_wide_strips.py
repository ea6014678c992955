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
