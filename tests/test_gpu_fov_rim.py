"""Which pixels the backprojectors give a value: those whose FP64 centre lies in the FOV disc,
whatever precision the kernels decide it in.  Image sizes with centres within 1e-6 of the rim
(their FP32 radii round to either side), non-square images, and radii whose squares FP32 cannot
hold."""
from __future__ import annotations

import numpy as np
import pytest

from fanbeamctrecon_tensorflowop_gb300.geometry import angle, fan_param16

pytestmark = pytest.mark.gpu


def _disc(g):
    """The backprojector's test: centres (FP32 origin and pitch, FP64 arithmetic) in the disc."""
    x = np.float64(g.xmin) + np.float64(g.dx) * (np.arange(g.nx) + 0.5)
    y = np.float64(g.ymin) + np.float64(g.dy) * (np.arange(g.ny) + 0.5)
    r = np.float64(g.rfov)
    return x[None, :] ** 2 + y[:, None] ** 2 <= r * r


@pytest.mark.parametrize("n,ny", [(1, None), (5, None), (13, 9), (512, None), (719, 1001),
                                  (2048, None), (3001, None)])
@pytest.mark.parametrize("scale", [1.0, 1e-21, 1e21])
@pytest.mark.parametrize("nb", [1, 4])
def test_bp_fills_the_disc(cuda, n, ny, scale, nb):
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import FanPlan
    p = fan_param16(sdd=949.0 * scale, sid=541.0 * scale, n_views=3, n_cols=40, n=n, ny=ny,
                    pixel_mm=358.4 / n * scale, dcol_rad=2 * 0.47 / 40)
    plan = FanPlan(p, angle(3, 0.2), device=cuda)
    got = plan.bp(torch.ones((nb, 3, 40), device=cuda))
    want = torch.from_numpy(_disc(plan.geom)).to(cuda)
    assert 0 < int(want.sum()) < n * (ny or n) or n == 1
    # three views of ones: weights 1 - f and f sum to one within two roundings each
    assert bool(((got - 3.0 * want).abs() <= 3e-6).all())


@pytest.mark.parametrize("n,nz", [(9, 5), (512, 3), (719, 9)])
def test_fdk_fills_the_disc(cuda, n, nz):
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import ConePlan
    p = fan_param16(sdd=949.0, sid=541.0, n_views=3, n_cols=40, n=n, pixel_mm=358.4 / n,
                    dcol_rad=2 * 0.47 / 40, det_bottom=-24.0, drow=6.0, dz=40.0 / nz)
    plan = ConePlan(p, angle(3, 0.2), 8, nz, device=cuda)
    # random projections: hardly any voxel's sum is exactly zero
    proj = torch.rand((1, 3, 8, 40), device=cuda)
    got = plan.fdk(proj)[0]
    want = torch.from_numpy(_disc(plan.geom)).to(cuda)
    assert not bool(got[:, ~want].any())
    assert bool((got[:, want] != 0).float().mean() > 0.999)
