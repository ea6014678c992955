"""The pixel-driven backprojector where its pixel blocks, view shares and slice
groups end: images around the 8 x 4 block, fewer views than shares, odd view
counts, slice counts around the groups of 1, 2, 4, 8, 12 and 16, and plans on
either side of the rule that drops the detector range test; likewise the
cone-beam backprojector's 8 x 4 x 8 voxel blocks and the transpose's strips."""
from __future__ import annotations

import math

import numpy as np
import pytest

from fanbeamctrecon_tensorflowop_gb300.geometry import angle, fan_param16

pytestmark = pytest.mark.gpu

# The FP32 column position (up to 100 channels, half a dozen roundings of 2^-24)
# moves an interpolated U[0,1) value by at most 5e-5 of a channel times 1, at
# random over the views; the sums add 2^-24 each: 2e-5 of the result.
TOL = 2e-5


def _plan(n, views=45, cols=71, ny=None, half=0.37, **kw):
    """A fan of +-half rad about a FOV of +-0.3377 rad."""
    from fanbeamctrecon_tensorflowop_gb300 import FanPlan
    p = fan_param16(sdd=949.0, sid=541.0, n_views=views, n_cols=cols, n=n, ny=ny,
                    pixel_mm=358.4 / n, dcol_rad=2 * half / cols)
    a = angle(views, 0.2)
    return p, a, FanPlan(p, a, **kw)


def _rel(a, b):
    return np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n,ny,views,nb", [(1, None, 45, 1), (3, None, 1, 2), (7, None, 2, 3),
                                           (8, 5, 15, 4), (9, 4, 16, 5), (31, None, 17, 8),
                                           (33, 40, 45, 9), (32, None, 44, 12), (40, 33, 45, 13),
                                           (36, None, 45, 17), (24, None, 7, 66)])
@pytest.mark.parametrize("half", [0.37, 0.30])  # covers the FOV, or truncates it
def test_bp_edges_and_slice_groups(cuda, orc, n, ny, views, nb, half):
    import torch
    p, a, plan = _plan(n, views, ny=ny, half=half)
    g = orc.decode(p)
    y = np.random.default_rng(n).random((nb, views, 71), dtype=np.float32)
    yt = torch.from_numpy(y).to(cuda)
    got, fbp = plan.bp(yt), plan.fbp(yt)
    pick = sorted({0, nb // 2, nb - 1})
    ref = orc.bp_fan(g, a, y[pick])
    assert _rel(got[pick].cpu().numpy(), ref) <= TOL
    for b in pick:  # the same arithmetic whatever the group
        assert torch.equal(plan.bp(yt[b:b + 1])[0], got[b]), b
        assert torch.equal(plan.fbp(yt[b:b + 1])[0], fbp[b]), b


@pytest.mark.parametrize("channels", [0.9, 1.0, 1.005, 1.02, 1.2])
def test_bp_range_test_rule(cuda, orc, channels):
    """Fans that extend beyond the FOV by about one channel, where the form
    without range test and clamp begins: both meet the oracle."""
    import torch
    cols, need = 90, math.asin(179.2 / 541.0)
    # the FOV's edge lies at column position y = `channels`
    half = need * (cols / 2) / (cols / 2 + 0.5 - channels)
    p, a, plan = _plan(48, 33, cols, half=half)
    y = np.random.default_rng(3).random((4, 33, cols), dtype=np.float32)
    got = plan.bp(torch.from_numpy(y).to(cuda)).cpu().numpy()
    assert _rel(got, orc.bp_fan(orc.decode(p), a, y)) <= TOL


@pytest.mark.parametrize("nb", [1, 2, 4, 16])
def test_bp_nonfinite_value_stays_on_its_pixels(cuda, nb):
    """A non-finite detector value reaches the pixels that interpolate it and no
    others (the pixels outside the FOV stay zero)."""
    import torch
    _, _, plan = _plan(40)
    y = torch.rand((nb, 45, 71), device=cuda)
    delta = torch.zeros_like(y)
    delta[:, 12, 30] = 1.0
    clean, touched = plan.bp(y * (1 - delta)), plan.bp(delta) > 0
    for bad in (float("inf"), float("nan")):
        z = y.clone()
        z[:, 12, 30] = bad
        got = plan.bp(z)
        assert torch.equal(got[~touched], clean[~touched])
        hit = got[touched]
        assert bool((torch.isnan(hit) if bad != bad else torch.isposinf(hit)).all())


@pytest.mark.parametrize("n,nz,rows,views,batch", [(1, 1, 2, 3, 1), (7, 7, 5, 1, 2), (8, 8, 8, 4, 1),
                                                   (9, 9, 6, 9, 2), (17, 17, 12, 15, 1),
                                                   (33, 3, 9, 16, 3)])
@pytest.mark.parametrize("half", [0.37, 0.30])
def test_fdk_edges(cuda, orc, n, nz, rows, views, batch, half):
    """FDK against the oracle at its 1e-4 contract (the filter amplifies the
    column rounding), and a volume of a batch against the volume alone."""
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import ConePlan
    p = fan_param16(sdd=949.0, sid=541.0, n_views=views, n_cols=72, n=n, pixel_mm=358.4 / n,
                    dcol_rad=2 * half / 72, det_bottom=-24.0, drow=48.0 / rows, dz=40.0 / nz)
    a = angle(views, 0.1)
    plan = ConePlan(p, a, rows, nz)
    y = np.random.default_rng(n).random((batch, views, rows, 72), dtype=np.float32)
    yt = torch.from_numpy(y).to(cuda)
    got = plan.fdk(yt)
    assert _rel(got.cpu().numpy(), orc.fdk_cone(orc.decode(p), rows, nz, a, y)) <= 1e-4
    assert torch.equal(plan.fdk(yt[-1:])[0], got[-1])


@pytest.mark.parametrize("n,ny,cols,nb", [(5, None, 40, 1), (33, 40, 71, 2), (64, None, 9, 1),
                                          (64, None, 16, 5), (40, 31, 200, 9), (48, None, 62, 17),
                                          (96, None, 12, 4)])
@pytest.mark.parametrize("half", [0.37, 0.30])
def test_bp_adjoint_strips(cuda, orc, n, ny, cols, nb, half):
    """Strips from a fraction of a pixel to a dozen pixels wide, with channel
    counts around the 31 of a warp: the column fractions carry ~1e-7 and the
    sums 2^-24 per add, 2e-6 of the result."""
    import torch
    p, a, plan = _plan(n, 37, cols, ny=ny, half=half)
    g = orc.decode(p)
    x = np.random.default_rng(n).random((nb, g.ny, g.nx), dtype=np.float32)
    xt = torch.from_numpy(x).to(cuda)
    got = plan.bp_adjoint(xt)
    assert _rel(got.cpu().numpy(), orc.bp_fan_transpose(g, a, x)) <= 2e-6
    assert torch.equal(plan.bp_adjoint(xt[-1:])[0], got[-1])


@pytest.mark.parametrize("views", [1988, 2012])
@pytest.mark.parametrize("nb", [1, 3])
def test_bp_adjoint_split_views(cuda, orc, views, nb):
    """Either side of the block count below which a block's warps share one view's lines
    (three channel groups of 497 and 503 view quads): 2e-6 as above, a slice of a batch as alone."""
    import torch
    p, a, plan = _plan(13, views, 70)
    g = orc.decode(p)
    x = np.random.default_rng(nb).random((nb, g.ny, g.nx), dtype=np.float32)
    xt = torch.from_numpy(x).to(cuda)
    got = plan.bp_adjoint(xt)
    assert _rel(got.cpu().numpy(), orc.bp_fan_transpose(g, a, x)) <= 2e-6
    assert torch.equal(plan.bp_adjoint(xt[-1:])[0], got[-1])
