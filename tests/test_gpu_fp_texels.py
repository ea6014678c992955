"""The forward projector's texel walk and its transpose where their tiles, slice
groups and rays end: image edges around the 32-texel build tile and the 4 x 8
cell patch, slice counts around the groups of 1, 2, 4, 8 and 16 slices, rays at
the layout diagonals, and non-finite pixels."""
from __future__ import annotations

import numpy as np
import pytest

from fanbeamctrecon_tensorflowop_gb300.geometry import angle, fan_param16

pytestmark = pytest.mark.gpu

# Each texel weight of a ray is a sum of a dozen FP32 operations on values of
# order one (2^-24 each, independent), and the ray's position carries the FP32
# table's rounding, at most 2^-18 texel for images of up to 66 texels, times a
# texel difference of up to one: 1e-6 of the ray's sum at most, doubled.
TOL = 2e-6


def _plan(n, views=45, cols=71, ny=None):
    from fanbeamctrecon_tensorflowop_gb300 import FanPlan
    # a fan of +-0.34 rad about a field of view of 179.2 mm: the outer rays miss it
    p = fan_param16(sdd=949.0, sid=541.0, n_views=views, n_cols=cols, n=n, ny=ny,
                    pixel_mm=358.4 / n, dcol_rad=0.75 / cols)
    a = angle(views, 0.0)
    return p, a, FanPlan(p, a)


def _rel(a, b):
    return np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n,ny,nb", [(1, None, 1), (2, None, 2), (29, None, 3), (30, None, 4),
                                     (31, None, 5), (33, None, 8), (62, None, 9), (63, 40, 16),
                                     (65, None, 17), (64, 70, 33), (34, None, 66)])
def test_fp_edges_and_slice_groups(cuda, orc, n, ny, nb):
    import torch
    p, a, plan = _plan(n, ny=ny)
    g = orc.decode(p)
    x = np.random.default_rng(n).random((nb, g.ny, g.nx), dtype=np.float32)
    xt = torch.from_numpy(x).to(cuda)
    got = plan.fp(xt)
    pick = sorted({0, nb // 2, nb - 1})
    ref = orc.fp_fan(g, a, x[pick])
    assert _rel(got[pick].cpu().numpy(), ref) <= TOL
    for b in pick:  # the same arithmetic whatever the group
        assert torch.equal(plan.fp(xt[b:b + 1])[0], got[b]), b


@pytest.mark.parametrize("nb", [1, 2, 4, 8, 16])
def test_fp_nonfinite_pixel_stays_on_its_rays(cuda, nb):
    """An infinite pixel makes the rays that touch it infinite (not NaN) and
    leaves the others as they are; a NaN pixel likewise."""
    import torch
    _, _, plan = _plan(40)
    x = torch.rand((nb, 40, 40), device=cuda)
    delta = torch.zeros_like(x)
    delta[:, 13, 22] = 1.0
    clean, touched = plan.fp(x * (1 - delta)), plan.fp(delta) > 0
    for bad in (float("inf"), float("nan")):
        y = x.clone()
        y[:, 13, 22] = bad
        got = plan.fp(y)
        assert torch.equal(got[~touched], clean[~touched])
        hit = got[touched]
        assert bool((torch.isnan(hit) if bad != bad else torch.isposinf(hit)).all())


@pytest.mark.parametrize("n,ny,views,nb", [(1, None, 3, 1), (2, None, 45, 2), (4, None, 16, 4),
                                           (5, None, 17, 5), (9, None, 1, 8), (33, 20, 45, 9),
                                           (40, 47, 45, 16), (36, None, 44, 17),
                                           (64, None, 45, 3), (30, None, 45, 66)])
def test_fp_adjoint_edges_and_slice_groups(cuda, orc, n, ny, views, nb):
    """Against the oracle's transpose: a texel sums at most 2 x views rays, each
    with the weight rounding of TOL, in FP32 (2^-24 per add): twice TOL."""
    import torch
    p, a, plan = _plan(n, views=views, ny=ny)
    g = orc.decode(p)
    y = np.random.default_rng(n).random((nb, views, 71), dtype=np.float32)
    yt = torch.from_numpy(y).to(cuda)
    got = plan.fp_adjoint(yt)
    pick = sorted({0, nb // 2, nb - 1})
    assert _rel(got[pick].cpu().numpy(), orc.fp_fan_adjoint(g, a, y[pick])) <= 2 * TOL
    for b in pick:
        assert torch.equal(plan.fp_adjoint(yt[b:b + 1])[0], got[b]), b
