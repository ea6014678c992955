"""Backprojections without a workspace: BP of up to three slices allocates nothing, and the
groups of one, two, three and four slices that read the sinograms themselves give each slice
the bits it has alone."""
from __future__ import annotations

import numpy as np
import pytest

from fanbeamctrecon_tensorflowop_gb300.geometry import angle, fan_param16

pytestmark = pytest.mark.gpu


def _plan(half, **kw):
    from fanbeamctrecon_tensorflowop_gb300 import FanPlan
    p = fan_param16(sdd=949.0, sid=541.0, n_views=45, n_cols=71, n=37, ny=30,
                    pixel_mm=358.4 / 37, dcol_rad=2 * half / 71)
    a = angle(45, 0.2)
    return p, a, FanPlan(p, a, **kw)


@pytest.mark.parametrize("nb", [1, 2, 3])
@pytest.mark.parametrize("half", [0.37, 0.30])  # covers the FOV, or truncates it
@pytest.mark.parametrize("tex", [False, True])
def test_bp_of_few_slices_allocates_nothing(cuda, orc, nb, half, tex):
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import _lib
    p, a, plan = _plan(half, texture_weights=tex)
    y = np.random.default_rng(nb).random((nb, 45, 71), dtype=np.float32)
    yt = torch.from_numpy(y).to(cuda)
    count = _lib.load().ct_device_alloc_count()
    got = plan.bp(yt)
    assert _lib.load().ct_device_alloc_count() == count
    for b in range(nb):
        assert torch.equal(plan.bp(yt[b:b + 1])[0], got[b])
    if not tex:  # FP32 column positions: 2e-5 of the result, as for larger batches
        ref = orc.bp_fan(orc.decode(p), a, y)
        assert np.linalg.norm(got.cpu().numpy() - ref) <= 2e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("nb", [3, 5, 6, 7, 8])
@pytest.mark.parametrize("half", [0.37, 0.30])
def test_static_scratch_groups(cuda, nb, half):
    """4 + 1, 4 + 2, 4 + 3 slices and whole groups, against the planes of ct_fbp_fan."""
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import _lib
    _, _, plan = _plan(half)
    y = torch.rand((nb, 45, 71), device=cuda)
    out = torch.full((nb, *plan.image_shape), float("nan"), device=cuda)
    lib = _lib.load()
    assert lib.ct_fbp_fan_static_scratch(plan._h, y.data_ptr(), out.data_ptr(), nb,
                                         torch.cuda.current_stream(cuda).cuda_stream) == 0
    assert torch.equal(out, plan.fbp(y))
