"""The FP adjoint of few views, where a warp takes all views of its cells: either side of the rule
(views * 8000 <= pixels, at most 24), odd view counts, images around the block's 16 x 16 cells,
slice groups of 1, 4, 8 and 16, a fan that truncates the FOV and one of 92 degrees."""
from __future__ import annotations

import numpy as np
import pytest

from fanbeamctrecon_tensorflowop_gb300.geometry import angle, fan_param16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ny,views,nb", [(200, None, 5, 1), (200, None, 6, 1), (193, 209, 5, 3),
                                           (177, 130, 2, 8), (178, 131, 3, 13), (90, None, 1, 17),
                                           (89, 90, 1, 1), (450, None, 24, 2), (450, None, 25, 2)])
@pytest.mark.parametrize("sid", [541.0, 260.0])  # FOV within +-0.34 and +-0.76 rad
def test_fp_adjoint_of_few_views(cuda, orc, n, ny, views, nb, sid):
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import FanPlan
    half = 0.30 if sid > 500 else 0.8  # truncating, and wider than the FOV
    p = fan_param16(sdd=2 * sid, sid=sid, n_views=views, n_cols=120, n=n, ny=ny,
                    pixel_mm=358.4 / n, dcol_rad=2 * half / 120)
    a = angle(views, 0.2)
    plan = FanPlan(p, a, device=cuda)
    y = np.random.default_rng(n).random((nb, views, 120), dtype=np.float32)
    yt = torch.from_numpy(y).to(cuda)
    got = plan.fp_adjoint(yt)
    ref = orc.fp_fan_adjoint(orc.decode(p), a, y[[0, nb - 1]])
    # a sample's texture coordinates (up to 450) round by 2^-16, and its weights with them
    err = np.linalg.norm(got[[0, nb - 1]].cpu().numpy() - ref)
    assert err <= 2e-5 * np.linalg.norm(ref)
    assert torch.equal(plan.fp_adjoint(yt[-1:])[0], got[-1])
