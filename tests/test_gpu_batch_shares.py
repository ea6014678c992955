"""Uneven batches whose blocks share a unit among their warps: every FP, BP, FBP and
FBP-adjoint item gives the bits of its plan's own call, with fewer views than the
backprojector's eight shares (warps without views write their sums at once), odd view counts,
images around the 8 x 4 pixel block and the 32-pixel tile, tiles that are partly outside the
FOV disc, and fans that cover and truncate it, under both schedules and both tile heights."""
from __future__ import annotations

import pytest

from fanbeamctrecon_tensorflowop_gb300.geometry import angle, fan_param16

pytestmark = pytest.mark.gpu

# n, ny, views, half fan (the FOV is +-0.3377 rad)
SHAPES = [(8, None, 1, 0.37), (64, None, 1, 0.30), (33, 40, 2, 0.37), (96, None, 2, 0.37),
          (32, None, 7, 0.30), (160, 97, 7, 0.37), (31, 64, 14, 0.37), (200, None, 14, 0.30),
          (70, 129, 45, 0.37), (128, None, 45, 0.30)]
OPS = ("bp", "fbp", "fp", "fbp_adjoint")


@pytest.mark.parametrize("rows", [16, 32])
@pytest.mark.parametrize("dynamic", [0, 1])
@pytest.mark.parametrize("blocks", [1, 4])
def test_batch_units_equal_the_plans_calls(cuda, rows, dynamic, blocks):
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import FanPlan
    from fanbeamctrecon_tensorflowop_gb300.batch import UnevenBatch
    gen = torch.Generator(device=cuda).manual_seed(rows + dynamic)
    items, want = [], []
    for n, ny, views, half in SHAPES:
        p = fan_param16(sdd=949.0, sid=541.0, n_views=views, n_cols=71, n=n, ny=ny,
                        pixel_mm=358.4 / n, dcol_rad=2 * half / 71)
        plan = FanPlan(p, angle(views, 0.2), device=cuda)
        for op in OPS:
            to_sino = op in ("fp", "fbp_adjoint")
            x = torch.rand(plan.image_shape if to_sino else plan.sino_shape, device=cuda,
                           generator=gen)
            y = torch.full(plan.sino_shape if to_sino else plan.image_shape, float("nan"),
                           device=cuda)
            items.append((plan, op, x, y))
            want.append(getattr(plan, op)(x)[0])
    ub = UnevenBatch(items)
    ub.set_config(dict(fp_blocks_per_sm=blocks, fp_dynamic=dynamic, bp_blocks_per_sm=blocks,
                       bp_dynamic=dynamic, bp_tile_rows=rows))
    try:
        for _ in range(3):
            for *_, y in items:
                y.fill_(float("nan"))
            ub.run()
            for (plan, op, _, y), w in zip(items, want):
                assert torch.equal(y, w), (op, plan.image_shape, plan.sino_shape)
    finally:
        ub.set_config(None)
