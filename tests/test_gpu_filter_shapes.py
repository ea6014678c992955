"""The ramp filter's forms at their edges: the direct FP32 form's row groups
(1, 2, 4, 8 rows per block) and output quads, the tensor-core form's tile
widths, and the pre-weights' vector and scalar forms."""
from __future__ import annotations

import numpy as np
import pytest

from fanbeamctrecon_tensorflowop_gb300.geometry import angle, fan_param16

pytestmark = pytest.mark.gpu

# A filtered value is a sum of up to 100 FP32 products (2^-24 each) whose
# magnitudes sum to some ten times the result: 6e-5; the contract is 1e-4.
TOL = 1e-4


def _geom(cols, views=5):
    return (fan_param16(sdd=949.0, sid=541.0, n_views=views, n_cols=cols, n=16, pixel_mm=20.0,
                        dcol_rad=0.74 / cols), angle(views, 0.0))


def _rel(a, b):
    return np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("cols", [1, 2, 3, 4, 5, 7, 8, 9, 15, 17, 33, 71, 98])
@pytest.mark.parametrize("window", [0, 1])
def test_direct_filter_widths_and_row_groups(cuda, orc, cols, window):
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import FanPlan, _lib
    p, a = _geom(cols)
    plan = FanPlan(p, a, window=window, filter_algo=_lib.FILTER_DIRECT)
    g = orc.decode(p)
    y = np.random.default_rng(cols).random((487, 5, cols), dtype=np.float32)
    yt = torch.from_numpy(y).to(cuda)
    whole = plan.ramp_filter(yt)  # 2,435 rows: eight per block, the last block ragged
    ref = orc.ramp_filter(g, y[-3:], window)
    assert _rel(whole[-3:].cpu().numpy(), ref.reshape(3, 5, cols)) <= TOL
    for nb in (1, 61, 122):  # 5, 305 and 610 rows: one, two and four per block
        assert torch.equal(plan.ramp_filter(yt[:nb]), whole[:nb]), nb


@pytest.mark.parametrize("cols", [32, 64, 68, 200, 228, 888])
def test_tensor_core_filter_tile_widths(cuda, cols):
    """Few rows take narrow tiles, many wide ones: the same bits."""
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import FanPlan, _lib
    p, a = _geom(cols, views=41)
    plan = FanPlan(p, a, filter_algo=_lib.FILTER_TOEPLITZ_TC)
    wide = 152 * 128 // 41 + 1  # more row tiles than SMs
    yt = torch.rand((wide, 41, cols), device=cuda)
    whole = plan.ramp_filter(yt)
    for nb in (1, 4, 35, 75, 160):
        assert torch.equal(plan.ramp_filter(yt[:nb]), whole[:nb]), nb


@pytest.mark.parametrize("cols", [70, 72])
@pytest.mark.parametrize("shift", [0, 1])
def test_preweight_forms(cuda, orc, cols, shift):
    """Rows as float4, rows whose length is not a multiple of four, and buffers
    that do not start on a 16-byte boundary."""
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import FanPlan, _lib
    p, a = _geom(cols, views=33)
    plan = FanPlan(p, a, cosine_weight=True, filter_algo=_lib.FILTER_DIRECT)
    y = np.random.default_rng(0).random((3, 33, cols), dtype=np.float32)
    buf = torch.empty(3 * 33 * cols + 1, device=cuda)
    yt = buf[shift:shift + 3 * 33 * cols].view(3, 33, cols)
    yt.copy_(torch.from_numpy(y))
    got = plan.fbp(yt).cpu().numpy()
    assert _rel(got, orc.fbp_fan(orc.decode(p), a, y, cosine=True)) <= TOL
