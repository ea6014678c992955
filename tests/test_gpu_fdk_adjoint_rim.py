"""The FDK adjoint with the source on the FOV's rim, one ulp outside: the FP32 distance U of a
pixel beside the source is negative, and the pixel's detector rows run backwards from the last row.
Its additions stay in the accumulators (the last column, an odd number of rows); the results mean
nothing there (1 / U^2 bounds the fixed point), so they are only finite."""
from __future__ import annotations

import numpy as np
import pytest

from fanbeamctrecon_tensorflowop_gb300.geometry import fan_param16

f32 = np.float32


def _geometry():
    p = fan_param16(sdd=220.0, sid=float(np.nextafter(f32(100), f32(200))), n_views=1, n_cols=4,
                    n=31387, ny=6, pixel_mm=1.0, dcol_rad=0.8, det_bottom=-20.0, drow=8.0, dz=5.0)
    p[7] = 100.0
    return p, np.array([0.16744612], f32)


def test_the_pixel_lies_behind_the_source():
    p, a = _geometry()
    nx, ny, rfov = int(p[5]), int(p[6]), f32(p[7])

    def centre(n, i):
        d = f32(2) * rfov / f32(n)
        return np.float64(f32(-0.5) * f32(n) * d) + np.float64(d) * (i + 0.5)

    y, x = centre(ny, 3), centre(nx, np.arange(nx))
    x = x[x * x + y * y <= 1e4].max()
    c, s = f32(-np.cos(np.float64(a[0]))), f32(-np.sin(np.float64(a[0])))
    inner = f32(np.float64(f32(y)) * np.float64(s) + np.float64(f32(p[1])))
    assert f32(np.float64(f32(x)) * np.float64(c) + np.float64(inner)) < 0


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [5, 8])
@pytest.mark.parametrize("nz", [8, 11])
def test_rows_running_backwards(cuda, rows, nz):
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import ConePlan
    p, a = _geometry()
    plan = ConePlan(p, a, rows, nz, device=cuda)
    vol = torch.rand((1, nz, 6, 31387), device=cuda)
    assert bool(torch.isfinite(plan.fdk_adjoint(vol)).all())
    torch.cuda.synchronize()
