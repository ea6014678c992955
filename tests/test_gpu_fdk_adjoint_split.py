"""The FDK adjoint on either side of the rule that gives a view one block or a cluster of two
(pixels and slices against the accumulators that each block clears and writes): FP64 oracle at the
operators' 1e-4, and a volume of a pair, whose views are split otherwise, gives the bits it gives
alone."""
from __future__ import annotations

import numpy as np
import pytest

import geometries as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 17, 18, 30])
@pytest.mark.parametrize("views, rows", [(60, 12), (160, 12), (160, 33)])
def test_fdk_adjoint_one_or_two_blocks_per_view(cuda, orc, n, views, rows):
    import torch
    from fanbeamctrecon_tensorflowop_gb300.ops import ConePlan
    p, a, nr, nz = G.cone_small(n=n, views=views, cols=41, n_rows=rows, nz=13, pixel=160.0 / n,
                                dz=2.0, drow=36.0 / rows)
    plan = ConePlan(p, a, nr, nz, device=cuda)
    g = orc.decode(p)
    x = np.random.default_rng(n).uniform(-0.3, 1.0, (2, nz, g.ny, g.nx)).astype(np.float32)
    xt = torch.from_numpy(x).to(cuda)
    got = plan.fdk_adjoint(xt)
    ref = orc.fdk_cone_adjoint(g, nr, nz, a, x)
    assert np.linalg.norm(got.double().cpu().numpy() - ref) <= 1e-4 * np.linalg.norm(ref)
    assert torch.equal(plan.fdk_adjoint(xt[1:])[0], got[1])
