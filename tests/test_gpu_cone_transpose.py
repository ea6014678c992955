"""The cone-beam projector's segment counts, and the FDK adjoint's lanes-along-z transpose:
row steps that repeat, advance by one and jump over detector rows, a single row, and both splits of a view over blocks, against the FP64 oracle
(relative L2 <= 1e-4, as the other cone-beam operators)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import rel_l2
from fanbeamctrecon_tensorflowop_gb300.ops import ConePlan
import geometries as G

pytestmark = pytest.mark.gpu

# rows, slices, row and slice pitch (mm): the row step per slice is about 1.75 dz / drow
SHAPES = [
    (1, 9, 4.0, 1.0),    # one detector row: both clamps fall on it
    (2, 17, 2.0, 1.0),   # no row between the edge rows
    (12, 33, 3.0, 1.0),  # steps of half a row: slices that share both rows
    (15, 16, 1.7, 1.0),  # steps of about one row
    (40, 7, 1.0, 3.0),   # jumps over four rows
]


@pytest.mark.parametrize("views", [76, 160])
@pytest.mark.parametrize("rows, nz, drow, dz", SHAPES)
def test_fdk_adjoint_row_steps(cuda, orc, rows, nz, drow, dz, views):
    """76 views: a lone volume's views are split in two, those of a pair are not; 160 views: both
    are.  A volume of the pair gives the bits that it gives alone."""
    p, a, nr, nz = G.cone_small(n=23, views=views, cols=41, n_rows=rows, nz=nz, pixel=7.0,
                                dz=dz, drow=drow)
    plan = ConePlan(p, a, nr, nz, device=cuda)
    g = orc.decode(p)
    x = np.random.default_rng(rows).uniform(-0.3, 1.0, (2, nz, g.ny, g.nx)).astype(np.float32)
    xt = torch.from_numpy(x).to(cuda)
    got = plan.fdk_adjoint(xt)
    ref = orc.fdk_cone_adjoint(g, nr, nz, a, x)
    assert rel_l2(got.double().cpu().numpy(), ref) <= 1e-4
    assert torch.equal(plan.fdk_adjoint(xt[1:])[0], got[1])


@pytest.mark.parametrize("rows", [1, 32])
@pytest.mark.parametrize("n", [3, 8, 33])
def test_cone_fp_segment_counts(cuda, orc, n, rows):
    """Cone projections whose chunks hold few, odd and full numbers of in-plane segments (the
    projector takes them two at a time, then the last one alone)."""
    p, a, nr, nz = G.cone_small(n=n, views=19, cols=37, n_rows=rows, nz=5, pixel=180.0 / n,
                                dz=4.0, drow=60.0 / rows)
    plan = ConePlan(p, a, nr, nz, device=cuda)
    g = orc.decode(p)
    x = np.random.default_rng(n).uniform(0.0, 1.0, (1, nz, g.ny, g.nx)).astype(np.float32)
    got = plan.fp_cone(torch.from_numpy(x).to(cuda))
    assert rel_l2(got.double().cpu().numpy(), orc.cone_fp(g, nr, nz, a, x)) <= 1e-4


@pytest.mark.parametrize("rows", [2, 8, 9, 16, 17, 24, 25, 33, 48, 49])
def test_cone_fp_row_groups(cuda, orc, rows):
    """Row counts on either side of every split of a warp's lanes into groups; a volume of a pair
    gives the bits that it gives alone."""
    p, a, nr, nz = G.cone_small(n=21, views=17, cols=29, n_rows=rows, nz=6, pixel=8.0, dz=4.0,
                                drow=70.0 / rows)
    plan = ConePlan(p, a, nr, nz, device=cuda)
    g = orc.decode(p)
    x = np.random.default_rng(rows).uniform(0.0, 1.0, (2, nz, g.ny, g.nx)).astype(np.float32)
    xt = torch.from_numpy(x).to(cuda)
    got = plan.fp_cone(xt)
    assert rel_l2(got.double().cpu().numpy(), orc.cone_fp(g, nr, nz, a, x)) <= 1e-4
    assert torch.equal(plan.fp_cone(xt[1:])[0], got[1])
