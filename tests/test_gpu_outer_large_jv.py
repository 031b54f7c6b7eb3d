"""The plain J.v at K = 7 on large batches: the pair kernel where its tiles fit, else the outer-product kernel, never the gather
kernel; against the gather kernel at the FP64 tolerance."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import per_cell_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,B,name", [(9, 1600, "pair"), (10, 1600, "outer_8"), (10, 1500, "outer_8")])
def test_large_plain_jv(L, B, name, cuda_available):
    import torch

    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    K = 7
    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    op = cf_b200.CollisionOperator(geo.labels, geo.vals, geo.ic_map,
                                   workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=K), geo.n_q, K)
    f, v = (torch.from_numpy(np.random.default_rng(s).standard_normal((B, K, geo.n_q))).cuda() for s in (L, B))
    out = op.jv(f, v)
    assert op.last_kernel() == name
    op.set_kernel_path("gather")
    assert per_cell_err(out.cpu().numpy(), op.jv(f, v).cpu().numpy()) <= 1e-12
    op.close()
