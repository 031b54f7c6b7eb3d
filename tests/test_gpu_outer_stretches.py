"""The outer-product kernels' share-out of rows: stretches that start and end inside units, within one unit, with more
CTAs than rows, and at operators below the sizes of the other tests.

Every row of every cell is summed by one team in one order, wherever the cuts fall, so a cell's result does not depend
on the batch it is in: bit for bit, and against the oracle at the FP64 tolerance.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import per_cell_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,K", [(1, 8), (3, 8), (6, 7), (8, 8)])
def test_results_do_not_depend_on_the_cuts(L, K, cuda_available, oracle_lib):
    import torch

    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=L)
    args = (geo.labels, geo.vals, geo.ic_map, R, geo.n_q, K)
    cells = workloads.maxwellian_cells(K, L, 2500, seed=K)
    ref = np.zeros((geo.n_q, K, 64), order="F")
    oracle_lib.af_batch(ref, np.asfortranarray(cells[:64].transpose(2, 1, 0)), *args)
    op = cf_b200.CollisionOperator(*args)
    f, v = torch.from_numpy(cells).cuda(), torch.from_numpy(cells[::-1].copy()).cuda()
    for form in ("af", "af_sym"):
        whole, jwhole = op.q(f, form=form), op.jv(f, v, folded=form == "af_sym")
        assert per_cell_err(whole[:64].cpu().numpy(), ref.transpose(2, 1, 0)) <= 1e-12
        for B in (9, 40, 290, 593, 1184, 2369):  # 8-cell units: 2 .. 297, 16-cell units: 1 .. 149
            assert torch.equal(op.q(f[:B].contiguous(), form=form), whole[:B]), (form, B)
            if K == 8 or form == "af_sym":
                assert torch.equal(op.jv(f[:B].contiguous(), v[:B].contiguous(), folded=form == "af_sym"), jwhole[:B]), (form, B)
    op.close()
