"""The l-block kernels' run records: runs of one, two and more entries with the same q2 (a list with repeated entries
has longer runs than the selection rules give), and slices of more runs than a record buffer holds.

Tolerance: 1e-12 normwise per cell for FP64 and 1e-5 for the FP32 forms against the oracle, as for the lists without
repeats; the split entries' G values add up to the original ones within rounding.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import per_cell_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,L,B,copies", [(12, 3, 17, 3), (12, 8, 9, 1), (12, 9, 33, 2), (8, 5, 23, 5), (8, 11, 12, 1)])
def test_lblock_runs_vs_oracle(K, L, B, copies, cuda_available, oracle_lib):
    import torch

    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = np.asfortranarray(workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=L))
    w = np.random.default_rng(K).dirichlet(np.ones(copies), size=geo.vals.size)  # each entry's G in `copies` shares
    labels = np.asfortranarray(np.repeat(geo.labels, copies, axis=0))
    vals, ic = (np.repeat(np.ravel(geo.vals), copies) * w.ravel(), np.repeat(np.ravel(geo.ic_map), copies))
    cells = workloads.maxwellian_cells(K, L, B, seed=B)
    f = np.asfortranarray(cells.transpose(2, 1, 0))
    ref = np.zeros_like(f, order="F")
    oracle_lib.af_batch(ref, f, labels, vals, ic, R, geo.n_q, K)
    ref = np.ascontiguousarray(ref.transpose(2, 1, 0))
    op = cf_b200.CollisionOperator(labels, vals, ic, R, geo.n_q, K)
    op.set_kernel_path("lblock")
    ft = torch.from_numpy(cells).cuda()
    for form, tol in (("af", 1e-12), ("af_f32", 1e-5), ("af_sym", 1e-12), ("af_sym_f32", 1e-5)):
        if "sym" in form and copies > 1:
            continue  # the shares of (q2, q3) and (q3, q2) differ, so this list does not fold
        q = [torch.zeros_like(ft) for _ in range(2)]
        for out in q:
            op.q(ft, out=out, form=form)
        assert op.info()["last_path"] == 14, form
        assert torch.equal(q[0], q[1]), form
        assert per_cell_err(q[0].cpu().numpy(), ref) <= tol, form
    op.close()
