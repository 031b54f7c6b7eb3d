"""The pair kernel's share-out of items: stretches over parts of several half-tiles, with whole items, items shared by parts
and the routes they run on (cell-major Q and J.v, the tiled exact and FP32 forms), from one half-tile to several per CTA.

A row of a cell is summed in the same parts in the same order wherever the cuts fall, so a cell's result does not depend on
the batch it is in: bit for bit, and against the oracle at the tolerances of the forms.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import per_cell_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,K", [(0, 1), (2, 3), (5, 5), (8, 6), (13, 4), (15, 5)])
def test_results_do_not_depend_on_the_cuts(L, K, cuda_available, oracle_lib):
    import torch

    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=L)
    args = (geo.labels, geo.vals, geo.ic_map, R, geo.n_q, K)
    n = 600 if L > 8 else 5000
    cells = workloads.maxwellian_cells(K, L, n, seed=K)
    few = np.asfortranarray(cells[:30].transpose(2, 1, 0))
    ref, jref = np.zeros_like(few, order="F"), np.zeros_like(few, order="F")
    oracle_lib.af_batch(ref, few, *args)
    oracle_lib.jv_batch(jref, few, np.asfortranarray(cells[::-1][:30].transpose(2, 1, 0)), *args)
    op = cf_b200.CollisionOperator(*args)
    op.set_kernel_path("pair")
    f, v = torch.from_numpy(cells).cuda(), torch.from_numpy(cells[::-1].copy()).cuda()
    runs = {"af": (lambda m: op.q(f[:m].contiguous(), form="af"), ref, 1e-12),
            "jv": (lambda m: op.jv(f[:m].contiguous(), v[:m].contiguous()), jref, 1e-12),
            "exact": (lambda m: op.q(f[:m].contiguous(), form="af_exact"), ref, 0.0)}
    if K in (4, 6):
        runs["f32"] = (lambda m: op.q(f[:m].contiguous(), form="af_f32"), ref, 1e-5)
    if L == 15:
        del runs["jv"]  # f and v of 16 cells do not fit
    for name, (run, want, tol) in runs.items():
        whole = run(n)
        assert per_cell_err(whole[:30].cpu().numpy(), want.transpose(2, 1, 0)) <= tol, name
        for m in (17, 90, 333, 1185, 2370):
            if m < n:
                assert torch.equal(run(m), whole[:m]), (name, m)
    op.close()
