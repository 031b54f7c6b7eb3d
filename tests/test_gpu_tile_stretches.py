"""The tile kernel's share-out of rows: stretches over parts of several half-tiles, as many resident at a time as fit, from
batches of less than a half-tile to several per CTA, on the cell-major (Q) and the tiled route (J.v up to
L = 11 at K = 6, the exact form).

A row of a cell is summed by one warp in one order wherever the cuts fall, so a cell's result does not depend on the
batch it is in: bit for bit, and against the oracle at the FP64 tolerance.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import per_cell_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,K", [(0, 2), (2, 4), (7, 2), (6, 6), (13, 6)])
def test_results_do_not_depend_on_the_cuts(L, K, cuda_available, oracle_lib):
    import torch

    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=L)
    args = (geo.labels, geo.vals, geo.ic_map, R, geo.n_q, K)
    n = 900 if L == 13 else 9700
    cells = workloads.maxwellian_cells(K, L, n, seed=K)
    few = np.asfortranarray(cells[:40].transpose(2, 1, 0))
    ref, jref = np.zeros_like(few, order="F"), np.zeros_like(few, order="F")
    oracle_lib.af_batch(ref, few, *args)
    oracle_lib.jv_batch(jref, few, np.asfortranarray(cells[::-1][:40].transpose(2, 1, 0)), *args)
    op = cf_b200.CollisionOperator(*args)
    f, v = torch.from_numpy(cells).cuda(), torch.from_numpy(cells[::-1].copy()).cuda()

    def run(m):
        return op.q(f[:m].contiguous(), form="af_sym"), op.jv(f[:m].contiguous(), v[:m].contiguous(), folded=True)

    q, j = run(n)
    op.q(f, form="af_sym")
    assert cf_b200._lib.PATH_NAMES[op.info()["last_path"]] == "tile"
    assert per_cell_err(q[:40].cpu().numpy(), ref.transpose(2, 1, 0)) <= 1e-12
    assert per_cell_err(j[:40].cpu().numpy(), jref.transpose(2, 1, 0)) <= 1e-12
    for m in (17, 250, 700, 2369, 4737):
        if m < n:
            qm, jm = run(m)
            assert torch.equal(qm, q[:m]) and torch.equal(jm, j[:m]), m
    op.set_kernel_path("tile")
    exact = op.q(f, form="af_exact")
    for m in (17, 700):
        assert torch.equal(op.q(f[:m].contiguous(), form="af_exact"), exact[:m]), m
    op.close()
