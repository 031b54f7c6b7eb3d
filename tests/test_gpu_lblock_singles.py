"""The FP64 l-block kernel's reads of run records: a run of two entries may have one q3 twice (each its own G), which is
read once as a run of one is.  Tolerance 1e-12 normwise per cell, as for the other lists."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import per_cell_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [8, 12])
@pytest.mark.parametrize("kind", ["ones", "same_q3", "mixed"])
def test_lblock_runs_of_one_q3(K, kind, cuda_available, oracle_lib):
    import torch

    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(5))
    R = np.asfortranarray(workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=K))
    labels, vals, ic = np.asarray(geo.labels), np.ravel(geo.vals), np.ravel(geo.ic_map)
    if kind != "mixed":  # the first entry of each (t, q1, q2)
        keep = np.unique(np.column_stack([ic, labels[:, 0], labels[:, 1]]), axis=0, return_index=True)[1]
        keep.sort()
        labels, vals, ic = labels[keep], vals[keep], ic[keep]
    times = np.ones(vals.size, int) if kind == "ones" else np.full(vals.size, 2) if kind == "same_q3" else 1 + np.arange(vals.size) % 3
    labels, vals, ic = (np.repeat(x, times, axis=0) for x in (labels, vals, ic))
    vals = vals * np.random.default_rng(K).uniform(0.2, 1.0, vals.size)
    labels = np.asfortranarray(labels)
    cells = workloads.maxwellian_cells(K, 5, 19, seed=K)
    f = np.asfortranarray(cells.transpose(2, 1, 0))
    ref = np.zeros_like(f, order="F")
    oracle_lib.af_batch(ref, f, labels, vals, ic, R, geo.n_q, K)
    op = cf_b200.CollisionOperator(labels, vals, ic, R, geo.n_q, K)
    op.set_kernel_path("lblock")
    q = op.q(torch.from_numpy(cells).cuda(), form="af")
    assert op.last_kernel() == "lblock"
    assert per_cell_err(q.cpu().numpy(), np.ascontiguousarray(ref.transpose(2, 1, 0))) <= 1e-12
    op.close()
