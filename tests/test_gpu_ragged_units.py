"""The ragged step's work table: half-tiles whole, several together, in quarters and in sixteenths, by their share of the work.

The routine is the plans' tile routine and a row is summed by one warp in one order however the half-tiles are cut, so
every bucket equals its plan's tile kernel bit for bit.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tail_split", [0, 4, 16])
@pytest.mark.parametrize("counts", [(300, 40, 33), (9000, 700, 100), (40000, 33, 1), (1, 0, 2000)])
def test_every_cut_equals_the_plans(counts, tail_split, cuda_available):
    import torch

    import cf_b200
    from cf_b200 import geometry, ragged, workloads
    from oracle import rtensor

    ops, fs = [], []
    for i, ((L, K), n) in enumerate(zip(((2, 4), (5, 6), (8, 8)), counts)):
        geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
        R = workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=L)
        ops.append(cf_b200.CollisionOperator(geo.labels, geo.vals, geo.ic_map, R, geo.n_q, K))
        ops[-1].set_kernel_path("tile")
        fs.append(torch.from_numpy(workloads.maxwellian_cells(K, L, max(n, 1), seed=i)[:n].copy()).cuda())
    qs = [torch.full_like(f, 1e-3) for f in fs]
    rb = ragged.RaggedBatch(ops, list(counts), ["af_sym"] * 3, tail_split=tail_split, family="tile")
    rb.q(fs, qs)
    for op, f, q in zip(ops, fs, qs):
        if f.shape[0] == 0:
            continue
        n = f.shape[0]  # up to 8 cells a plan takes the few-cell kernel: its tile kernel gets at least 16
        more = torch.cat([f, f[:1].expand(max(0, 16 - n), -1, -1)]).contiguous()
        want = op.q(more, out=torch.full_like(more, 1e-3), form="af_sym")[:n]
        assert np.array_equal(q.cpu().numpy(), want.cpu().numpy())
    rb.close()
    for op in ops:
        op.close()
