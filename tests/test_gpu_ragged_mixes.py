"""Ragged steps of mixes other than 40, 30, 20, 10 %: whichever way the work table cuts the half-tiles (by a CTA's share or the
last ones), every bucket equals its plan's tile kernel bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("buckets,counts", [(((8, 8),), (3000,)), (((8, 8),), (8000,)), (((2, 4), (6, 6)), (4000, 4000)),
                                            (((4, 4), (6, 6), (8, 6)), (2000, 2000, 4000)), (((2, 2), (7, 6)), (9000, 40))])
@pytest.mark.parametrize("tail_split", [0, 4, 16])
def test_every_mix_equals_the_plans(buckets, counts, tail_split, cuda_available):
    import torch

    import cf_b200
    from cf_b200 import geometry, ragged, workloads
    from oracle import rtensor

    ops, fs = [], []
    for (L, K), n in zip(buckets, counts):
        geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
        R = workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=L)
        ops.append(cf_b200.CollisionOperator(geo.labels, geo.vals, geo.ic_map, R, geo.n_q, K))
        ops[-1].set_kernel_path("tile")
        fs.append(torch.from_numpy(np.random.default_rng(L).standard_normal((n, K, geo.n_q))).cuda())
    qs = [torch.full_like(f, 1e-3) for f in fs]
    rb = ragged.RaggedBatch(ops, list(counts), ["af_sym"] * len(ops), tail_split=tail_split, family="tile")
    rb.q_graph(fs, qs)
    for op, f, q in zip(ops, fs, qs):
        assert torch.equal(q, op.q(f, out=torch.full_like(f, 1e-3), form="af_sym"))
    rb.close()
    for op in ops:
        op.close()
