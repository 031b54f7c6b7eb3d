"""The pinned memory that host calls from pageable arrays are staged through: bounded over all operators, counted, and given
back with them; a call without any copies directly."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operator(L, K, seed):
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    return geo.labels, geo.vals, geo.ic_map, workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=seed), geo.n_q, K


def test_pinned_memory_is_bounded_and_given_back(cuda_available):
    import cf_b200

    pinned = cf_b200._lib.load().cf_pinned_bytes

    def push_out():  # the cache of host calls' operators holds eight
        for seed in range(8):
            args = _operator(1, 2, 100 + seed)
            cf_b200.contract_batched(np.zeros((4, 2, 9), order="F"), np.ones((4, 2, 9), order="F"), *args)

    push_out()
    base = pinned()  # of operators that other code holds
    L, K, B = 6, 8, 14000  # Q and f: 88 MB a call
    f = np.asfortranarray(np.random.default_rng(1).standard_normal((49, K, B)))
    for seed in range(4):
        args = _operator(L, K, seed)
        outs = []
        for _ in range(6):
            q = np.zeros_like(f, order="F")
            cf_b200.contract_batched(q, f, *args, form="af_sym")
            outs.append(q)
        assert all(np.array_equal(q, outs[0]) for q in outs[1:])
        assert pinned() <= 256 << 20
        if seed == 0:
            assert pinned() - base >= 2 * f.nbytes  # the later calls were staged
    push_out()
    assert pinned() == base
