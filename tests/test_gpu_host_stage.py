"""Batched host calls from pageable memory, direct and staged through the plan's pinned memory.

A plan's first calls copy directly, later ones through pinned memory with several threads; arrays that are pinned go
direct always.  The kernels are the same, so every call's result has to be the same bytes, Q on entry included.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALLS = 7  # more than the calls that go direct first


@pytest.mark.parametrize("L,K,B,form", [(6, 6, 3333, "af_sym"), (4, 5, 2590, "af"), (4, 4, 512, "af"), (5, 4, 2049, "rf"),
                                        (8, 8, 1031, "af_sym")])
def test_staged_calls_equal_direct_ones(L, K, B, form, cuda_available):
    import torch

    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=L)
    args = (geo.labels, geo.vals, geo.ic_map, R, geo.n_q, K)
    rng = np.random.default_rng(B)
    states = [np.asfortranarray(workloads.maxwellian_cells(K, L, B, seed=s).transpose(2, 1, 0)) for s in (1, 2)]
    q0 = np.asfortranarray(rng.standard_normal(states[0].shape) * 1e-3)
    want = []
    for f in states:  # pinned memory
        fp, qp = (torch.from_numpy(a.transpose(2, 1, 0).copy()).pin_memory().numpy().transpose(2, 1, 0) for a in (f, q0))
        cf_b200.contract_batched(qp, fp, *args, form=form)
        want.append(qp.copy(order="F"))
    for call in range(CALLS):  # each with new arrays, and the other state than the call before
        Q = q0.copy(order="F")
        n0 = cf_b200.launch_count()
        cf_b200.contract_batched(Q, states[call % 2].copy(order="F"), *args, form=form)
        launches = cf_b200.launch_count() - n0
        assert np.array_equal(Q, want[call % 2]), call
        if form == "af_sym" and K % 2 == 0 and call > 0:
            assert launches == 1, call


@pytest.mark.parametrize("exact", [0, 2])
def test_staged_jacobian_calls_equal_direct_ones(exact, cuda_available):
    import cf_b200
    from cf_b200 import geometry, mex, workloads
    from oracle import rtensor

    L, K, B = 4, 6, 2500
    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=L)
    f, v = (np.asfortranarray(workloads.maxwellian_cells(K, L, B, seed=s).transpose(2, 1, 0)) for s in (1, 2))
    want = None
    for call in range(CALLS):
        out = np.zeros_like(f, order="F")
        mex.collision_jacobian_apply_mex(out, f, v, geo.labels, geo.vals, geo.ic_map, R, geo.n_q, K, exact=exact)
        want = out if want is None else want
        assert np.array_equal(out, want), call


def test_an_operator_changed_in_place_is_seen_by_a_staged_call(cuda_available):
    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    L, K, B = 6, 6, 1500
    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = np.asfortranarray(workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=L))
    f = np.asfortranarray(workloads.maxwellian_cells(K, L, B, seed=3).transpose(2, 1, 0))
    q0 = np.asfortranarray(np.random.default_rng(4).standard_normal(f.shape) * 1e-3)

    def call(R_now):
        Q = q0.copy(order="F")
        cf_b200.contract_batched(Q, f, geo.labels, geo.vals, geo.ic_map, R_now, geo.n_q, K, form="af_sym")
        return Q

    for _ in range(CALLS):
        first = call(R)
    R *= 2.0  # the same address, other contents: guessed wrongly, noticed, contracted again
    assert np.array_equal(call(R), call(R.copy(order="F")))
    assert not np.array_equal(call(R), first)
