"""An operator's device arrays are one allocation: making, using and closing operators gives all device memory back."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,K", [(8, 7), (10, 8), (6, 5), (5, 12)])
def test_operators_give_their_memory_back(L, K, cuda_available):
    import torch

    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = np.asfortranarray(workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=L))
    f = torch.from_numpy(workloads.maxwellian_cells(K, L, 20, seed=K)).cuda()
    free, outs = [], []
    for _ in range(4):
        op = cf_b200.CollisionOperator(geo.labels, geo.vals, geo.ic_map, R, geo.n_q, K)
        assert op.info()["device_bytes"] >= 8 * R.size
        outs.append([op.q(f, form=form) for form in ("af", "af_sym")])
        torch.cuda.synchronize()
        op.close()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[-1] >= free[1]  # the first use of a kernel takes memory for its code
    for o in outs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(o, outs[0]))
