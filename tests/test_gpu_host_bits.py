"""Host calls of 512 cells up give the device entry points' bits, streamed or chunked, from pageable and pinned arrays."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,K,B,form", [(10, 8, 600, "af_sym"), (11, 8, 600, "af_sym"), (11, 8, 520, "af"),
                                        (5, 7, 700, "af_sym"), (6, 6, 900, "af_sym"), (6, 5, 900, "af")])
def test_host_call_gives_the_device_bits(L, K, B, form, cuda_available):
    import torch

    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=K)
    args = (geo.labels, geo.vals, geo.ic_map, R, geo.n_q, K)
    f = torch.from_numpy(np.random.default_rng(L).standard_normal((B, K, geo.n_q)))
    op = cf_b200.CollisionOperator(*args)
    ref = op.q(f.cuda(), form=form).cpu().numpy()
    for x in (f, f.pin_memory()):
        q = torch.zeros_like(x, pin_memory=x.is_pinned())
        cf_b200.contract_batched(q.numpy().transpose(2, 1, 0), x.numpy().transpose(2, 1, 0), *args, form=form)
        assert np.array_equal(q.numpy(), ref)
    op.close()
