"""The pair kernel at the largest operators that its tile fits for, with as many warps as fit beside it: the automatic
order and the explicit path still take it there, against the gather kernel."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import per_cell_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,K,B,form,path", [(17, 5, 20, "af", "auto"), (17, 5, 12, "af", "pair"), (17, 5, 20, "af_sym", "auto"),
                                             (15, 6, 330, "af", "auto"), (15, 6, 12, "af", "pair"), (15, 6, 20, "af_sym", "pair"),
                                             (15, 5, 20, "af", "auto"), (14, 6, 20, "af", "auto"), (10, 5, 20, "jv", "pair")])
def test_pair_kernel_at_its_limits(L, K, B, form, path, cuda_available):
    import torch

    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=K)
    op = cf_b200.CollisionOperator(geo.labels, geo.vals, geo.ic_map, R, geo.n_q, K)
    f, v = (torch.from_numpy(np.random.default_rng(s).standard_normal((B, K, geo.n_q))).cuda() for s in (L, K))
    run = (lambda: op.jv(f, v)) if form == "jv" else (lambda: op.q(f, form=form))
    op.set_kernel_path(path)
    out = run()
    assert cf_b200._lib.PATH_NAMES[op.info()["last_path"]] == "pair"
    op.set_kernel_path("gather")
    ref = run()
    assert per_cell_err(out.cpu().numpy(), ref.cpu().numpy()) <= 1e-12  # as the FP64 fast forms elsewhere
    op.close()
