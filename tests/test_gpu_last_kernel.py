"""Which kernel a call ran on, by its own name: the outer-product kernel is told from the tile kernels whose codes it
reports in last_path."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,K,B,mode,path,name,code", [
    (4, 8, 40, "af_sym", "auto", "outer", "tile"), (4, 8, 40, "af", "auto", "outer", "tile"),
    (4, 7, 40, "jv", "auto", "outer_8", "tile_quarter"), (11, 8, 20, "af_sym", "auto", "outer_8", "tile_quarter"),
    (10, 8, 20, "jv_folded", "auto", "outer_8", "tile_quarter"), (4, 8, 40, "af_sym", "tile", "tile", "tile"),
    (4, 6, 40, "af_sym", "auto", "tile", "tile"), (4, 5, 40, "af", "auto", "pair", "pair"),
    (4, 7, 9000, "jv", "auto", "pair", "pair"), (4, 8, 5, "af", "auto", "few", "few")])
def test_last_kernel(L, K, B, mode, path, name, code, cuda_available):
    import torch

    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    op = cf_b200.CollisionOperator(geo.labels, geo.vals, geo.ic_map,
                                   workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=K), geo.n_q, K)
    assert op.last_kernel() == "none"
    op.set_kernel_path(path)
    f = torch.from_numpy(np.random.default_rng(L).standard_normal((B, K, geo.n_q))).cuda()
    if mode.startswith("jv"):
        op.jv(f, f, folded=mode == "jv_folded")
    else:
        op.q(f, form=mode)
    assert op.last_kernel() == name
    assert cf_b200._lib.PATH_NAMES[op.info()["last_path"]] == code
    op.close()
