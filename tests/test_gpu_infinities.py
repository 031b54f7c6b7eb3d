"""An infinite coefficient (or one that overflows FP32) of an operator and cells without negative numbers: the rows it
enters are infinite, not NaN, and the others keep their bits -- whatever the kernels pad their lists with."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,K,B,path,kind,mode", [
    (3, 8, 20, "auto", "q", "af"), (3, 8, 20, "auto", "q", "af_sym"), (6, 7, 33, "auto", "q", "af"),
    (10, 8, 17, "auto", "q", "af_sym"), (11, 8, 18, "auto", "q", "af"), (4, 8, 20, "auto", "jv", True),
    (5, 7, 20, "auto", "jv", False), (4, 8, 20, "lblock", "q", "af"), (5, 12, 20, "auto", "q", "af_sym"),
    (5, 12, 20, "auto", "q", "af_sym_f32"), (4, 5, 20, "auto", "q", "af"), (4, 6, 20, "auto", "q", "af_sym")])
def test_infinite_coefficient(L, K, B, path, kind, mode, cuda_available):
    import torch

    import cf_b200
    from cf_b200 import geometry

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    rng = np.random.default_rng(L)
    R = np.asfortranarray(rng.uniform(0.5, 1.0, (K, K, K, int(np.max(geo.ic_map)))))
    op = cf_b200.CollisionOperator(geo.labels, np.abs(geo.vals), geo.ic_map, R, geo.n_q, K)
    op.set_kernel_path(path)
    f, v = (torch.from_numpy(rng.uniform(0.5, 1.0, (B, K, geo.n_q))).cuda() for _ in range(2))
    run = (lambda x: op.q(x, form=mode)) if kind == "q" else (lambda x: op.jv(x, v, folded=mode))
    ref = run(f)
    assert torch.isfinite(ref).all()
    lab = np.asarray(geo.labels).astype(int) - 1
    for q in range(0, geo.n_q, max(1, geo.n_q // 9)):
        g = f.clone()
        g[1, K - 1, q] = 1e200 if mode == "af_sym_f32" else float("inf")
        out = run(g)
        touched = sorted(set(lab[(lab[:, 1] == q) | (lab[:, 2] == q), 0]))
        rest = sorted(set(range(geo.n_q)) - set(touched))
        assert torch.equal(out[1][:, touched], torch.full_like(out[1][:, touched], float("inf"))), q
        assert torch.equal(out[1][:, rest], ref[1][:, rest]), q
        others = [b for b in range(B) if b != 1]
        assert torch.equal(out[others], ref[others])
    op.close()
