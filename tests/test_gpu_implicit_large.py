"""The batched solve of more than 65535 tiles of cells, with enough of them done early that the others are gathered."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_solve_of_many_tiles(cuda_available):
    import torch

    import cf_b200
    from cf_b200 import _lib, geometry, workloads
    from oracle import rtensor

    K, restart, n_tiles, tol = 2, 8, 93000, 1e-11
    geo = geometry.sort_for_contraction(geometry.generate_geometry(1))
    op = cf_b200.CollisionOperator(geo.labels, geo.vals, geo.ic_map,
                                   workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=1), geo.n_q, K)
    gen = torch.Generator(device="cuda").manual_seed(3)
    f, b = (0.3 * torch.randn((n_tiles, geo.n_q, K, 32), dtype=torch.float64, device="cuda", generator=gen) for _ in range(2))
    b[66000:] = 0.0  # solved before the first step: 71 % of the cells stay, on 66000 tiles
    x = torch.zeros_like(b)
    n = n_tiles * 32
    lib, need = _lib.load(), C.c_size_t()
    _lib.check(lib.cf_gmres_workspace_size(op._h, n, restart, C.byref(need)))
    ws = torch.empty(need.value // 8 + 1, dtype=torch.float64, device="cuda")
    iters, rel = np.zeros(n, dtype=np.int32), np.zeros(n)
    _lib.check(lib.cf_gmres_solve_tiled(op._h, f.data_ptr(), 0.2, b.data_ptr(), x.data_ptr(), n, restart, 64, tol, None, 0,
                                        iters.ctypes.data, rel.ctypes.data, ws.data_ptr(), ws.numel() * 8,
                                        int(torch.cuda.current_stream().cuda_stream)))
    assert rel.max() <= tol  # the true residual, from a J.v of all cells
    assert iters[: 66000 * 32].min() >= 2 and iters[66000 * 32:].max() == 0
    assert not x[66000:].any()
    op.close()
    del f, b, x, ws
    torch.cuda.empty_cache()
