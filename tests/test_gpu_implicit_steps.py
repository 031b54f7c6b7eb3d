"""The vector kernels of the batched GMRES at the edges of their tiles, against a dense solve: bases past 16 vectors
(the two-sweep form), restarts, cells that finish at different steps (J.v on the gathered active cells), one to a
few cells, per-cell, shared and no preconditioner."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _device_memory_given_back():
    yield
    import torch

    torch.cuda.empty_cache()  # tests that watch the free memory find none of this file's blocks


@pytest.mark.parametrize("L,K,B,restart,precond", [(2, 3, 1, 30, "none"), (2, 3, 3, 5, "shared"), (3, 5, 45, 63, "none"),
                                                   (2, 8, 33, 4, "none"), (3, 4, 70, 30, "cell"), (3, 7, 17, 20, "shared")])
def test_gmres_vs_dense_solve(L, K, B, restart, precond, cuda_available):
    """Tolerance: GMRES stops at |r| <= 1e-12 |b|; with I - dt J within a factor of about 100 of the identity the
    solution is within 1e-10 of the dense one."""
    import torch

    import cf_b200
    from cf_b200 import geometry, implicit, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=L * K)
    op = cf_b200.CollisionOperator(geo.labels, geo.vals, geo.ic_map, R, geo.n_q, K)
    rng = np.random.default_rng(B)
    M = geo.n_q * K
    # the cells' Jacobians differ in size by up to 100, so they need very different numbers of steps
    f = torch.from_numpy(rng.standard_normal((B, K, geo.n_q)) * 10.0 ** rng.uniform(-2, 0, (B, 1, 1))).cuda()
    b = torch.from_numpy(rng.standard_normal((B, K, geo.n_q))).cuda()
    eye = torch.eye(M, dtype=torch.float64, device="cuda").view(M, K, geo.n_q)
    J = torch.stack([op.jv(f[i:i + 1].expand(M, -1, -1).contiguous(), eye).view(M, M).T.cpu() for i in range(B)])
    dt = 0.5 / float(torch.linalg.matrix_norm(J, ord=2).max())
    A = torch.eye(M, dtype=torch.float64) - dt * J
    ref = torch.linalg.solve(A, b.cpu().reshape(B, M, 1)).view_as(b).cuda()
    P = None
    if precond != "none":
        P = rng.standard_normal(((B,) if precond == "cell" else ()) + (geo.n_q, K, K)) * 0.02 + np.eye(K)
    x, iters, rel = implicit.gmres_solve(op, f, b, dt, restart=restart, tol=1e-12, precond=P)
    assert rel.max() <= 1e-12 and iters.min() >= 1
    assert float((x - ref).abs().max() / ref.abs().max()) <= 1e-10
    # a second solve from the solution needs no step and leaves it alone
    x2, iters2, _ = implicit.gmres_solve(op, f, b, dt, x0=x, restart=restart, tol=1e-11, precond=P)
    assert iters2.max() == 0 and torch.equal(x2, x)
    op.close()
