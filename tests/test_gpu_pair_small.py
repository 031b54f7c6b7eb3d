"""The pair kernel on the caller's cell-major arrays (the fast forms it takes by itself): part half-tiles, rows of
fewer slices than parts, shared and unshared part sums, against the oracle; and the same bits whichever
warps took a row's parts."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import per_cell_err

pytestmark = pytest.mark.gpu


def _operator(L, K):
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    return geo.labels, geo.vals, geo.ic_map, workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=K), geo.n_q


@pytest.mark.parametrize("L,K,B", [(1, 1, 17), (2, 3, 18), (4, 5, 33), (4, 4, 47), (6, 6, 31), (12, 5, 20), (16, 3, 40)])
def test_pair_kernel_cell_major_vs_oracle(L, K, B, cuda_available, oracle_lib):
    import torch

    import cf_b200

    args = _operator(L, K)
    rng = np.random.default_rng(L)
    f, v, q0 = (rng.standard_normal((B, K, args[4])) * w for w in (1.0, 1.0, 1e-2))
    cm = lambda a: np.asfortranarray(a.transpose(2, 1, 0))  # noqa: E731
    ref, jref = np.zeros((args[4], K, B), order="F"), np.zeros((args[4], K, B), order="F")
    oracle_lib.af_batch(ref, cm(f), *args, K)
    oracle_lib.jv_batch(jref, cm(f), cm(v), *args, K)
    op = cf_b200.CollisionOperator(*args, K)
    ft, vt = torch.from_numpy(f).cuda(), torch.from_numpy(v).cuda()
    for form in ("af", "af_sym"):
        out = op.q(ft, out=torch.from_numpy(q0.copy()).cuda(), form=form).cpu().numpy() - q0
        assert per_cell_err(out, ref.transpose(2, 1, 0)) <= 1e-12, form
    for folded in (False, True):
        out = op.jv(ft, vt, folded=folded).cpu().numpy()
        assert per_cell_err(out, jref.transpose(2, 1, 0)) <= 1e-12, folded
    op.close()


@pytest.mark.parametrize("L,K,form", [(4, 5, "af"), (4, 5, "af_sym"), (6, 6, "af"), (3, 4, "af")])
def test_small_and_large_batches_give_the_same_bits(L, K, form, cuda_available):
    """A batch of fewer half-tiles than SMs shares out the parts of a row; a larger one does not; the tiled
    entries of the explicit pair path are the same routine."""
    import torch

    import cf_b200

    args = _operator(L, K)
    op = cf_b200.CollisionOperator(*args, K)
    f = torch.from_numpy(np.random.default_rng(5).standard_normal((5000, K, args[4]))).cuda()
    large = op.q(f, form=form)
    for B in (17, 100, 640):
        assert torch.equal(op.q(f[:B].contiguous(), form=form), large[:B])
    op.set_kernel_path("pair")
    assert torch.equal(op.q(f, form=form), large)
    op.close()
