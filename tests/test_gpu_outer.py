"""The outer-product kernels (K = 7 and 8, Phi on the FP64 tensor cores) at the edges of their tiles, against the
oracle: both row widths (L <= 10, L <= 15), units of 16 and of 8 cells, part batches, rows of very few slices,
lists whose slices are longer than a ring stage, unsorted lists, and a cell that is not finite."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import per_cell_err

pytestmark = pytest.mark.gpu

TOL_FP64 = 1e-12  # as the FP64 fast forms elsewhere


def _hard_spheres(L, K, seed):
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=seed)
    return geo.labels, geo.vals, geo.ic_map, R, geo.n_q


def _random_list(n_q, K, n_t, n_g, seed):
    """Entries with no structure: long runs of one q2, repeated (t, q1) runs, rows without entries."""
    rng = np.random.default_rng(seed)
    lab = np.asfortranarray(np.stack([rng.integers(1, n_q, n_g), np.minimum(rng.integers(1, 2 * n_q, n_g), n_q),
                                      rng.integers(1, n_q + 1, n_g)], axis=1).astype(float))
    ic = rng.integers(1, n_t + 1, n_g).astype(float)
    o = np.lexsort((lab[:, 0], ic))
    o[: n_g // 2] = o[: n_g // 2][::-1]  # half of the list keeps no order that the sort gave
    R = np.asfortranarray(rng.standard_normal((K, K, K, n_t)))
    return np.asfortranarray(lab[o]), rng.standard_normal(n_g), ic[o], R, n_q


def _check(oracle_lib, args, K, B, forms, seed):
    import torch

    import cf_b200

    n_q = args[4]
    rng = np.random.default_rng(seed)
    f, v, q0 = (rng.standard_normal((B, K, n_q)) * w for w in (1.0, 1.0, 1e-2))
    cm = lambda a: np.asfortranarray(a.transpose(2, 1, 0))  # noqa: E731
    ref, jref = np.zeros((n_q, K, B), order="F"), np.zeros((n_q, K, B), order="F")
    oracle_lib.af_batch(ref, cm(f), *args, K)
    oracle_lib.jv_batch(jref, cm(f), cm(v), *args, K)
    op = cf_b200.CollisionOperator(*args, K)
    ft, vt = torch.from_numpy(f).cuda(), torch.from_numpy(v).cuda()
    for form in forms:
        out = op.q(ft, out=torch.from_numpy(q0.copy()).cuda(), form=form).cpu().numpy() - q0
        assert cf_b200._lib.PATH_NAMES[op.info()["last_path"]] in ("tile", "tile_quarter")
        assert per_cell_err(out, ref.transpose(2, 1, 0)) <= TOL_FP64, form
    for folded in ([False, True] if "af_sym" in forms else [False]):
        out = op.jv(ft, vt, folded=folded).cpu().numpy()
        assert per_cell_err(out, jref.transpose(2, 1, 0)) <= TOL_FP64, folded
    op.close()


@pytest.mark.parametrize("L,K,B", [(0, 8, 9), (1, 7, 17), (2, 8, 33), (5, 7, 23), (10, 7, 16), (10, 8, 41), (11, 8, 15),
                                   (14, 8, 12), (15, 7, 9)])
def test_outer_kernel_vs_oracle(L, K, B, cuda_available, oracle_lib):
    _check(oracle_lib, _hard_spheres(L, K, seed=L + K), K, B, ("af", "af_sym"), seed=B)


@pytest.mark.parametrize("n_q,K,n_t,n_g,B", [(4, 8, 2, 900, 20), (30, 7, 3, 4000, 11), (131, 8, 5, 3000, 18),
                                             (133, 8, 40, 3000, 10)])
def test_outer_kernel_on_lists_without_structure(n_q, K, n_t, n_g, B, cuda_available, oracle_lib):
    _check(oracle_lib, _random_list(n_q, K, n_t, n_g, seed=n_q), K, B, ("af",), seed=B)


def test_outer_kernel_keeps_a_non_finite_cell_to_itself(cuda_available):
    import torch

    import cf_b200

    args, K, B = _hard_spheres(6, 8, seed=1), 8, 40
    op = cf_b200.CollisionOperator(*args, K)
    f = torch.from_numpy(np.random.default_rng(2).standard_normal((B, K, args[4]))).cuda()
    ref = op.q(f, form="af_sym")
    g = f.clone()
    g[5, 3, 10], g[17, 0, 48] = float("nan"), float("inf")
    out = op.q(g, form="af_sym")
    others = [b for b in range(B) if b not in (5, 17)]
    assert torch.equal(out[others], ref[others])
    assert not torch.isfinite(out[5]).all() and not torch.isfinite(out[17]).all()
    # rows no entry of which touches the bad coefficient stay as they are
    lab = np.asarray(args[0]).astype(int) - 1
    touched = set(lab[(lab[:, 1] == 10) | (lab[:, 2] == 10), 0])
    clean = [q for q in range(args[4]) if q not in touched]
    if clean:
        assert torch.equal(out[5][:, clean], ref[5][:, clean])
    op.close()
