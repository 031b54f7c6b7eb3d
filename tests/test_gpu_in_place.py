"""Device calls whose output is, or overlaps, an input: the inputs count as they were before the call, on every route
that reads them and adds to Q in the caller's arrays (and on those that pack them first)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operator(L, K):
    import cf_b200
    from cf_b200 import geometry, workloads
    from oracle import rtensor

    geo = geometry.sort_for_contraction(geometry.generate_geometry(L))
    R = workloads.synthetic_R(rtensor.l_triplets_of(geo), K, seed=K)
    return cf_b200.CollisionOperator(geo.labels, geo.vals, geo.ic_map, R, geo.n_q, K)


def _cells(op, B, seed):
    import torch

    return torch.from_numpy(np.random.default_rng(seed).standard_normal((B, op.K, op.N_Q))).cuda()


# outer-product, pair, tile, few-cell, gather, l-block and exact row routes; more half-tiles than fit beside each other
@pytest.mark.parametrize("L,K,B,form,path", [(8, 8, 700, "af", "auto"), (8, 8, 700, "af_sym", "auto"),
                                             (5, 7, 300, "af_sym", "auto"), (8, 5, 900, "af", "auto"),
                                             (8, 6, 700, "af", "auto"), (6, 6, 900, "af_sym", "auto"),
                                             (6, 8, 700, "af", "pair"), (6, 5, 5, "af", "auto"),
                                             (4, 8, 3, "rf", "auto"), (4, 9, 60, "af", "auto"), (4, 12, 90, "af", "auto"),
                                             (3, 9, 40, "af_exact", "auto"), (4, 8, 90, "af", "band"),
                                             (6, 8, 90, "af_sym_i8", "auto"), (6, 8, 90, "rf_dense", "auto"),
                                             (6, 4, 300, "af_sym_f32", "auto"), (6, 12, 90, "af_sym_bf16", "auto")])
def test_q_in_place(L, K, B, form, path, cuda_available):
    import torch

    op = _operator(L, K)
    op.set_kernel_path(path)
    f = _cells(op, B, seed=L)
    ref = op.q(f, out=f.clone(), form=form)
    assert torch.equal(op.q(f, out=f, form=form), ref)
    # one cell further on: every cell but the first is also an output
    buf = _cells(op, B + 1, seed=L + 1)
    ref = op.q(buf[1:].clone(), out=buf[:-1].clone(), form=form)
    assert torch.equal(op.q(buf[1:], out=buf[:-1], form=form), ref)
    op.close()


@pytest.mark.parametrize("L,K,B,mode", [(8, 8, 700, {}), (8, 8, 700, {"folded": True}), (8, 5, 900, {}),
                                        (6, 6, 900, {"folded": True}), (5, 7, 300, {"folded": True}), (5, 3, 9, {}),
                                        (3, 9, 40, {"exact": True}), (4, 12, 90, {}), (6, 4, 300, {"fp32": True})])
@pytest.mark.parametrize("which", ["f", "v"])
def test_jv_in_place(L, K, B, mode, which, cuda_available):
    import torch

    op = _operator(L, K)
    f, v = _cells(op, B, seed=L), _cells(op, B, seed=L + 9)
    ref = op.jv(f, v, out=(f if which == "f" else v).clone(), **mode)
    out = f if which == "f" else v
    assert torch.equal(op.jv(f, v, out=out, **mode), ref)
    op.close()


def test_a_workspace_that_cannot_hold_the_copy_is_refused(cuda_available):
    """An overlapping call never runs on inputs that change under it."""
    import torch

    import cf_b200

    op = _operator(4, 4)
    f = _cells(op, 5, seed=1)
    before = f.clone()
    with pytest.raises(cf_b200.CFError) as e:
        op.q(f, out=f, workspace=torch.empty(8, dtype=torch.float64, device="cuda"))
    assert e.value.status == cf_b200._lib.CF_EINVAL and torch.equal(f, before)
    op.close()
