"""The GPU quadrature of R against a plain numpy restatement, at the edges of its kernels' tiles: K of one
and two MMA column tiles, inner points that do and do not fill the rounds of 4, gain tables with sine harmonics
(azimuths not merged) and without (merged), a dropped pair, and a patch without nodes."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _numpy_sumfac(args):
    """The raw quadrature from the 26 inputs, item by item."""
    from cf_b200 import basis

    K_max, NL, NQ, alpha = int(args[0]), int(args[1]), int(args[2]), float(args[3])
    (x, wx, u1, wu1, t1, wt1, y2, wy2, t2, wt2, chi, wchi, eps, weps) = [np.asarray(a).ravel() for a in args[4:18]]
    rnorm, trip, qi, pl1, pg1, pl2, pg2 = args[18], args[20], args[21], args[22], args[23], args[24], args[25]
    K, L = K_max + 1, int(round(math.sqrt(NQ))) - 1
    l1, l2, l3 = (np.asarray(trip)[:, j].astype(int) for j in range(3))
    n, e = np.meshgrid(np.arange(chi.size), np.arange(eps.size), indexing="ij")
    cc, W = chi[n].ravel(), (wchi[n] * weps[e]).ravel()
    sc = np.sqrt(np.maximum(1 - cc * cc, 0))
    up = np.stack([sc * np.cos(eps[e]).ravel(), sc * np.sin(eps[e]).ravel(), cc])

    def radial(v):  # [K, L+1, ...]
        v = np.asarray(v, dtype=float)
        return np.array([[rnorm[k, l] * basis.laguerre(k, l + 0.5, v * v) * v**l for l in range(L + 1)] for k in range(K)])

    def gain(vo, vz, cb, sb, pg):  # pg [NQ, NL] -> [K, NL]
        U, u = np.array([vo * sb, 0, vz + vo * cb]), np.array([-vo * sb, vz - vo * cb])
        um = math.sqrt(max(u @ u, 1e-15))
        zx, zz = u / um
        r = np.stack([up[0] * zz + up[2] * zx, up[1], -up[0] * zx + up[2] * zz])
        v = 0.5 * (U[:, None] + um * r)
        vm = np.sqrt(np.maximum((v * v).sum(0), 1e-15))
        Y = basis.real_sh(L, np.arccos(np.clip(v[2] / vm, -1, 1)), np.arctan2(v[1], v[0]))  # [points, NQ]
        return np.einsum("p,pc,kcp->kc", W, Y @ pg, radial(vm)[:, l1])

    valid = np.zeros((NQ, NL))
    for c in range(NL):
        for q in np.asarray(qi)[:, c].astype(int):
            if q == -1:
                break
            valid[q - 1, c] = 1.0
    R = np.zeros((K, K, K, NL))

    def add(vL, vS, Jo, net1, net2):
        rL, rS = radial(vL), radial(vS)
        R[...] += Jo * (np.einsum("ac,bc,dc->abdc", net1, rL[:, l2], rS[:, l3])
                        + np.einsum("ac,bc,dc->abdc", net2, rS[:, l2], rL[:, l3]))

    def nets(vL, vS, cb, umag, xi, Jt, pg, pl):
        sb = math.sqrt(max(1 - cb * cb, 1e-15))
        B = (umag * math.sqrt(2)) ** alpha / xi ** (alpha / 2)
        lw = B * 4 * math.pi * Jt * pl
        return (B * Jt * gain(vS, vL, cb, sb, pg * valid) - lw * radial(vL)[:, l1],
                B * Jt * gain(vL, vS, cb, sb, pg * valid) - lw * radial(vS)[:, l1])

    for i, xi in enumerate(x):
        a = math.sqrt(xi / 2)
        for o, u in enumerate(u1):
            vL, vS = a * (1 + u), a * (1 - u)
            Jo = 0.5 * wx[i] * wu1[o] * u * math.exp(-xi * u * u) * (vL * vL * vS * vS)
            n1, n2 = np.zeros((K, NL)), np.zeros((K, NL))
            for j, t in enumerate(t1):
                um = math.sqrt(2 * xi) * u * math.sqrt(1 + (1 - u * u) * t * t)
                p, q = nets(vL, vS, 1 - 2 * (u * t) ** 2, um, xi, wt1[j] * 4 * u * t, pg1[j, o], pl1[j, o])
                n1 += p
                n2 += q
            add(vL, vS, Jo, n1, n2)
        for o, y in enumerate(y2):
            for j, t in enumerate(t2):
                u = y * t
                vL, vS = a * (1 + u), a * (1 - u)
                um = math.sqrt(2 * xi) * y * math.sqrt(t * t + 1 - y * y * t * t)
                Jt = wt2[j] * math.exp(-xi * u * u) * (vL * vL * vS * vS)
                p, q = nets(vL, vS, 1 - 2 * y * y, um, xi, Jt, pg2[o], pl2[o])
                add(vL, vS, 0.5 * wx[i] * wy2[o] * 4 * y * y, p, q)
    return R


def _thin(args, n_x, n_chi, n_eps, n_t1=3, n_t2=5):
    """Fewer nodes of every rule (the quadrature need not be accurate, only the same)."""
    a = list(args)
    col = lambda v, n: np.asarray(v).reshape(-1, 1)[:n]  # noqa: E731
    for j, n in ((4, n_x), (5, n_x), (6, 4), (7, 4), (8, n_t1), (9, n_t1), (10, 3), (11, 3), (12, n_t2), (13, n_t2),
                 (14, n_chi), (15, n_chi)):
        a[j] = col(a[j], n)
    a[16] = 2 * math.pi * np.arange(n_eps).reshape(-1, 1) / max(n_eps, 1)
    a[17] = np.full((n_eps, 1), 2 * math.pi / max(n_eps, 1))
    a[22], a[23] = np.asfortranarray(a[22][:n_t1, :4]), np.asfortranarray(a[23][:n_t1, :4])
    a[24], a[25] = np.asfortranarray(a[24][:3]), np.asfortranarray(a[25][:3])
    return a


@pytest.mark.parametrize("K_max,L,n_chi,n_eps,sine,n_t1,n_t2", [
    (0, 2, 1, 1, False, 3, 5), (0, 3, 3, 3, False, 3, 5), (2, 3, 5, 7, False, 3, 66), (7, 2, 4, 4, False, 3, 5),
    (8, 3, 5, 9, True, 3, 5), (11, 9, 9, 16, False, 2, 2), (4, 8, 9, 15, True, 2, 2), (3, 2, 2, 5, False, 0, 5),
    (3, 2, 2, 5, False, 3, 0)])
def test_sumfac_edges_vs_numpy(K_max, L, n_chi, n_eps, sine, n_t1, n_t2, cuda_available):
    """Tolerance: FP64 sums of some 1e3 terms on both sides, normwise 1e-12 as the quadrature's other tests."""
    from cf_b200 import geometry, rtensor

    geo = geometry.generate_geometry(L)
    pad = max(66 - 3 * K_max, 2) if n_t2 == 66 else 6
    args = _thin(rtensor.sumfac_inputs(geo, K_max, 0.7, pad, pad), 2, n_chi, n_eps, n_t1, n_t2)
    # gain and loss tables of their own: with the rule cut short the true ones leave a difference gain - loss
    # far below either, in which only rounding could be compared
    rng = np.random.default_rng(K_max + L)
    for j in (22, 23, 24, 25):
        args[j] = np.asfortranarray(rng.standard_normal(args[j].shape))
    if sine:
        args[16] = np.sort(rng.uniform(0, 2 * math.pi, n_eps)).reshape(-1, 1)
    else:
        l = np.floor(np.sqrt(np.arange((L + 1) ** 2)))
        cosine = (np.arange((L + 1) ** 2) >= l * l + l).astype(float)  # no entry for m < 0
        args[23], args[25] = args[23] * cosine[:, None], args[25] * cosine[:, None]
    args[23][:, :, :, -1] = args[25][:, :, -1] = 0.0  # a channel whose every pair is dropped
    ref = _numpy_sumfac(args)
    R = rtensor.compute_R(args, zero_conservation=False)
    assert R.shape == ref.shape
    scale = np.abs(ref).max()
    assert np.abs(R - ref).max() <= 1e-12 * scale, np.abs(R - ref).max() / scale
