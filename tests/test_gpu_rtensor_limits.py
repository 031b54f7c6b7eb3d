"""The quadrature of R where its point sums do not fit in shared memory as they are kept for the shipped operators: all
harmonics at a large L and K, and lists of valid q that do not keep to the channel's band."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_rtensor_edges import _numpy_sumfac, _thin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,K_max,n_ch,every_q", [(23, 11, 24, False), (12, 11, 13, True), (9, 7, 10, True), (22, 11, 23, False)])
def test_sumfac_of_large_lists_vs_numpy(L, K_max, n_ch, every_q, cuda_available):
    """Tolerance: normwise 1e-12, as the quadrature's other tests."""
    from cf_b200 import basis, geometry, rtensor

    a = _thin(rtensor.sumfac_inputs(geometry.generate_geometry(2), K_max, 0.7, 6, 6), 2, 3, 5)
    nq, rng = (L + 1) ** 2, np.random.default_rng(L)
    a[1], a[2] = float(n_ch), float(nq)
    a[16] = np.sort(rng.uniform(0, 2 * np.pi, 5)).reshape(-1, 1)  # no two azimuths mirror each other
    a[18] = np.array([[basis.radial_norm(k, l) for l in range(L + 1)] for k in range(K_max + 1)])
    a[19] = np.array([basis.sh_norm(l, m) for l in range(L + 1) for m in range(-l, l + 1)]).reshape(-1, 1)
    l1 = np.arange(n_ch)
    a[20] = np.stack([l1, rng.integers(0, L + 1, n_ch), rng.integers(0, L + 1, n_ch)], axis=1).astype(float)
    qi = -np.ones((nq, n_ch))
    for c, l in enumerate(l1):
        q = np.arange(1, nq + 1) if every_q else np.arange(l * l + 1, (l + 1) ** 2 + 1)
        qi[: q.size, c] = q
    a[21] = qi
    for j in (22, 23, 24, 25):
        shape = a[j].shape[: a[j].ndim - (2 if j in (23, 25) else 1)] + ((nq, n_ch) if j in (23, 25) else (n_ch,))
        a[j] = np.asfortranarray(rng.standard_normal(shape))
    ref = _numpy_sumfac(a)
    R = rtensor.compute_R(a, zero_conservation=False)
    scale = np.abs(ref).max()
    assert np.abs(R - ref).max() <= 1e-12 * scale, np.abs(R - ref).max() / scale
