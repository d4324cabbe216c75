"""dL/dV of arbitrary psi and lambda against numpy: grids, windows, batches, subsets.

The sums are of up to 3 x 120 products of normal numbers; both sides round each
of them once: 360 eps = 8e-14 of the largest sum, bound 1e-12.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from multiscat_b200 import ScatteringPlan

from .test_gpu_dmma import _plan

pytestmark = pytest.mark.gpu


def _numpy_gradient(v, systems, psi, lam):
    nkx, nky, n = v.shape
    corr = np.zeros((nkx, nky, n), complex)
    row = 0
    for s in systems:
        c = len(s.channel_ix)
        for g in range(c):
            for h in range(c):
                d = ((s.channel_ix[g] - s.channel_ix[h]) % nkx, (s.channel_iy[g] - s.channel_iy[h]) % nky)
                corr[d] += np.conj(lam[row + g]) * psi[row + h]
        row += c
    grad = -2.0 * np.conj(corr)
    grad[0, 0] = -2.0 * corr[0, 0].real
    return grad


# offsets per thread 5 to 8 with and without padding, windows, tori of 1 to 9 rows,
# several systems, and (95 x 95) the form without shared-memory planes
@pytest.mark.parametrize("torus,counts,n,window", [
    (2, (4,), 2, None), (3, (9,), 5, None), (5, (25, 11), 7, None), (6, (36,), 3, (1, 2)),
    (7, (20, 30, 49), 4, None), (7, (49,), 4, (2, 1)), (8, (64,), 3, None), (9, (60,), 9, (0, 3)),
    (11, (121,), 6, None), (11, (121,), 6, (4, 4)), (95, (60, 50), 3, (3, 3)),
])
def test_potential_gradient_matches_numpy(torus, counts, n, window):
    rng = np.random.default_rng(torus + n)
    _, v, systems, plan = _plan(n, counts, torus, rng)
    rows = sum(counts)
    psi = rng.standard_normal((rows, n)) + 1j * rng.standard_normal((rows, n))
    lam = rng.standard_normal((rows, n)) + 1j * rng.standard_normal((rows, n))
    want = _numpy_gradient(v, systems, psi, lam)
    if window is not None:
        keep = np.zeros(v.shape[:2], bool)
        for a in range(-window[0], window[0] + 1):
            for b in range(-window[1], window[1] + 1):
                keep[a % torus, b % torus] = True
        want[~keep] = 0
    got = plan.potential_gradient(torch.as_tensor(psi, device="cuda"),
                                  torch.as_tensor(lam, device="cuda"), window).cpu().numpy()
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * np.abs(want).max())
    plan.close()
