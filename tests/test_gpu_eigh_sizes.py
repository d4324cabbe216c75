"""Eigen-decomposition at the edges of its forms: one CTA, clusters of 8 and 16 and the
form from L2 for the reduction, 32 and 16 rows per CTA for the rotations, 4 to 32
entries a lane for the back-transformation; the bounds of test_gpu_eigh.py."""

from __future__ import annotations

import numpy as np
import pytest

from .test_gpu_eigh import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 5, 31, 33, 128, 129, 256, 257, 448, 456, 512, 513, 624, 632, 860, 1024])
def test_sizes(n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    _check(a + a.T)


@pytest.mark.parametrize("n", [90, 200, 470, 640])
def test_decoupled_and_repeated_eigenvalues(n):
    """Columns that need no reflection, blocks that deflate at once, groups of sweeps of
    different ranges, equal eigenvalues."""
    rng = np.random.default_rng(n)
    h = np.zeros((n, n))
    sizes, at = (1, 7, 30, 1, 2, 40), 0
    while at < n:
        for m in sizes:
            m = min(m, n - at)
            b = rng.standard_normal((m, m))
            h[at:at + m, at:at + m] = b + b.T
            at += m
    _check(h)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    h = (q * np.repeat([1.0, 2.0, 2.0 + 1e-9, -3.0, 0.0], -(-n // 5))[:n]) @ q.T
    _check(0.5 * (h + h.T))
