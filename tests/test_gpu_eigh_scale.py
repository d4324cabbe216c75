"""The eigensolver on matrices with very large and very small entries.

A power of two changes no bit of the significands: w scales with the matrix and the
eigenvectors stay, so the residual and orthogonality bounds of test_gpu_eigh.py hold
relative to the largest eigenvalue.  A column below the diagonal whose square is just
denormal (over 40 bits left) or zero couples nothing at that scale.
"""

from __future__ import annotations

import numpy as np
import pytest

from .test_gpu_eigh import _device_eigh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 40, 200])
@pytest.mark.parametrize("exponent", [-480, -400, -360, 360, 400, 480])
def test_scaled_matrix(n, exponent):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    a = 0.5 * (a + a.T)
    w, v = _device_eigh(np.ldexp(a, exponent))
    w = np.ldexp(w, -exponent)
    want = np.linalg.eigvalsh(a)
    scale = np.abs(want).max()
    assert np.abs(w - want).max() <= 1e-13 * n * scale
    assert np.abs(a @ v - v * w).max() <= 1e-13 * n * scale
    assert np.abs(v.T @ v - np.eye(n)).max() <= 1e-13 * n


@pytest.mark.parametrize("n", [4, 40, 200])
@pytest.mark.parametrize("tiny", [1e-154, 1e-155, 1e-200])
def test_nearly_decoupled_rows(n, tiny):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    a = 0.5 * (a + a.T)
    for k in (0, n // 2):
        a[k, k + 1:] *= tiny
        a[k + 1:, k] = a[k, k + 1:]
    w, v = _device_eigh(a)
    want = np.linalg.eigvalsh(a)
    scale = np.abs(want).max()
    assert np.abs(w - want).max() <= 1e-13 * n * scale
    assert np.abs(a @ v - v * w).max() <= 1e-13 * n * scale
    assert np.abs(v.T @ v - np.eye(n)).max() <= 1e-13 * n
