"""The mixed form's default block inverse keeps FP32 products above 224 nodes.

Random well-conditioned D (as in test_gpu_dmma.py).  A chain of n FP32 products and
sums is off by about sqrt(n) 2^-24 of its result (2-norm, rounding errors at random);
D^-1 is two such products, so 2 sqrt(n) 2^-24 bounds it (1.8e-6 at n = 225, 2.8e-6 at
560).  Operands cut to two BF16 parts without the product of the low parts are off by
2^-17 of each term, 4e-6 and more after both products, whatever n is.
"""

from __future__ import annotations

import math

import numpy as np
import pytest
import torch

from multiscat_b200 import ScatteringPlan

from .test_gpu_dmma import _plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,counts,torus", [(225, (70,), 9), (300, (121, 100), 11), (301, (64, 1), 9), (560, (33,), 6)])
def test_default_inner_inverse_has_fp32_accuracy(n, counts, torus):
    rng = np.random.default_rng(n + sum(counts))
    t, v, systems, fp64 = _plan(n, counts, torus, rng)
    mixed = ScatteringPlan(v, t, systems, precision="mixed")
    shape = (mixed.total_rows, n)
    x = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    got = mixed.apply_block_inverse_f32(torch.as_tensor(x, device="cuda")).cpu().numpy().astype(np.complex128)
    want = fp64.apply_block_inverse(torch.as_tensor(x.astype(np.complex128), device="cuda")).cpu().numpy()
    assert np.linalg.norm(got - want) <= 2.0 * math.sqrt(n) * 2.0**-24 * np.linalg.norm(want)
    mixed.close()
    fp64.close()
