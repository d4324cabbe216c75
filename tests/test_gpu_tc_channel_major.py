"""Channel-major tcgen05 block inverse: node counts from one to eleven 16-node blocks
(unequal 8-column units per warp, none for some), odd and even (direct or bulk copies
in and out), inputs off the 16-byte grid, partial tiles and several tiles per CTA.

Random well-conditioned D (as in test_gpu_dmma.py).  BF16x3 keeps 16 bits of each
operand and drops the product of the low parts, about 2.3e-5 of a product's terms;
2e-4 of the largest result is the bound of the other tcgen05 forms.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from multiscat_b200 import ScatteringPlan

from .test_gpu_dmma import _plan

pytestmark = pytest.mark.gpu
TC_TOL = 2e-4


@pytest.mark.parametrize("n,counts,torus,shift", [
    (16, (65,), 9, 0), (17, (64, 1), 9, 0), (24, (3,), 3, 0), (33, (121,), 11, 0), (48, (9,), 3, 1),
    (100, (121, 100), 11, 0), (100, (9800,), 99, 1), (128, (9801, 63), 99, 0), (151, (9700,), 99, 0),
    (160, (127,), 12, 0), (175, (64,), 8, 0), (176, (9540,), 99, 0), (176, (66,), 9, 1),
])
def test_channel_major_inverse_matches_fp64(n, counts, torus, shift, monkeypatch):
    rng = np.random.default_rng(n + sum(counts))
    t, v, systems, fp64 = _plan(n, counts, torus, rng)
    monkeypatch.setenv("MSC_TUNE", "c64=0,c32=0,bi=128,bg=3")
    mixed = ScatteringPlan(v, t, systems, precision="mixed", tensor_cores=True)
    shape = (mixed.total_rows, n)
    x = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    room = torch.empty(x.size + shift, dtype=torch.complex64, device="cuda")
    xd = room[shift:].view(shape)
    xd.copy_(torch.as_tensor(x))
    assert xd.data_ptr() % 16 == 8 * shift
    got = mixed.apply_block_inverse_f32(xd).cpu().numpy()
    assert "block_inverse32=tcc" in mixed.tuning_report()["chosen"]
    want = fp64.apply_block_inverse(torch.as_tensor(x.astype(np.complex128), device="cuda")).cpu().numpy()
    np.testing.assert_allclose(got, want, rtol=0, atol=TC_TOL * np.abs(want).max())
    mixed.close()
    fp64.close()
