"""tcgen05 block inverse with E streamed from L2 (n > 224).

Random well-conditioned D (as in test_gpu_dmma.py).  BF16x3 keeps 16 bits of
each operand and drops the product of the low parts, about 2.3e-5 of a
product's terms; the terms of both products add up at random, so 2e-4 of the
largest result (the bound of the other tcgen05 forms) has a wide margin.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from multiscat_b200 import ScatteringPlan
from multiscat_b200.workloads import cfg4_batch

from .test_gpu_dmma import _plan

pytestmark = pytest.mark.gpu
TC_TOL = 2e-4


# odd and even n up to the largest that fits (560), n = kp and n < kp, 2 to 5 M tiles, partial tiles, several
# tiles per CTA (9800 rows), both tile widths where they fit
@pytest.mark.parametrize("n,counts,torus,width", [
    (226, (65,), 9, 64), (240, (64, 1), 9, 128), (257, (3,), 3, 64), (300, (121, 100), 11, 128),
    (300, (100, 121), 11, 64), (304, (9800,), 99, 128), (301, (5000, 4803), 99, 64), (400, (70,), 9, 64),
    (550, (100,), 10, 64), (560, (33,), 6, 64),
])
def test_streamed_inverse_matches_fp64(n, counts, torus, width, monkeypatch):
    rng = np.random.default_rng(n + sum(counts))
    t, v, systems, fp64 = _plan(n, counts, torus, rng)
    monkeypatch.setenv("MSC_TUNE", f"c64=0,c32=0,bi={width}")
    mixed = ScatteringPlan(v, t, systems, precision="mixed", tensor_cores=True)
    shape = (mixed.total_rows, n)
    x = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    got = mixed.apply_block_inverse_f32(torch.as_tensor(x, device="cuda")).cpu().numpy()
    assert f"block_inverse32=tc_stream_N{width}" in mixed.tuning_report()["chosen"]
    want = fp64.apply_block_inverse(torch.as_tensor(x.astype(np.complex128), device="cuda")).cpu().numpy()
    np.testing.assert_allclose(got, want, rtol=0, atol=TC_TOL * np.abs(want).max())
    mixed.close()
    fp64.close()


def test_mixed_solve_with_streamed_inverse_matches_fp64():
    case, systems = cfg4_batch(n_azimuths=3, nz=240, nk=19)
    mixed = ScatteringPlan(case.v, case.t, systems, rtol=1e-10, precision="mixed", tensor_cores=True)
    res = mixed.solve()
    assert (res.status == 0).all() and mixed.tensor_core_tile > 0
    ref = ScatteringPlan(case.v, case.t, systems, rtol=1e-10).solve().intensities
    assert float((res.intensities - ref).abs().max()) <= 1e-6
    mixed.close()
