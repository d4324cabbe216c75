"""Grids of the FP64 kernels and the Arnoldi chunks follow the device's SM count.

One 11 x 11-channel system: 16 narrow tiles.  A tile's nodes are split over a cluster
while every CTA still has an SM to itself, and a pass takes at most two blocks per SM.
"""

from __future__ import annotations

import pytest

from . import fake_cuda


@pytest.mark.parametrize("sms,cluster", [(148, 4), (64, 4), (40, 2), (20, 1)])
def test_split_of_one_small_system(sms, cluster):
    out = fake_cuda.run('''
h = plan(100, 11, separable=False)
res = nat.Result()
assert lib.msc_solve(h, None, None, ctypes.byref(res), side) == 0, nat.last_error()
grids = {x.split(" ")[2]: x.split(" ")[0] for x in report("grid")}
for key in ("k_block_inverse_dmma", "k_dcgs_reduce"):
    print([v for k, v in grids.items() if key in k][0])
lib.msc_plan_destroy(h)
''', FAKE_CUDA_SMS=str(sms), MSC_TUNE="c64=0")
    inverse, reduction = (int(x) for x in out.split())
    assert inverse == 16 * cluster
    assert reduction <= 2 * sms
