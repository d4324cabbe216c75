"""Lower-block solve as the first call on a fresh plan, on a caller's own stream.

Two sweeps of the same kernel on the same values: equal to the last bit.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from multiscat_b200 import ScatteringPlan
from multiscat_b200.workloads import cfg0_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [31, 40])
def test_first_lower_block_solve_on_a_side_stream(nz):
    case = cfg0_case(nz=nz)
    rng = np.random.default_rng(nz)
    x = torch.as_tensor(rng.standard_normal((121, nz)) + 1j * rng.standard_normal((121, nz)), device="cuda")
    kept = ScatteringPlan(case.v, case.t, [case.system()])
    want = kept.solve_lower_block(x)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for _ in range(5):
        plan = ScatteringPlan(case.v, case.t, [case.system()])
        with torch.cuda.stream(side):
            got = plan.solve_lower_block(x)
        side.synchronize()
        assert torch.equal(got, want)
        plan.close()
    kept.close()
