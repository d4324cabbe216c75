"""Plans for one solve run their FP64 cycles as plain launches: the same kernels, bit for
bit, as the graph of a kept plan, and the same count."""

from __future__ import annotations

import pytest
import torch

from multiscat_b200 import ScatteringPlan
from multiscat_b200.workloads import cfg0_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("options", [{}, {"precision": "mixed"}, {"gram_schmidt": "cgs2"}, {"restart": 5},
                                     {"preconditioner_order": 1}, {"gauss_seidel": True}])
def test_plain_cycles_equal_the_graph(options):
    case = cfg0_case(nz=40)
    out = []
    for single in (False, True):
        plan = ScatteringPlan(case.v, case.t, [case.system()], rtol=1e-8, _single_use=single, **options)
        for _ in range(2):
            out.append((plan.solve(), plan.launches_per_solve()))
        plan.close()
    for res, launches in out[1:]:
        assert torch.equal(res.psi, out[0][0].psi)
        assert launches == out[0][1] > 0
