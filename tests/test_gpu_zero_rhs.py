"""A solve with zero right-hand sides takes no cycle and returns zero."""

from __future__ import annotations

import pytest
import torch

from multiscat_b200 import ScatteringPlan
from multiscat_b200.workloads import cfg0_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_zero_right_hand_side(precision):
    case = cfg0_case(nz=40)
    plan = ScatteringPlan(case.v, case.t, [case.system()], rtol=1e-9, precision=precision)
    first = plan.solve()
    assert plan.info().cycles_last == first.cycles.max() > 0
    plan.set_boundary_rhs(torch.zeros(121, dtype=torch.complex128, device="cuda"))
    res = plan.solve()
    assert plan.info().cycles_last == 0 and res.iterations[0] == 0 and not res.psi.any()
    plan.set_boundary_rhs(None)
    assert torch.equal(plan.solve().psi, first.psi)
    plan.close()
