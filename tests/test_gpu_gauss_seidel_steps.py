"""Inner steps of the mixed Gauss-Seidel solves: the stop rule at the tolerance itself.

The counts are those of the solver whose inner solves stop there; half the tolerance
takes one or two steps more on each.
"""

from __future__ import annotations

import pytest

from multiscat_b200 import ScatteringPlan
from multiscat_b200.workloads import cfg0_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,order,rtol,steps", [(30, 0, 1e-8, 17), (33, 1, 1e-8, 16), (40, 1, 1e-8, 10),
                                                 (48, 0, 1e-10, 16), (60, 0, 1e-9, 14)])
def test_inner_steps(nz, order, rtol, steps):
    case = cfg0_case(nz=nz)
    plan = ScatteringPlan(case.v, case.t, [case.system()], rtol=rtol, precision="mixed", gauss_seidel=True,
                          preconditioner_order=order)
    res = plan.solve()
    assert (res.status == 0).all() and (res.residual <= rtol).all()
    assert res.iterations[0] <= steps
    plan.close()
