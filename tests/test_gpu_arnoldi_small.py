"""The Arnoldi reduction's splits on small systems, restart lengths past a warp.

Chunks of 1 to 8 pieces of 32 U elements (the warps left over share the
vectors), restarts of 1 to 64 (triangular solve over one and two rows per lane,
1 to 130 reduction slots).  DCGS2 and CGS2 build the same Krylov space, so their
solutions agree to the residual bound times the operator's conditioning
(below 40, as in test_gpu_dmma.py): 1e-12 x 40, bound 1e-10.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from multiscat_b200 import ScatteringPlan

from .test_gpu_dmma import _plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("restart", [1, 5, 33, 64])
@pytest.mark.parametrize("n,counts,torus", [(20, (5, 1, 9), 4), (100, (9,), 3), (131, (25, 7), 5),
                                            (400, (6,), 3), (1000, (3,), 2), (64, (700,), 30)])
def test_dcgs2_matches_cgs2(n, counts, torus, restart):
    rng = np.random.default_rng(n + restart)
    t, v, systems, plan = _plan(n, counts, torus, rng)
    plan.close()
    # coupling of the size of D, so that a solve takes tens of steps
    f = rng.uniform(0.3, 0.6, n)
    v[1, 0] = f
    v[torus - 1, 0] = f
    psi = {}
    for gs in ("dcgs2", "cgs2"):
        plan = ScatteringPlan(v, t, systems, rtol=1e-12, restart=restart, gram_schmidt=gs,
                              max_iterations=4000)
        res = plan.solve()
        assert (res.status == 0).all()
        psi[gs] = res.psi
        plan.close()
    torch.testing.assert_close(psi["dcgs2"], psi["cgs2"], rtol=0,
                               atol=1e-10 * float(psi["cgs2"].abs().max()))
