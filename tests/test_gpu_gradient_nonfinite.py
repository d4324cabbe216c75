"""dL/dV with infinities and NaN in psi or lambda: offsets whose channel pairs are all
finite keep their values, as in the sum over pairs that numpy forms.

The finite sums are bounded as in test_gpu_gradient.py; non-finite entries have to stand
where numpy has them.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from .test_gpu_dmma import _plan
from .test_gpu_gradient import _numpy_gradient

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("torus,counts,n", [(7, (9, 12), 3), (11, (30,), 4), (9, (81, 5), 2)])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("where", ["psi", "lam"])
def test_nonfinite_values_stay_with_their_pairs(torus, counts, n, value, where):
    rng = np.random.default_rng(torus + n)
    _, v, systems, plan = _plan(n, counts, torus, rng)
    rows = sum(counts)
    a = {k: rng.standard_normal((rows, n)) + 1j * rng.standard_normal((rows, n)) for k in ("psi", "lam")}
    a[where][rows - 1, 1] = value * (1 + 1j) if np.isinf(value) else value
    with np.errstate(invalid="ignore"):
        want = _numpy_gradient(v, systems, a["psi"], a["lam"])
    got = plan.potential_gradient(torch.as_tensor(a["psi"], device="cuda"),
                                  torch.as_tensor(a["lam"], device="cuda")).cpu().numpy()
    fine = np.isfinite(want)
    np.testing.assert_array_equal(np.isfinite(got), fine)
    np.testing.assert_allclose(got[fine], want[fine], rtol=0, atol=1e-12 * np.abs(want[fine]).max())
    plan.close()
