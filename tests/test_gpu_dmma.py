"""FP64 tensor-core block inverse and residual at the edges of their tiles.

Random symmetric positive definite T (eigenvalues in [1, 11]), real V_00 of
order 1 and pkd in [1, 10], so D is well conditioned (below 40) and both
results are fixed to about 40 eps sqrt(n) of their largest value, 3e-13 at
n = 1024; the bound is 2e-12.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from multiscat_b200 import ScatteringPlan
from multiscat_b200.solver import SystemSpec

pytestmark = pytest.mark.gpu
TOL = 2e-12


def _plan(n, counts, torus, rng):
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    t = (q * rng.uniform(1.0, 11.0, n)) @ q.T
    t = 0.5 * (t + t.T)
    v = np.zeros((torus, torus, n), complex)
    v[0, 0] = rng.uniform(0.0, 1.0, n)
    systems = []
    for c in counts:
        pos = rng.permutation(torus * torus)[:c]
        ix, iy = np.divmod(pos, torus)
        wc = (rng.uniform(-1, 0, c) + 0.3j * rng.uniform(-1, 1, c))
        systems.append(SystemSpec(ix, iy, rng.uniform(1.0, 10.0, c), np.ones(c, complex),
                                  np.ones(c, complex), wc, 0))
    return t, v, systems, ScatteringPlan(v, t, systems)


# n: one k-step, partial and odd k-steps, each split of the nodes over a
# cluster (1, 2, 4, 8 CTAs); rows: partial tiles, tiles across systems, and
# (2500 rows) the wide tiles
@pytest.mark.parametrize("n,counts,torus", [
    (2, (3,), 3), (7, (8, 1), 3), (8, (5, 9, 1), 3), (9, (9,), 3), (33, (25, 24), 5),
    (100, (121,), 11), (160, (9,), 3), (161, (17,), 5), (320, (8,), 3), (325, (3, 4), 3),
    (641, (10,), 4), (1024, (4,), 2), (24, (2500,), 50), (150, (1100, 1399), 50), (171, (2500,), 50),
])
def test_block_inverse_and_operator_match_numpy(n, counts, torus):
    rng = np.random.default_rng(n + sum(counts))
    t, v, systems, plan = _plan(n, counts, torus, rng)
    pkd = np.concatenate([s.pkd for s in systems])
    c = np.concatenate([s.wave_c for s in systems])
    rows = pkd.size
    x = rng.standard_normal((rows, n)) + 1j * rng.standard_normal((rows, n))
    # D^-1 x through the eigenvectors of H0 and the rank-one boundary term
    lam, e = np.linalg.eigh(t + np.diag(v[0, 0].real))
    inv = 1.0 / (pkd[:, None] + lam[None, :])
    xt = x @ e
    en = e[-1]
    beta = c * (xt * inv * en).sum(1) / (1.0 - c * (inv * en**2).sum(1))
    want = ((xt + beta[:, None] * en) * inv) @ e.T
    xd = torch.as_tensor(x, device="cuda")
    got = plan.apply_block_inverse(xd).cpu().numpy()
    np.testing.assert_allclose(got, want, rtol=0, atol=TOL * np.abs(want).max())
    # D x (there is no coupling)
    want = x @ t.T + (v[0, 0].real[None, :] + pkd[:, None]) * x
    want[:, -1] -= c * x[:, -1]
    got = plan.apply_operator(xd).cpu().numpy()
    np.testing.assert_allclose(got, want, rtol=0, atol=TOL * np.abs(want).max())
    plan.close()


def test_solve_leaves_finished_systems_alone():
    """Tiles that hold rows of finished and of unfinished systems: a batch in which
    one system is warm-started with its solution gives each system's own solve."""
    rng = np.random.default_rng(5)
    t, v, systems, plan = _plan(40, (5, 6, 7), 5, rng)
    v[1, 0] = v[4, 0] = 0.2 * rng.standard_normal(40)
    plan.close()
    plan = ScatteringPlan(v, t, systems, rtol=1e-13)
    ref = plan.solve()
    guess = ref.psi.clone()
    guess[5:11] = 0
    plan.set_initial_guess(guess)
    res = plan.solve()
    assert res.iterations[0] == 0 and res.iterations[2] == 0 and res.iterations[1] > 0
    assert torch.equal(res.psi[:5], ref.psi[:5]) and torch.equal(res.psi[11:], ref.psi[11:])
    torch.testing.assert_close(res.psi, ref.psi, rtol=0, atol=1e-11 * float(ref.psi.abs().max()))
    plan.close()
