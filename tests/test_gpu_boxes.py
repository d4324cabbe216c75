"""Separable channel coupling over channel boxes: the edges of its geometry.

A potential V_d(z) = p_dx(z) q_dy(z) with complex p, q makes every plan
separable; each form is held against the neighbour-table kernel.  Both sum
the same (2 hx + 1)(2 hy + 1) - 1 terms of order 1 in another order, at most
17^2 of them: 289 eps = 6e-14 of the largest term's sum, bound 1e-12.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from multiscat_b200 import ScatteringPlan
from multiscat_b200.solver import SystemSpec

pytestmark = pytest.mark.gpu
NAMES = {3: "separable", 4: "separable_z2", 5: "separable_rows"}


def _case(nkx, nky, hx, hy, nz, channels, rng):
    v = np.zeros((nkx, nky, nz), complex)
    p = rng.standard_normal((2 * hx + 1, nz)) + 1j * rng.standard_normal((2 * hx + 1, nz))
    q = rng.standard_normal((2 * hy + 1, nz)) + 1j * rng.standard_normal((2 * hy + 1, nz))
    for a in range(-hx, hx + 1):
        for b in range(-hy, hy + 1):
            v[a % nkx, b % nky] = p[a + hx] * q[b + hy]
    v[0, 0] = rng.uniform(0.0, 1.0, nz)
    t = np.diag(rng.uniform(1.0, 2.0, nz))
    systems = []
    for ix, iy in channels:
        c = len(ix)
        systems.append(SystemSpec(np.asarray(ix), np.asarray(iy), rng.uniform(1.0, 2.0, c),
                                  np.ones(c, complex), np.ones(c, complex), -np.ones(c, complex), 0))
    return v, t, systems


def _full(nkx, nky):
    return [np.repeat(np.arange(nkx), nky), np.tile(np.arange(nky), nkx)]


def _disk(nkx, nky, cx, cy, r, rng):
    ix, iy = np.meshgrid(np.arange(-r, r + 1), np.arange(-r, r + 1), indexing="ij")
    keep = ix**2 + iy**2 <= r * r
    order = rng.permutation(int(keep.sum()))
    return [((cx + ix[keep]) % nkx)[order], ((cy + iy[keep]) % nky)[order]]


def _columns(nkx, cols):
    return [np.array(cols), np.full(len(cols), 3)]


GEOMETRIES = {
    # around the torus in both directions; windows at and below the kernel's reach
    "full_11x7_h4x3": (11, 7, 4, 3, 33, lambda rng: [_full(11, 7)]),
    "full_3x3_h1": (3, 3, 1, 1, 5, lambda rng: [_full(3, 3)]),
    "full_17x4_h8x1": (17, 4, 8, 1, 21, lambda rng: [_full(17, 4)]),       # torus smaller than H rows
    "full_21x23_h5": (21, 23, 5, 5, 18, lambda rng: [_full(21, 23)]),
    "full_81x81_h8": (81, 81, 8, 8, 9, lambda rng: [_full(81, 81)]),       # strips of rows
    "full_150x9_h2": (150, 9, 2, 2, 7, lambda rng: [_full(150, 9)]),       # cut along x
    # boxes across the torus edge, of several sizes, a lone channel, a box whose free
    # run is shorter than H (it couples around the torus), two far columns
    "disks_32_h4": (32, 32, 4, 4, 30, lambda rng: [_disk(32, 32, 0, 0, 9, rng), _disk(32, 32, 30, 3, 5, rng),
                                                   _disk(32, 32, 5, 17, 1, rng), _disk(32, 32, 2, 2, 0, rng)]),
    "wide_disk_h4": (20, 24, 4, 4, 13, lambda rng: [_disk(20, 24, 3, 7, 8, rng)]),
    "columns_h2": (40, 7, 2, 2, 16, lambda rng: [_columns(40, [0, 1, 20, 21, 39])]),
}


@pytest.mark.parametrize("kind", sorted(NAMES))
@pytest.mark.parametrize("name", sorted(GEOMETRIES))
def test_box_forms_match_neighbour_table(name, kind, monkeypatch):
    nkx, nky, hx, hy, nz, channels = GEOMETRIES[name]
    rng = np.random.default_rng(11)
    v, t, systems = _case(nkx, nky, hx, hy, nz, channels(rng), rng)
    rows = sum(len(s.channel_ix) for s in systems)
    x = torch.as_tensor(rng.standard_normal((rows, nz)) + 1j * rng.standard_normal((rows, nz)),
                        device="cuda")
    out = {}
    for k in (0, kind):
        monkeypatch.setenv("MSC_TUNE", f"c64={k},c32={k},bi=0")
        plan = ScatteringPlan(v, t, systems)
        out[k] = plan.apply_coupling(x)
        plan.set_adjoint(True)
        out[k, "adjoint"] = plan.apply_coupling(x)
        chosen = plan.tuning_report()["chosen"]
        assert "separable" in chosen if k else "coupling64=neighbour" in chosen
        plan.close()
    for key in (kind, (kind, "adjoint")):
        ref = out[0] if key == kind else out[0, "adjoint"]
        scale = max(float(ref.abs().max()), 1e-3)
        assert float((out[key] - ref).abs().max()) <= 1e-12 * scale


@pytest.mark.parametrize("kind", sorted(NAMES))
@pytest.mark.parametrize("nz", [37, 38])
def test_fp32_box_forms_in_a_mixed_solve(kind, nz, monkeypatch):
    """The FP32 instances (8- and 16-byte copies) inside the refinement: the mixed solve
    on each form needs as many inner steps as on the neighbour table, up to two."""
    rng = np.random.default_rng(5)
    channels = [_disk(16, 16, 14, 1, 5, rng), _full(16, 16)]
    v, t, systems = _case(16, 16, 3, 2, nz, channels, rng)
    v *= 0.01
    res = {}
    for k in (0, kind):
        monkeypatch.setenv("MSC_TUNE", f"c64={k},c32={k},bi=0")
        plan = ScatteringPlan(v, t, systems, rtol=1e-12, precision="mixed", tensor_cores=False)
        res[k] = plan.solve()
        plan.close()
    assert np.abs(res[kind].iterations - res[0].iterations).max() <= 2
    torch.testing.assert_close(res[kind].psi, res[0].psi, rtol=0,
                               atol=1e-10 * float(res[0].psi.abs().max()))
