"""Channel coupling over halo tiles: patches of one and two segments, tori smaller
than a patch or the window, windows of every reach, odd and even z, truncated sets,
the adjoint's taps and the triangular parts.

The taps do not factorise.  Each output is a sum of at most 17^2 complex products,
taken in another order than the reference's: 289 eps = 6e-14 of the sum's magnitude,
bound 1e-12 of the largest output.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from multiscat_b200 import ScatteringPlan
from multiscat_b200.solver import SystemSpec

pytestmark = pytest.mark.gpu
NAMES = {1: "halo_y8", 2: "halo_y4"}


def _system(ix, iy, rng):
    c = len(ix)
    return SystemSpec(np.asarray(ix), np.asarray(iy), rng.uniform(1.0, 2.0, c), np.ones(c, complex),
                      np.ones(c, complex), -np.ones(c, complex), 0)


def _full(nkx, nky):
    return np.repeat(np.arange(nkx), nky), np.tile(np.arange(nky), nkx)


def _disk(nkx, nky, cx, cy, r, rng):
    ix, iy = np.meshgrid(np.arange(-r, r + 1), np.arange(-r, r + 1), indexing="ij")
    keep = ix**2 + iy**2 <= r * r
    order = rng.permutation(int(keep.sum()))
    return ((cx + ix[keep]) % nkx)[order], ((cy + iy[keep]) % nky)[order]


# (nkx, nky), (hx, hy), nz, channel sets
CASES = {
    "1x1": ((1, 1), (0, 0), 5, lambda rng: [_full(1, 1)]),
    "2x1": ((2, 1), (1, 0), 9, lambda rng: [_full(2, 1)]),
    "3x4_h1x2": ((3, 4), (1, 2), 8, lambda rng: [_full(3, 4)]),
    "7x5_h3x2": ((7, 5), (3, 2), 33, lambda rng: [_full(7, 5)]),
    "9x9_h3": ((9, 9), (3, 3), 17, lambda rng: [_full(9, 9)]),
    "11x10_h5": ((11, 10), (5, 5), 16, lambda rng: [_full(11, 10)]),
    "17x17_h8": ((17, 17), (8, 8), 12, lambda rng: [_full(17, 17)]),
    "41x9_h1x4": ((41, 9), (1, 4), 31, lambda rng: [_full(41, 9)]),
    "disks": ((32, 32), (4, 4), 30, lambda rng: [_disk(32, 32, 0, 0, 9, rng), _disk(32, 32, 30, 3, 5, rng),
                                                 _disk(32, 32, 2, 2, 0, rng)]),
    # enough blocks for patches of two segments: columns of 11 and 14, 12 and 9 of 16
    "two_segments_11": ((17, 33), (2, 3), 64, lambda rng: [_full(17, 33)] * 7),
    "two_segments_14": ((41, 41), (4, 4), 97, lambda rng: [_full(41, 41)] * 2),
    "two_segments_12": ((24, 12), (8, 6), 41, lambda rng: [_full(24, 12)] * 25),
    "two_segments_9": ((8, 9), (1, 2), 40, lambda rng: [_full(8, 9)] * 89),
}


def _potential(nkx, nky, hx, hy, nz, rng):
    v = np.zeros((nkx, nky, nz), complex)
    for a in range(-hx, hx + 1):
        for b in range(-hy, hy + 1):
            v[a % nkx, b % nky] = rng.standard_normal(nz) + 1j * rng.standard_normal(nz)
    v[0, 0] = rng.uniform(0.0, 1.0, nz)
    return v


def _reference(v, systems, x, part="all"):
    """sum over taps, and over the source channels below / above the output's."""
    nkx, nky, nz = v.shape
    out, at = np.zeros_like(x), 0
    for s in systems:
        c = len(s.channel_ix)
        for j in range(c):
            d = v[(s.channel_ix[j] - s.channel_ix) % nkx, (s.channel_iy[j] - s.channel_iy) % nky].copy()
            d[j] = 0.0
            if part == "lower":
                d[j:] = 0.0
            out[at + j] = (d * x[at:at + c]).sum(0)
        at += c
    return out


@pytest.mark.parametrize("kind", sorted(NAMES))
@pytest.mark.parametrize("name", sorted(CASES))
def test_halo_tiles(name, kind, monkeypatch):
    (nkx, nky), (hx, hy), nz, channels = CASES[name]
    rng = np.random.default_rng(3)
    v = _potential(nkx, nky, hx, hy, nz, rng)
    systems = [_system(*c, rng) for c in channels(rng)]
    t = np.diag(rng.uniform(1.0, 2.0, nz))
    rows = sum(len(s.channel_ix) for s in systems)
    x = rng.standard_normal((rows, nz)) + 1j * rng.standard_normal((rows, nz))
    xd = torch.as_tensor(x, device="cuda")
    monkeypatch.setenv("MSC_TUNE", f"c64={kind},c32={kind},bi=0")
    plan = ScatteringPlan(v, t, systems)
    got = plan.apply_coupling(xd).cpu().numpy()
    assert f"coupling64={NAMES[kind]}" in plan.tuning_report()["chosen"]
    lower = plan.apply_lower_block(xd).cpu().numpy()
    plan.set_adjoint(True)
    adjoint = plan.apply_coupling(xd).cpu().numpy()
    plan.close()
    diagonal = np.zeros_like(v)
    diagonal[0, 0] = v[0, 0]
    plan = ScatteringPlan(diagonal, t, systems)
    lower -= plan.apply_lower_block(xd).cpu().numpy()
    plan.close()
    some = slice(None) if rows <= 2000 else slice(rows - len(systems[-1].channel_ix), None)
    keep = systems if rows <= 2000 else systems[-1:]
    flip = np.conj(v[(-np.arange(nkx)) % nkx][:, (-np.arange(nky)) % nky])
    for have, ref in ((got, _reference(v, keep, x[some])), (adjoint, _reference(flip, keep, x[some])),
                      (lower, _reference(v, keep, x[some], "lower"))):
        scale = max(float(np.abs(ref).max()), 1.0)
        assert float(np.abs(have[some] - ref).max()) <= 1e-12 * scale


@pytest.mark.parametrize("kind", sorted(NAMES))
@pytest.mark.parametrize("nz", [37, 38])
def test_fp32_halo_tiles_in_a_mixed_solve(kind, nz, monkeypatch):
    """The FP32 instances (8- and 16-byte copies) inside the refinement: the mixed solve
    on each form needs as many inner steps as on the neighbour table, up to two."""
    rng = np.random.default_rng(5)
    channels = [_disk(16, 16, 14, 1, 5, rng), _full(16, 16)]
    v = 0.01 * _potential(16, 16, 3, 2, nz, rng)
    systems = [_system(*c, rng) for c in channels]
    t = np.diag(rng.uniform(1.0, 2.0, nz))
    res = {}
    for k in (0, kind):
        monkeypatch.setenv("MSC_TUNE", f"c64={k},c32={k},bi=0")
        plan = ScatteringPlan(v, t, systems, rtol=1e-12, precision="mixed", tensor_cores=False)
        res[k] = plan.solve()
        plan.close()
    assert np.abs(res[kind].iterations - res[0].iterations).max() <= 2
    torch.testing.assert_close(res[kind].psi, res[0].psi, rtol=0,
                               atol=1e-10 * float(res[0].psi.abs().max()))
