"""Plans share streams, pinned blocks and a memory pool: threads, sizes, release, growth."""

from __future__ import annotations

import threading

import numpy as np
import pytest
import torch

from multiscat_b200 import ScatteringPlan, release_cached_memory
from multiscat_b200.workloads import cfg0_case, cfg2_batch

pytestmark = pytest.mark.gpu


def test_plans_built_and_destroyed_by_several_threads():
    """Each thread builds, solves and closes plans of changing sizes and precisions while
    another releases idle resources; every result equals the one found alone."""
    cases = []
    for k, (beams, nz) in enumerate([(1, 60), (40, 50), (700, 24), (3, 61)]):
        case, systems = cfg2_batch(n_solves=beams, seed=k, nz=nz, torus=20, cutoff_mev=90.0)
        cases.append((case, systems))

    def solve(k, precision):
        case, systems = cases[k]
        plan = ScatteringPlan(case.v, case.t, systems, rtol=1e-6, precision=precision)
        res = plan.solve(raise_on_error=False)
        out = res.intensities.cpu().numpy(), res.iterations.copy(), res.status.copy()
        plan.close()
        return out

    want = {(k, p): solve(k, p) for k in range(len(cases)) for p in ("fp64", "mixed")}
    errors = []

    def work(seed):
        rng = np.random.default_rng(seed)
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(6):
                    key = (int(rng.integers(len(cases))), ("fp64", "mixed")[int(rng.integers(2))])
                    got = solve(*key)
                    for a, b in zip(got, want[key]):
                        np.testing.assert_array_equal(a, b)
        except BaseException as e:      # noqa: BLE001 - reported by the test
            errors.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    while any(t.is_alive() for t in threads):
        release_cached_memory()
        threads[0].join(0.01)
    for t in threads:
        t.join()
    assert not errors, errors


def test_a_kept_plan_survives_release_and_other_plans():
    case = cfg0_case(nz=40)
    plan = ScatteringPlan(case.v, case.t, [case.system()], rtol=1e-10)
    first = plan.solve().intensities.clone()
    release_cached_memory()
    for nz in (30, 50, 230):
        other = cfg0_case(nz=nz)
        p = ScatteringPlan(other.v, other.t, [other.system()], rtol=1e-8, precision="mixed")
        p.solve()
        p.close()
    release_cached_memory()
    assert torch.equal(plan.solve().intensities, first)
    plan.close()


def test_new_potentials_do_not_accumulate_device_memory():
    case = cfg0_case(nz=160)

    def one(k):
        v = case.v.copy()
        v[0, 0] += 1e-3 * k
        plan = ScatteringPlan(v, case.t, [case.system()], rtol=1e-4)
        plan.solve()
        plan.close()

    one(0)
    torch.cuda.synchronize()
    release_cached_memory()
    before = torch.cuda.mem_get_info()[0]
    for k in range(1, 25):
        one(k)
    torch.cuda.synchronize()
    release_cached_memory()
    # one eigendecomposition's buffers at n = 160 are about 2 MB: 24 leaked sets would be 48 MB
    assert before - torch.cuda.mem_get_info()[0] < 16 << 20


@pytest.mark.parametrize("options", [{}, {"precision": "mixed"}, {"gram_schmidt": "cgs2"},
                                     {"preconditioner_order": 1}, {"gauss_seidel": True},
                                     {"precision": "mixed", "preconditioner_order": 1, "restart": 7},
                                     {"precision": "mixed", "inner_gram_schmidt_passes": 1}])
def test_plain_and_graph_cycles_are_the_same_launches(options):
    """The first two solves launch a cycle's kernels one by one, later ones as a graph:
    same results bit for bit, same number of kernels (counted in the graph)."""
    case = cfg0_case(nz=40)
    plan = ScatteringPlan(case.v, case.t, [case.system()], rtol=1e-8, **options)
    seen = [(plan.solve(), plan.launches_per_solve()) for _ in range(4)]
    for res, launches in seen[1:]:
        assert torch.equal(res.psi, seen[0][0].psi)
        assert launches == seen[0][1] > 0
    plan.close()
