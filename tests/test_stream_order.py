"""Set-up tables reach the device before kernels on other streams read them.

The native library runs on a recording stand-in for the CUDA runtime: a launch on a
plan's or a caller's stream counts as unordered while allocations, copies or kernels of
the legacy stream have neither been waited for nor ordered by an event.
"""

from __future__ import annotations

import pytest

from . import fake_cuda


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [30, 33])
def test_autotuner_waits_for_the_box_lists(mixed, n):
    fake_cuda.run(f'''
h = plan({n}, 9, separable=True, mixed={mixed})
res = nat.Result()
lib.msc_solve(h, None, None, ctypes.byref(res), side)
assert any("k_coupling_box" in x for x in report("launch"))
assert report("unordered") == [], report("unordered")
lib.msc_plan_destroy(h)
''')


@pytest.mark.parametrize("call", ["msc_solve_lower_block", "msc_apply_lower_block"])
@pytest.mark.parametrize("solved_before", [False, True])
def test_lower_block_waits_for_its_tables(call, solved_before):
    # on a plan that was not made for Gauss-Seidel: the level tables are built by this call
    fake_cuda.run(f'''
h = plan(30, 9, separable=False)
res = nat.Result()
if {solved_before}:
    lib.msc_solve(h, None, None, ctypes.byref(res), side)
assert lib.{call}(h, buf(h), buf(h), side) == 0
assert report("unordered") == [], report("unordered")
lib.msc_plan_destroy(h)
''')
