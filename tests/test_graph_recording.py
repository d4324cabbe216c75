"""When a plan records its CUDA graph.

While one thread records, a device-wide wait of another (torch.cuda.synchronize) fails.
A kept plan records in its first call, when programs warm up, and never later; a plan
for one solve records only if the solve is long or mixed.
"""

from __future__ import annotations

import pytest

from . import fake_cuda


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("first", ["msc_solve", "msc_debug_apply_operator"])
def test_a_kept_plan_records_in_its_first_call_only(mixed, first):
    fake_cuda.run(f'''
h = plan(30, 5, separable=False, mixed={mixed})
res = nat.Result()
solve = lambda: lib.msc_solve(h, None, None, ctypes.byref(res), side)
assert (solve() if "{first}" == "msc_solve" else lib.{first}(h, buf(h), buf(h), side)) == 0, nat.last_error()
assert report("capture") == ["begin"]
fake.fake_reset()
for k in range(5):
    assert solve() == 0, nat.last_error()
    lib.msc_plan_set_adjoint(h, k % 2)
assert report("capture") == []
lib.msc_plan_destroy(h)
''', MSC_TUNE="c64=0,c32=0,bi=0")


def test_a_short_solve_of_a_single_use_plan_records_nothing():
    fake_cuda.run('''
h = plan(30, 5, separable=False, flags=64)
res = nat.Result()
assert lib.msc_solve(h, None, None, ctypes.byref(res), side) == 0, nat.last_error()
assert report("capture") == []
lib.msc_plan_destroy(h)
''', MSC_TUNE="c64=0,c32=0,bi=0")
