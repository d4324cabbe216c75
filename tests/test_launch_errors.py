"""A kernel launch that fails is reported by the call it belongs to.

On the stand-in runtime, launches of the named kernel return an error on the host, as a
refused launch does; the library's calls must not come back with success.
"""

from __future__ import annotations

import pytest

from . import fake_cuda

CASES = [
    ("k_residual_dmma", "plan(30, 5, separable=False)"),
    ("k_block_inverse_dmma", "plan(30, 5, separable=False)"),
    ("k_residual_dmma", "plan(30, 5, separable=False, mixed=True)"),
    ("k_block_inverse_tcs", "plan(240, 5, separable=False, mixed=True, flags=2)"),
    ("k_dcgs_reduce", "plan(30, 5, separable=False)"),
]
CALLS = {
    "k_residual_dmma": "lib.msc_debug_apply_operator(h, buf(h), buf(h), side)",
    "k_block_inverse_dmma": "lib.msc_debug_apply_block_inverse(h, buf(h), buf(h), side)",
    "k_block_inverse_tcs": "lib.msc_debug_apply_block_inverse_f32(h, buf(h), buf(h), side)",
}


@pytest.mark.parametrize("kernel,made", CASES)
def test_a_failed_launch_is_an_error(kernel, made):
    # MSC_TUNE: the streamed form stays chosen, nothing is measured
    fake_cuda.run(f'''
h = {made}
res = nat.Result()
st = lib.msc_solve(h, None, None, ctypes.byref(res), side)
assert any("{kernel}" in x for x in report("launch"))
assert st == nat.MSC_ERR_CUDA, (st, nat.last_error())
lib.msc_plan_destroy(h)
h = {made}
st = {CALLS.get(kernel, "nat.MSC_ERR_CUDA")}
assert st == nat.MSC_ERR_CUDA, (st, nat.last_error())
lib.msc_plan_destroy(h)
''', FAKE_CUDA_FAIL=kernel, MSC_TUNE="c64=0,c32=0,bi=128")


@pytest.mark.parametrize("made", sorted({m for _, m in CASES}))
def test_without_a_failure_the_solve_succeeds(made):
    fake_cuda.run(f'''
h = {made}
res = nat.Result()
assert lib.msc_solve(h, None, None, ctypes.byref(res), side) == 0, nat.last_error()
lib.msc_plan_destroy(h)
''', MSC_TUNE="c64=0,c32=0,bi=128")
