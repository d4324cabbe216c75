"""Which form of the separable coupling a plan runs, field by field of its report.

The forms differ in the z per block: "separable" the most, "separable_z2" half,
"separable_rows" a quarter.  A box that does not fit a form's shared memory is cut into
strips of rows; where not even a strip of one row fits, the next form is taken.  FP64,
reach 4, bytes = 16 zc (cells of src + cells of t) + rows: one-row strips fit 112 KB up to
42 columns at zc = 8, up to 63 at zc = 4, and up to the 96 columns of any box at zc = 2.
"""

from __future__ import annotations

import pytest

from . import fake_cuda

NAMES = {3: "separable", 4: "separable_z2", 5: "separable_rows"}
# torus, reach: the FP64 and FP32 forms that run where 3, 4 and 5 are asked for
RUNS = {
    (3, 1): {3: (3, 3), 4: (4, 4), 5: (5, 5)},
    (9, 1): {3: (3, 3), 4: (4, 4), 5: (5, 5)},
    (33, 4): {3: (3, 3), 4: (4, 4), 5: (5, 5)},
    (50, 4): {3: (4, 4), 4: (4, 4), 5: (5, 5)},
    (81, 4): {3: (5, 4), 4: (5, 4), 5: (5, 5)},
    (81, 8): {3: (3, 3), 4: (4, 4), 5: (5, 5)},
}


@pytest.mark.parametrize("torus,reach", sorted(RUNS))
@pytest.mark.parametrize("kind", sorted(NAMES))
def test_the_form_that_fits_runs(kind, torus, reach):
    out = fake_cuda.run(f'''
h = plan(18, {torus}, separable=True, mixed=True, reach={reach})
assert lib.msc_debug_apply_coupling(h, buf(h), buf(h), side) == 0, nat.last_error()
print(lib.msc_plan_tuning_report(h).decode())
lib.msc_plan_destroy(h)
''', MSC_TUNE=f"c64={kind},c32={kind},bi=0")
    fields = out.split('"chosen": "')[1].split('"')[0].split(",")
    fp64, fp32 = RUNS[torus, reach][kind]
    assert f"coupling64={NAMES[fp64]}" in fields
    assert f"coupling32={NAMES[fp32]}" in fields
