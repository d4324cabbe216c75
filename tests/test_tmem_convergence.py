"""TMEM loads are issued by whole warps.

tcgen05.ld is an aligned instruction: all lanes have to arrive together.  In a loop that
some lanes leave a pass of early (a lane-dependent continue), a warp barrier has to
stand before the next pass's load.
"""

from __future__ import annotations

import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "multiscat_b200" / "csrc"
LANE_DEPENDENT = ("stage", "row_ok")


def loops():
    for f in ("msc_tc.cuh", "msc_tcc.cuh", "msc_tcs.cuh"):
        text = re.sub(r"//[^\n]*", "", (CSRC / f).read_text())
        for m in re.finditer(r"if \(!(\w+)\) continue;", text):
            if m.group(1) not in LANE_DEPENDENT:
                continue
            depth, i = 0, m.start()
            while depth >= 0:                    # back to the brace that opens the loop
                i -= 1
                depth += {"}": 1, "{": -1}.get(text[i], 0)
            yield f"{f}:{m.group(1)}", text[i: m.start()]


FOUND = dict(loops())


def test_the_loops_are_found():
    assert set(FOUND) == {"msc_tc.cuh:stage", "msc_tcc.cuh:row_ok"}


@pytest.mark.parametrize("name", sorted(FOUND))
def test_a_warp_barrier_stands_before_the_load(name):
    before = FOUND[name][: FOUND[name].index("tmem_ld")]
    assert "__syncwarp()" in before
