"""The rotation kernel's table ring and rows, by the sources' order of statements.

A slot of the ring is refilled while the chunk after next is used: the lanes may still
read its old chunk unless a warp barrier stands between their reads and the copy.  Of
the 32 lanes of a 16-row block two hold the same row, and one of them writes it.
"""

from __future__ import annotations

import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "multiscat_b200" / "csrc"


def body() -> str:
    text = re.sub(r"//[^\n]*", "", (CSRC / "msc_eigh_gpu.cuh").read_text())
    start = text.index("k_apply_rotations(")
    return text[start: text.index("\n}\n", start)]


def test_a_warp_barrier_stands_before_a_slot_is_refilled():
    loop = body()[body().index("for (int st = 0;"):]
    refill = loop.index("fetch(")
    assert "__syncwarp()" in loop[:refill]
    arrived = loop.index("wait_group 2", refill)
    assert "__syncwarp()" in loop[arrived: loop.index("step(st", arrived)]


def test_one_lane_writes_a_row():
    text = body()
    assert re.search(r"own = threadIdx\.x < RB;", text)
    stores = [m.start() for m in re.finditer(r"zs\[[^;=]*\]\s*=[^=]", text)]
    assert len(stores) == 3
    for s in stores:
        statement = text[max(text.rfind(";", 0, s), text.rfind("{", 0, s)): s]
        before = text[: s].rstrip()
        guarded = "own" in statement or re.search(r"if \(own\)\s*for \([^{}]*$", before)
        assert guarded, text[s - 80: s + 40]
