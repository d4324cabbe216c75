"""Kernels reach into another CTA's shared memory only after a cluster barrier.

CUDA asks that every CTA of a cluster has started before its shared memory is
touched; being launched together does not ensure it.  The sources' order of statements
is checked: loops here never bring a remote access before the barrier above it.
"""

from __future__ import annotations

import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "multiscat_b200" / "csrc"


def kernels():
    for f in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        starts = [m.start() for m in re.finditer(r"__global__", text)] + [len(text)]
        for a, b in zip(starts, starts[1:]):
            if "map_shared_rank" in text[a:b]:
                yield re.search(r"\b(k_\w+)", text[a:b]).group(1), text[a:b]


FOUND = dict(kernels())


def test_the_cluster_kernels_are_found():
    assert {"k_block_inverse_dmma", "k_tridiagonalize_cluster"} <= set(FOUND)


@pytest.mark.parametrize("name", sorted(FOUND))
def test_first_remote_access_follows_a_cluster_barrier(name):
    before = FOUND[name][: FOUND[name].index("map_shared_rank")]
    assert re.search(r"cluster\.sync\(\)|cluster_wait\(\)", before)
    if "cluster_wait" in before:
        assert "cluster_arrive()" in before[: before.index("cluster_wait")]
