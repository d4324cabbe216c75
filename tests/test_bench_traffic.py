"""The benchmark's DRAM figures come from captures whose vectors do not fit in L2."""

from __future__ import annotations

import pathlib
import sys

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

import bench  # noqa: E402

L2_BYTES = 126e6
NODES = 150


@pytest.mark.parametrize("kind", sorted(bench.NCU_TRAFFIC))
def test_captured_vectors_are_larger_than_l2(kind):
    total, rows, profile = bench.NCU_TRAFFIC[kind]
    assert rows * NODES * 8 > L2_BYTES
    assert total > 0 and (ROOT / "profiles" / profile).exists()
