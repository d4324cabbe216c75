"""Kept plans that have solved once go on while another thread waits for the device."""

from __future__ import annotations

import threading

import pytest
import torch

from multiscat_b200 import ScatteringPlan
from multiscat_b200.workloads import cfg0_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_device_wide_waits_beside_warm_plans(precision):
    case = cfg0_case(nz=40)
    plans = [ScatteringPlan(case.v, case.t, [case.system()], rtol=1e-8, precision=precision) for _ in range(40)]
    want = [p.solve().psi for p in plans]
    errors, done = [], threading.Event()

    def wait():
        while not done.is_set():
            try:
                torch.cuda.synchronize()
            except RuntimeError as e:
                errors.append(e)
                return

    waiter = threading.Thread(target=wait)
    waiter.start()
    try:
        for p, psi in zip(plans, want):
            for _ in range(4):
                assert torch.equal(p.solve().psi, psi)
    finally:
        done.set()
        waiter.join()
    assert not errors, errors
    for p in plans:
        p.close()
