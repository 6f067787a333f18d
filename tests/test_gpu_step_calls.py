"""Synchronous steps skip the control launch and the step counter's read where the
last call left both known: step counts, clocks and force histories over mixed
sequences of calls against one context that runs them in one go."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, cases

pytestmark = pytest.mark.gpu


def vortex():
    from dev_field_efvm_b200.device import Context

    grid, params, u, _ = cases.vortex_case(40, periodic=True, muscl=True, mean=(1.0, 1.0), cfl=0.4)
    c = Context(grid, params)
    c.upload(u)
    return c


def test_step_counts_over_mixed_calls():
    a, b = vortex(), vortex()
    total = 0
    for op in ("sync", "sync", "async", "sync", "sub", "sync", "stop", "sync", "restore", "sync", "profile", "sync", "tune", "sync"):
        if op == "sync":
            info = a.step(2)
            assert info.steps_done == 2 and info.substeps_done == 6
            total += 2
        elif op == "async":
            a.step_async(3)
            total += 3
        elif op == "sub":
            for _ in range(3):
                a.substep()
            total += 1
        elif op == "stop":
            s = a.solver_state()
            assert a.step(5, t_stop=s.time + 1.5 * s.dt).steps_done == 2
            total += 2
        elif op == "restore":
            s = a.solver_state()
            s.step += 100
            a.set_solver_state(s)
            s.step -= 100
            a.step(1)
            total += 1
        elif op == "profile":
            a.profile_steps(1)
            total += 1
        else:
            a.autotune_stage(1)
            a.set_stage_tiling(abi.STAGE_AUTO, 0)
    b.step(total)
    assert a.solver_state().step == total + 100
    assert np.array_equal(a.download(), b.download()) and a.solver_state().time == b.solver_state().time


def test_history_after_plain_and_async_calls():
    from dev_field_efvm_b200.device import Context

    def make():
        grid, params, u, ex = cases.cylinder_case(110, 41)
        c = Context(grid, params)
        c.set_cylinders(ex["cylinders"], ex["freestream"])
        c.upload(u)
        return c

    a, b = make(), make()
    _, full = b.step(9, history=True)
    a.step(1)
    _, h1 = a.step(2, history=True)
    a.step(1)
    a.step_async(2)
    _, h2 = a.step(3, history=True)
    assert np.array_equal(h1, full[3:9]) and np.array_equal(h2, full[18:27])
    assert np.array_equal(a.marker_force(), full[-1])
