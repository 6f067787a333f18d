"""The set-up inside the face-parallel stages (whole steps from the graph) against
the separate set-up launch of the substep path: the same clock, dt and state bit
for bit, a stop time inside the run, a restored clock, and the non-physical flag
raised in each RK stage."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, cases

pytestmark = pytest.mark.gpu


def context(fixed_dt=0.0, n=50):
    from dev_field_efvm_b200.device import Context

    grid, params, u, _ = cases.vortex_case(n, periodic=True, muscl=True, mean=(1.0, 1.0), cfl=0.4)
    params.fixed_dt = fixed_dt
    c = Context(grid, params)
    c.upload(u)
    return c, u


@pytest.mark.parametrize("fixed_dt", [0.0, 1e-3])
def test_graph_steps_equal_substeps(fixed_dt):
    a, _ = context(fixed_dt)
    b, _ = context(fixed_dt)
    a.step(4)
    a.step_async(1)
    for _ in range(15):
        b.substep()
    sa, sb = a.solver_state(), b.solver_state()
    assert (sa.dt, sa.time, sa.step) == (sb.dt, sb.time, sb.step)
    assert np.array_equal(a.download(), b.download())
    a.substep(), a.substep(), a.substep()  # the separate set-up after a folded step
    b.step(1)
    assert np.array_equal(a.download(), b.download()) and a.solver_state().dt == b.solver_state().dt


def test_stop_time_and_further_steps():
    a, _ = context()
    info = a.step(3)
    b, _ = context()
    got = b.step(40, t_stop=info.time - 0.5 * info.dt)
    assert got.steps_done == 3 and got.stopped_at_t_stop == 1
    assert np.array_equal(a.download(), b.download())
    a.step(2)
    b.step(2)
    assert np.array_equal(a.download(), b.download()) and a.solver_state().time == b.solver_state().time


def test_external_wave_speed_slot():
    a, _ = context()
    b, _ = context()
    b.wave_speed_slot()
    a.step(3)
    b.step(3)
    assert a.solver_state().dt == b.solver_state().dt
    assert np.array_equal(a.download(), b.download())


def test_nonphysical_state_stops_the_run():
    from dev_field_efvm_b200.device import EfvmError

    c, u = context()
    bad = u.copy()
    bad[20, 20, 0] = -1.0
    c.upload(bad)
    with pytest.raises(EfvmError) as e:
        c.step(3)
    assert e.value.code == abi.ERR_NONPHYSICAL
    assert c.L.efvm_step(c.h, 2, 0, 0.0, None, None) == abi.OK  # enqueues; the state stays stopped
    with pytest.raises(EfvmError):
        c.solver_state()
