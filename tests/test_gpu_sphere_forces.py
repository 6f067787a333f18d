"""The sphere forces of the step graph (stages 1 and 2 beside the next stage, stage
3 in the next step's first launch) against the same forces read after every
substep, for marker counts around the 128-thread block size.  Both paths run the
same kernel on the same states, so they agree bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, cases

pytestmark = pytest.mark.gpu


def make(n_markers):
    from dev_field_efvm_b200.device import Context

    grid, params, u, ex = cases.sphere_drag_case(48, 24, 24)
    c = Context(grid, params)
    c.set_spheres(ex["spheres"], ex["freestream"], n_markers)
    c.upload(u)
    return c, u, ex


@pytest.mark.parametrize("n_markers", [0, 12, 127, 128, 129, 2000])
def test_step_graph_forces_equal_substep_forces(n_markers):
    a, _, _ = make(n_markers)
    _, hist = a.step(3, history=True)
    b, _, _ = make(n_markers)
    rows = []
    for _ in range(9):
        b.substep()
        rows.append(b.marker_force())
    assert np.array_equal(hist, np.array(rows))
    assert np.array_equal(a.wall_force(), b.wall_force())
    assert np.array_equal(a.download(), b.download())


@pytest.mark.parametrize("change", ["none", "upload", "move"])
def test_pending_forces_survive_what_replaces_their_inputs(change):
    a, u, ex = make(500)
    a.step(2)
    ref = a.marker_force()
    b, _, _ = make(500)
    b.step_async(2)
    if change == "upload":
        b.upload(u)
    elif change == "move":
        b.set_spheres([abi.make_sphere((0.02, 0.0, 0.0), 0.05)], ex["freestream"], 500)
    assert np.array_equal(b.marker_force(), ref)


def test_stopped_run_keeps_the_last_steps_forces():
    a, _, _ = make(300)
    info = a.step(2)
    ref, wall = a.marker_force(), a.wall_force()
    b, _, _ = make(300)
    got = b.step(50, t_stop=0.5 * info.dt + info.time - info.dt)
    assert got.steps_done == 2
    assert np.array_equal(b.marker_force(), ref) and np.array_equal(b.wall_force(), wall)
