"""Bodies that are set again before every step: the one step on new geometry is
launched directly, a further one through the step graph.  Both equal single
substeps bit for bit, the marker forces and their history included."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, cases

pytestmark = pytest.mark.gpu


def contexts(kind):
    from dev_field_efvm_b200.device import Context

    if kind == "spheres":
        grid, params, u, ex = cases.sphere_drag_case(48, 24, 24)

        def place(c, k):
            c.set_spheres([abi.EfvmSphere(*([0.01 * k, 0.0, 0.0, 0.05] + [0.0] * 6))], ex["freestream"], 300)
    else:
        grid, params, u, ex = cases.cylinder_case(220, 41, muscl=True)

        def place(c, k):
            c.set_discs([abi.EfvmDisc(0.2 + 0.004 * k, 0.2, 0.05, 3.0, -1.0, 20.0)], ex["freestream"], 64)
    out = []
    for _ in range(2):
        c = Context(grid, params)
        c.upload(u)
        out.append(c)
    return out, place


@pytest.mark.parametrize("kind", ["discs", "spheres"])
@pytest.mark.parametrize("steps", [1, 2])
def test_steps_after_every_move_equal_substeps(kind, steps):
    (a, b), place = contexts(kind)
    for k in range(4):
        for c in (a, b):
            place(c, k)
        _, hist = a.step(1, history=True)
        if steps == 2:  # a second step on the same geometry: the graph
            _, h2 = a.step(1, history=True)
            hist = np.concatenate([hist, h2])
        forces = []
        for _ in range(3 * steps):
            b.substep()
            forces.append(b.marker_force())
        assert np.array_equal(a.download(), b.download()), k
        assert np.array_equal(hist, np.stack(forces).reshape(hist.shape)), k
        assert np.array_equal(a.marker_force(), b.marker_force()) and np.array_equal(a.wall_force(), b.wall_force())
    assert a.solver_state().time == b.solver_state().time


def test_asynchronous_steps_after_a_move():
    """Steps enqueued without a status read: the forces of the direct step's last stage
    stay pending and run with the next step, or when they are read."""
    (a, b), place = contexts("discs")
    for k in range(3):
        for c in (a, b):
            place(c, k)
        a.step_async(1)
        a.step_async(2)
        for _ in range(9):
            b.substep()
    assert np.array_equal(a.marker_force(), b.marker_force()) and np.array_equal(a.wall_force(), b.wall_force())
    assert np.array_equal(a.download(), b.download())
