"""The network's per-cell inputs left by the corrected stages for the next one, over
everything that replaces the state or changes the stage's form in between: each
run must continue exactly as a fresh context loaded with the same state does
(bit for bit), and track the form that makes a pass over the state before every
stage (the two round the same FP64 quotients before FP32; a flipped FP32 rounding
moves one input by 6e-8 and a correction of order 1e-3 by less: 1e-9)."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, learned

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net():
    return learned.load_trained()


def make(net, n=40):
    from dev_field_efvm_b200.device import Context

    grid, params = learned.grid_params(n, net[1] * 64.0 / n)
    c = Context(grid, params)
    u = learned.family_state(n, 11)
    c.set_flux_correction(net[0])
    c.upload(u)
    return c


def fresh_from(net, c):
    d = make(net)
    d.upload(c.download())
    d.set_solver_state(c.solver_state())
    return d


def test_graph_equals_substeps(net):
    a, b = make(net), make(net)
    a.step(3)
    for _ in range(9):
        b.substep()
    assert np.array_equal(a.download(), b.download())


def test_tracks_the_form_with_a_pass_per_stage(net):
    a, b = make(net), make(net)
    b.set_stage_tiling(abi.STAGE_STRIP, 0)
    a.step(4)
    b.step(4)
    assert np.max(np.abs(a.download() - b.download())) < 1e-9


@pytest.mark.parametrize("change", ["strip", "upload", "detach", "rk_stage", "prepare", "zero_steps", "stop"])
def test_continues_as_a_fresh_context(net, change):
    a = make(net)
    a.step(2)
    if change == "strip":
        a.set_stage_tiling(abi.STAGE_STRIP, 0)
        a.step(1)
        a.set_stage_tiling(abi.STAGE_AUTO, 0)
    elif change == "upload":
        a.upload(np.ascontiguousarray(a.download()[::-1, ::-1]) * np.array([1.0, -1.0, -1.0, 1.0, 1.0]))
    elif change == "detach":
        a.set_flux_correction(None)
        a.step(1)
        a.set_flux_correction(net[0])
    elif change == "rk_stage":
        a.substep()
        a.set_solver_state(a.solver_state())  # another buffer's state is current: stale inputs
        a.substep()
        a.substep()
    elif change == "prepare":
        a.prepare()
    elif change == "zero_steps":
        a.step(0)
    else:
        s = a.solver_state()
        assert a.step(70, t_stop=s.time + 0.5 * s.dt).steps_done == 1
    b = fresh_from(net, a)
    a.step(2)
    b.step(2)
    assert np.array_equal(a.download(), b.download())
