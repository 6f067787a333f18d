"""A stage launch that the runtime refuses (more than 65,535 blocks along y, by an
explicit one row per warp on a tall grid) is an error of every call that needs it,
and leaves the context usable; the stage autotuner does not time such tilings."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, cases

pytestmark = pytest.mark.gpu


def tall(nx, ny):
    bcs = {s: abi.BC_PERIODIC for s in (abi.XLO, abi.XHI, abi.YLO, abi.YHI)}
    grid = abi.make_grid(nx, ny, hi=(float(nx), float(ny), 1.0),
                         bcs=bcs | {abi.ZLO: abi.BC_SLIP_WALL, abi.ZHI: abi.BC_SLIP_WALL})
    f = np.random.default_rng(ny).uniform(-1.0, 1.0, (4, ny, nx))
    u = cases.prim_to_cons(1.0 + 0.1 * f[0], 0.2 * f[1], 0.2 * f[2], 1.0 + 0.1 * f[3])
    return grid, abi.make_params(cfl=0.3, r_gas=1.0, reconstruction=abi.RECON_MUSCL), u


def stepped(grid, params, u, steps):
    from dev_field_efvm_b200.device import Context

    c = Context(grid, params)
    c.upload(u)
    c.step(steps)
    out = c.download()
    c.close()
    return out


def test_every_call_reports_it():
    from dev_field_efvm_b200.device import Context, EfvmError

    grid, params, u = tall(4, 70000)
    c = Context(grid, params)
    c.upload(u)
    c.set_stage_tiling(abi.STAGE_STRIP, 1)
    for _ in range(2):
        with pytest.raises(EfvmError) as e:
            c.step(1)
        assert e.value.code == abi.ERR_CUDA
    assert np.array_equal(c.download(), u)
    c.set_stage_tiling(abi.STAGE_AUTO, 0)
    c.step(2)
    assert np.array_equal(c.download(), stepped(grid, params, u, 2))


def test_autotune_keeps_a_tiling_that_runs():
    from dev_field_efvm_b200.device import Context

    grid, params, u = tall(2, 270000)
    c = Context(grid, params)
    c.upload(u)
    assert c.autotune_stage(2) > 0.0
    c.step(2)
    assert np.array_equal(c.download(), stepped(grid, params, u, 2))
