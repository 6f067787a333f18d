"""Slabs of a viscous grid above the face-parallel kernel's number of cells: the
unsplit context runs the strip kernel, and so do its slabs, whatever their own
number of cells, so any split gives the unsplit result bit for bit.  (The two
kernels' viscous stencils differ by roundings.)  Below the line both run the
face-parallel kernel."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, cases, slab

pytestmark = pytest.mark.gpu


def channel(nx, ny):
    bcs = {abi.XLO: abi.BC_PERIODIC, abi.XHI: abi.BC_PERIODIC, abi.YLO: abi.BC_NO_SLIP_WALL, abi.YHI: abi.BC_NO_SLIP_WALL,
           abi.ZLO: abi.BC_SLIP_WALL, abi.ZHI: abi.BC_SLIP_WALL}
    grid = abi.make_grid(nx, ny, hi=(1.0, ny / nx, 1.0 / nx), bcs=bcs)
    params = abi.make_params(cfl=0.3, r_gas=1.0, reconstruction=abi.RECON_MUSCL, viscous=1, mu=1e-3,
                             viscosity_model=abi.VISC_CONSTANT)
    x, y = cases.centroids(grid)
    X, Y = np.meshgrid(2.0 * np.pi * x, np.pi * y * nx / ny)
    u = cases.prim_to_cons(1.0 + 0.3 * np.sin(X + 0.3) * np.cos(Y), 0.4 * np.sin(2 * Y), 0.3 * np.cos(X) * np.sin(Y),
                           1.0 + 0.2 * np.cos(X + Y))
    return grid, params, u


@pytest.mark.parametrize("nx,ny,cuts", [
    (1024, 800, (0, 400, 800)),        # 819,200 cells: two slabs below the line
    (1024, 800, (0, 20, 800)),         # one slab far below it, one just below
    (1021, 807, (0, 5, 807)),          # 823,947 cells, ragged
    (1024, 600, (0, 301, 600)),        # below the line: unsplit and slabs alike
])
def test_viscous_slabs_equal_the_unsplit_context(nx, ny, cuts):
    from dev_field_efvm_b200.device import Context

    grid, params, u = channel(nx, ny)
    ref = Context(grid, params)
    ref.upload(u)
    ref.step(2)
    want, s_ref = ref.download(), ref.solver_state()
    ref.close()
    engines = []
    for lo, hi in zip(cuts, cuts[1:]):
        e = slab.DeviceSlab(grid, params, lo, hi - lo)
        e.ctx.upload(u[lo:hi])
        engines.append(e)
    slab.PeerLocalSlabs(engines, False).step(2)
    got = np.concatenate([e.ctx.download() for e in engines])
    assert engines[0].ctx.solver_state().time == s_ref.time
    assert np.array_equal(got, want)
