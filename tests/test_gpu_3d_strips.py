"""The 3-D stage kernel's strips of 31 and 32 columns (the latter where they save a
strip) and its rows per warp, at the remainders where they change: one step of
periodic, walled and mixed boxes against the oracle within 1e-12 of each
variable's scale, and a shift by whole cells of the periodic box bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, cases
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def box(nx, ny, nz, side, muscl):
    P = abi.BC_PERIODIC if side == "periodic" else abi.BC_SLIP_WALL
    S = abi.BC_PERIODIC if side != "walls" else abi.BC_SLIP_WALL
    bcs = {abi.XLO: P, abi.XHI: P, abi.YLO: S, abi.YHI: S, abi.ZLO: S, abi.ZHI: S}
    grid = abi.make_grid(nx, ny, hi=(1.0, ny / nx, nz / nx), bcs=bcs, nz=nz)
    params = abi.make_params(cfl=0.3, r_gas=1.0, periodic_seam=abi.SEAM_TRUE_PERIODIC,
                             reconstruction=abi.RECON_MUSCL if muscl else abi.RECON_FIRST_ORDER)
    k, j, i = np.meshgrid(np.arange(nz) / nz, np.arange(ny) / ny, np.arange(nx) / nx, indexing="ij")
    t = 2.0 * np.pi
    rho = 1.0 + 0.2 * np.sin(t * (i + 0.1)) * np.cos(t * (j + k)) + 0.1 * (i > 0.4)
    u = cases.prim_to_cons3(rho, 0.3 * np.sin(t * j), 0.2 * np.cos(t * (k + i)), 0.25 * np.sin(t * (i + j)),
                            1.0 + 0.1 * np.cos(t * (i - k)))
    return grid, params, u


@pytest.mark.parametrize("nx,ny,nz", [(2, 2, 2), (31, 3, 5), (32, 4, 4), (33, 2, 3), (62, 5, 2), (63, 17, 4), (64, 18, 3),
                                      (65, 3, 6), (128, 7, 5)])
@pytest.mark.parametrize("side,muscl", [("periodic", True), ("walls", True), ("mixed", False)])
def test_step_matches_the_oracle(nx, ny, nz, side, muscl):
    from dev_field_efvm_b200.device import Context

    grid, params, u = box(nx, ny, nz, side, muscl)
    d, o = Context(grid, params), pyoracle.OracleCase(grid, params)
    for c in (d, o):
        c.upload(u)
        c.step(1)
    a, b = d.download(), o.download()
    scale = np.max(np.abs(b), axis=(0, 1, 2))
    scale[1:4] = np.max(np.sqrt(np.abs(b[..., 0] * b[..., 4])))
    assert np.max(np.abs(a - b) / scale) < 1e-12


@pytest.mark.parametrize("nx,ny,nz", [(64, 9, 6), (40, 12, 5)])
def test_step_commutes_with_whole_cell_shifts(nx, ny, nz):
    from dev_field_efvm_b200.device import Context

    grid, params, u = box(nx, ny, nz, "periodic", True)
    out = []
    for s in ((0, 0, 0), (1, 3, 5)):
        c = Context(grid, params)
        c.upload(np.roll(u, s, axis=(0, 1, 2)))
        c.step(2)
        out.append(np.roll(c.download(), tuple(-q for q in s), axis=(0, 1, 2)))
    assert np.array_equal(out[0], out[1])
