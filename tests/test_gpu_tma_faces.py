"""The TMA-fed stage kernel's x faces, read from the ring, against the strip
kernel's at the remainders of strips (31 columns) and blocks (124 columns), of
rows per warp, and on every kind of edge.  FP64: the same explicitly rounded
operations, so the same bits.  FP32 fluxes: the compiler may fuse differently in
the two kernels, a rounding of 2^-24 per operation: 2e-6 of each variable's scale."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, cases

pytestmark = pytest.mark.gpu


def run(nx, ny, sx, sy, rows, **kw):
    from dev_field_efvm_b200.device import Context

    bcs = {abi.XLO: sx, abi.XHI: sx, abi.YLO: sy, abi.YHI: sy, abi.ZLO: abi.BC_SLIP_WALL, abi.ZHI: abi.BC_SLIP_WALL}
    grid = abi.make_grid(nx, ny, hi=(1.0, ny / nx, 1.0 / nx), bcs=bcs)
    params = abi.make_params(**{"cfl": 0.3, "r_gas": 1.0, "reconstruction": abi.RECON_MUSCL, **kw})
    x, y = cases.centroids(grid)
    X, Y = np.meshgrid(2 * np.pi * x, 2 * np.pi * y * nx / ny)
    rho = 1.0 + 0.3 * np.sin(X + 0.3) * np.cos(Y) + 0.2 * (X > 2.0)
    u = cases.prim_to_cons(rho, 0.4 * np.sin(Y + 0.2), 0.3 * np.cos(X), 1.0 + 0.2 * np.cos(X + Y))
    out = []
    for form in (abi.STAGE_TMA, abi.STAGE_STRIP):
        c = Context(grid, params)
        c.set_stage_tiling(form, rows if form == abi.STAGE_TMA else 0)
        assert c.stage_tiling()[0] == form
        c.upload(u)
        info = c.step(2)
        out.append((c.download(), info.dt))
        c.close()
    return out


P, O, W = abi.BC_PERIODIC, abi.BC_SUPERSONIC_OUTFLOW, abi.BC_SLIP_WALL


@pytest.mark.parametrize("nx", [2, 3, 30, 31, 32, 62, 93, 123, 124, 125, 249])
@pytest.mark.parametrize("sx,sy", [(P, P), (O, W)])
def test_fp64_equals_the_strip_kernel(nx, sx, sy):
    a, b = run(nx, 19, sx, sy, 0)
    assert np.array_equal(a[0], b[0]) and a[1] == b[1]


@pytest.mark.parametrize("kw", [dict(limiter=abi.LIMITER_MC), dict(periodic_seam=abi.SEAM_TRUE_PERIODIC),
                                dict(reconstruction=abi.RECON_FIRST_ORDER), dict(flux_scheme=abi.FLUX_RUSANOV)])
@pytest.mark.parametrize("ny,rows", [(2, 1), (33, 7), (40, 64)])
def test_fp64_options_and_rows(kw, ny, rows):
    a, b = run(130, ny, P, P, rows, **kw)
    assert np.array_equal(a[0], b[0]) and a[1] == b[1]


@pytest.mark.parametrize("nx,ny,sx,sy", [(31, 5, P, P), (125, 18, P, P), (130, 33, O, W)])
def test_fp32_flux_tracks_the_strip_kernel(nx, ny, sx, sy):
    a, b = run(nx, ny, sx, sy, 0, precision=abi.PREC_FP32_FLUX)
    scale = np.array([1.5, 1.0, 1.0, 1.0, 3.0])
    assert np.max(np.abs(a[0] - b[0]) / scale) < 2e-6
