"""The face-parallel stage kernel (the built-in choice of the smaller FP64 cases: up
to 400,000 cells where the TMA-fed form applies, 800,000 elsewhere) against the strip
kernel on the same states.  Inviscid: both evaluate the same explicitly rounded
operations, so they agree bit for bit, whatever the grid's remainder against the
31 x 3 tile.  Viscous: the stencil's reciprocals are formed per cell instead of
shared, a few ulps: 1e-13 of each variable's scale per step."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, cases

pytestmark = pytest.mark.gpu


def state(grid, seed):
    rng = np.random.default_rng(seed)
    x, y = cases.centroids(grid)
    X, Y = np.meshgrid(x, y)
    k = rng.uniform(0.0, 2.0 * np.pi, 4)
    lx, ly = grid.hi[0] - grid.lo[0], grid.hi[1] - grid.lo[1]
    sx, sy = 2.0 * np.pi * (X - grid.lo[0]) / lx, 2.0 * np.pi * (Y - grid.lo[1]) / ly
    rho = 1.0 + 0.3 * np.sin(sx + k[0]) * np.cos(sy + k[1]) + 0.2 * (X > grid.lo[0] + 0.4 * lx)
    return cases.prim_to_cons(rho, 0.4 * np.sin(sy + k[2]), 0.3 * np.cos(sx + k[3]), 1.0 + 0.2 * np.cos(sx + sy))


def pair(grid, params, u, steps=2, euler=False):
    from dev_field_efvm_b200.device import Context

    out = []
    for form in (abi.STAGE_AUTO, abi.STAGE_STRIP):
        c = Context(grid, params)
        c.set_stage_tiling(form, 0)
        assert c.stage_tiling()[0] == abi.STAGE_STRIP
        c.upload(u)
        if euler:
            for _ in range(steps):
                c.substep()
        else:
            c.step(steps)
        out.append((c.download(), c.solver_state().dt, c.solver_state().time))
        c.close()
    return out


SIDES = {"periodic": abi.BC_PERIODIC, "open": abi.BC_SUPERSONIC_OUTFLOW, "slip": abi.BC_SLIP_WALL,
         "noslip": abi.BC_NO_SLIP_WALL}


def box(nx, ny, sx, sy):
    bcs = {abi.XLO: SIDES[sx], abi.XHI: SIDES[sx], abi.YLO: SIDES[sy], abi.YHI: SIDES[sy],
           abi.ZLO: abi.BC_SLIP_WALL, abi.ZHI: abi.BC_SLIP_WALL}
    return abi.make_grid(nx, ny, hi=(1.0, ny / nx, 1.0 / nx), bcs=bcs)


@pytest.mark.parametrize("nx,ny", [(2, 2), (3, 5), (30, 3), (31, 4), (32, 6), (62, 7), (63, 2), (94, 31)])
@pytest.mark.parametrize("sx,sy", [("periodic", "periodic"), ("open", "slip"), ("periodic", "open")])
def test_equals_the_strip_kernel_bit_for_bit(nx, ny, sx, sy):
    grid = box(nx, ny, sx, sy)
    params = abi.make_params(cfl=0.3, r_gas=1.0, reconstruction=abi.RECON_MUSCL)
    a, b = pair(grid, params, state(grid, nx + ny))
    assert np.array_equal(a[0], b[0]) and a[1:] == b[1:]


@pytest.mark.parametrize("kw", [dict(flux_scheme=abi.FLUX_RUSANOV), dict(flux_scheme=abi.FLUX_HLLC_TEXTBOOK),
                                dict(limiter=abi.LIMITER_MC), dict(periodic_seam=abi.SEAM_TRUE_PERIODIC),
                                dict(reconstruction=abi.RECON_FIRST_ORDER), dict(body_force_x=0.3),
                                dict(fixed_dt=1e-3), dict(integrator=abi.INTEGRATOR_EULER),
                                dict(sponge=1, sponge_x_start=0.6, sponge_x_end=1.0, sponge_sigma=5.0,
                                     sponge_u_max=0.1, sponge_height=0.6, sponge_rho=1.0, sponge_p=1.0)])
def test_equals_the_strip_kernel_for_every_option(kw):
    grid = box(67, 41, "periodic", "periodic")
    params = abi.make_params(**{"cfl": 0.3, "r_gas": 1.0, "reconstruction": abi.RECON_MUSCL, **kw})
    a, b = pair(grid, params, state(grid, 7), euler="integrator" in kw)
    assert np.array_equal(a[0], b[0]) and a[1:] == b[1:]


def test_one_row():
    grid, params, u, _ = cases.sod_case(100)
    a, b = pair(grid, params, u, steps=5)
    assert np.array_equal(a[0], b[0]) and a[1:] == b[1:]


@pytest.mark.parametrize("nx,ny", [(31, 3), (45, 20), (64, 31)])
@pytest.mark.parametrize("sx,sy,order", [("periodic", "noslip", 1), ("open", "open", 1), ("periodic", "periodic", 0)])
def test_viscous_terms_agree_with_the_strip_kernel(nx, ny, sx, sy, order):
    grid = box(nx, ny, sx, sy)
    params = abi.make_params(cfl=0.3, r_gas=1.0, reconstruction=order, viscous=1, mu=2e-3,
                             viscosity_model=abi.VISC_CONSTANT)
    u = state(grid, 5)
    (a, dta, _), (b, dtb, _) = pair(grid, params, u)
    scale = np.array([1.0, 1.0, 1.0, 1.0, 3.0])
    assert np.max(np.abs(a - b) / scale) < 2e-13
    assert abs(dta - dtb) < 1e-13 * dtb


def test_bodies_agree_with_the_strip_kernel():
    from dev_field_efvm_b200.device import Context

    grid, params, u, ex = cases.cylinder_case(220, 41, muscl=True)
    res = []
    for form in (abi.STAGE_AUTO, abi.STAGE_STRIP):
        c = Context(grid, params)
        c.set_stage_tiling(form, 0)
        c.set_cylinders(ex["cylinders"], ex["freestream"])
        c.upload(u)
        _, hist = c.step(3, history=True)
        res.append((c.download(), hist))
    scale = np.array([1.0, 75.0, 75.0, 1.0, 2.6e5])
    assert np.max(np.abs(res[0][0] - res[1][0]) / scale) < 1e-12
    assert np.max(np.abs(res[0][1] - res[1][1])) < 1e-9 * np.max(np.abs(res[1][1]))
