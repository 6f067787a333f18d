"""Which kernel a stage runs (efvm_get_stage_kernel), and that the tiling a context
reports names it: reading the tiling and setting it again changes nothing, in the
same context and in another one of the case."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, cases

pytestmark = pytest.mark.gpu


def box(nx, ny):
    bcs = {abi.XLO: abi.BC_PERIODIC, abi.XHI: abi.BC_PERIODIC}
    bcs[abi.YLO] = bcs[abi.YHI] = abi.BC_PERIODIC if ny > 1 else abi.BC_SLIP_WALL
    return abi.make_grid(nx, ny, hi=(1.0, ny / nx, 1.0), bcs=bcs | {abi.ZLO: abi.BC_SLIP_WALL, abi.ZHI: abi.BC_SLIP_WALL})


def context(nx, ny, **kw):
    from dev_field_efvm_b200.device import Context

    return Context(box(nx, ny), abi.make_params(**{"cfl": 0.3, "r_gas": 1.0, "reconstruction": abi.RECON_MUSCL, **kw}))


VISC = dict(viscous=1, mu=1e-3, viscosity_model=abi.VISC_CONSTANT)
F, S, T = abi.KERNEL_FACES, abi.KERNEL_STRIP, abi.KERNEL_TMA


@pytest.mark.parametrize("nx,ny,kw,kernel", [
    (64, 64, {}, F), (64, 64, VISC, F), (64, 64, dict(precision=abi.PREC_FP32_FLUX), T),
    (64, 64, dict(precision=abi.PREC_FP32_FLUX, **VISC), S), (1000, 300, {}, F), (1001, 300, {}, T),
    (1000, 813, VISC, F), (1000, 816, VISC, S), (2, 140000, {}, F), (2, 160000, {}, T), (4, 196605, VISC, F),
    (4, 196606, VISC, S), (18352, 1, {}, F), (18353, 1, {}, T), (40000, 1, VISC, S)])
def test_built_in_choice_and_round_trip(nx, ny, kw, kernel):
    c = context(nx, ny, **kw)
    ran, setting = c.stage_kernel(), c.stage_tiling()
    assert ran[0] == kernel
    if kernel == F:
        assert ran[1:] == (3, 4)
    c.set_stage_tiling(*setting)
    assert c.stage_kernel() == ran and c.stage_tiling() == setting
    d = context(nx, ny, **kw)
    for rows in (1, 3, 5, 0):  # the strip kernel, by explicit rows and by its own rule
        d.set_stage_tiling(abi.STAGE_STRIP, rows)
        strip = d.stage_kernel()
        assert strip[0] == S and strip[1] == (rows or strip[1])
        d.set_stage_tiling(*d.stage_tiling())
        assert d.stage_kernel() == strip
    d.set_stage_tiling(*setting)
    assert d.stage_kernel() == ran and d.stage_tiling() == setting


@pytest.mark.parametrize("kw", [{}, VISC])
def test_the_reported_tiling_gives_the_same_bits(kw):
    """45 x 20 cells: the face-parallel kernel; the strip form at three rows (no block
    count) is the other kernel, which differs by roundings with viscous terms."""
    rng = np.random.default_rng(1)
    f = rng.uniform(-1.0, 1.0, (4, 20, 45))
    u = cases.prim_to_cons(1.0 + 0.1 * f[0], 0.2 * f[1], 0.2 * f[2], 1.0 + 0.1 * f[3])
    a, b, s = (context(45, 20, **kw) for _ in range(3))
    b.set_stage_tiling(*a.stage_tiling())
    s.set_stage_tiling(abi.STAGE_STRIP, 3)
    assert (a.stage_kernel()[0], b.stage_kernel()[0], s.stage_kernel()[0]) == (F, F, S)
    for c in (a, b, s):
        c.upload(u)
        c.step(3)
    assert np.array_equal(a.download(), b.download())
    assert np.max(np.abs(a.download() - s.download())) < 1e-12
    if not kw:
        assert np.array_equal(a.download(), s.download())


def test_autotuned_setting_and_bodies_and_3d():
    from dev_field_efvm_b200.device import Context

    c = context(512, 512)
    c.upload(cases.prim_to_cons(np.ones((512, 512)), 0.1, 0.1, 1.0))
    c.autotune_stage(2)
    ran, setting = c.stage_kernel(), c.stage_tiling()
    c.set_stage_tiling(*setting)
    assert c.stage_kernel() == ran and c.stage_tiling() == setting
    grid, params, u, ex = cases.cylinder_case(220, 41, muscl=True)
    c = Context(grid, params)
    c.set_cylinders(ex["cylinders"], ex["freestream"])
    assert c.stage_kernel() == (F, 3, 4)
    grid, params, u, ex = cases.vortex_tube_case(16)
    kernel, rows, blocks = Context(grid, params).stage_kernel()
    assert kernel == S and 2 <= rows <= 16 and blocks == 4
