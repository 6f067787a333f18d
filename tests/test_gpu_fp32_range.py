"""FP32 fluxes of gases whose FP32 intermediates lie at the bottom of the normal range
and below it: FP32 reciprocals and reciprocal square roots take subnormal inputs
as long as the result is finite.

HLLC: a face's denominator is about 4 rho^3 a^4 = 7.84 rho p^2 for a gas at rest
(gamma 1.4), which for rho = p = 9e-14 is 5.7e-39, below the smallest normal FP32
number 1.18e-38 (and above 2.9e-39, whose reciprocal is the largest finite one).
Rusanov: p = 1e-39 at rho = 1 makes gamma p / rho subnormal.

The bar against FP64 fluxes is the FP32 form's own, 5e-5 of each variable's scale
after ten steps (a face flux carries about 1e-7); a uniform state has equal fluxes
on all faces and does not change at all."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, cases

pytestmark = pytest.mark.gpu


def box(n=96):
    side = {s: abi.BC_PERIODIC for s in (abi.XLO, abi.XHI, abi.YLO, abi.YHI)}
    return abi.make_grid(n, n, bcs={**side, abi.ZLO: abi.BC_SLIP_WALL, abi.ZHI: abi.BC_SLIP_WALL})


def run(u, steps, form, **kw):
    from dev_field_efvm_b200.device import Context

    c = Context(box(), abi.make_params(**{"cfl": 0.3, "r_gas": 1.0, "reconstruction": abi.RECON_MUSCL, **kw}))
    c.set_stage_tiling(form, 0)
    c.upload(u)
    c.step(steps)
    out = c.download()
    c.close()
    return out


@pytest.mark.parametrize("form", [abi.STAGE_TMA, abi.STAGE_STRIP])
def test_hllc_of_a_thin_gas(form):
    x, y = cases.centroids(box())
    X, Y = np.meshgrid(2.0 * np.pi * x, 2.0 * np.pi * y)
    rho0 = 9e-14
    u = cases.prim_to_cons(rho0 * (1.0 + 0.05 * np.sin(X) * np.cos(Y)), 0.02 * np.sin(Y), 0.02 * np.cos(X), rho0)
    got = run(u, 10, form, precision=abi.PREC_FP32_FLUX)
    want = run(u, 10, form)
    assert np.max(np.abs(got - want)) < 5e-5 * np.max(np.abs(want))
    assert not np.array_equal(got, u)


@pytest.mark.parametrize("form", [abi.STAGE_TMA, abi.STAGE_STRIP])
def test_rusanov_of_a_cold_gas(form):
    u = cases.prim_to_cons(np.ones((96, 96)), 0.0, 0.0, 1e-39)
    assert np.array_equal(run(u, 2, form, precision=abi.PREC_FP32_FLUX, flux_scheme=abi.FLUX_RUSANOV), u)


def test_batch_of_a_thin_gas():
    from dev_field_efvm_b200.device import Batch

    grid = box()
    params = abi.make_params(cfl=0.3, r_gas=1.0, reconstruction=abi.RECON_MUSCL, precision=abi.PREC_FP32_FLUX)
    x, y = cases.centroids(grid)
    X, Y = np.meshgrid(2.0 * np.pi * x, 2.0 * np.pi * y)
    rho0 = 9e-14
    u = cases.prim_to_cons(rho0 * (1.0 + 0.05 * np.sin(X) * np.cos(Y)), 0.02 * np.sin(Y), 0.02 * np.cos(X), rho0)
    b = Batch([grid], params)
    b.upload(0, u)
    b.run(1e30, max_steps=5)
    want = run(u, 5, abi.STAGE_STRIP)
    assert np.max(np.abs(b.download(0) - want)) < 5e-5 * np.max(np.abs(want))
