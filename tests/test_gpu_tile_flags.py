"""The non-physical flag of the face-parallel stages when one RK stage alone leaves a
non-physical cell: the later stages average the cell back to a physical state, so
only the flag of that stage can report it.  Stage 1, which does the step's set-up
itself, records it beside the flag that its blocks still read, and stage 2 merges
the two.  Whole steps from the graph against single substeps,
which use the separate set-up launch."""
from __future__ import annotations

import numpy as np
import pytest

from dev_field_efvm_b200 import abi, cases

pytestmark = pytest.mark.gpu
N = 8


def case(seed):
    """A low-pressure spot between jets, stepped beyond the CFL limit (textbook HLLC)."""
    r = np.random.default_rng(seed)
    recon, _ = int(r.integers(0, 2)), r.integers(0, 3)
    rho, ux, p = np.ones((N, N)), np.zeros((N, N)), np.ones((N, N))
    rho[4, 3:6] = r.uniform(0.2, 2, 3)
    ux[4, 2:7] = r.uniform(-1.5, 1.5, 5)
    p[4, 3:6] = 10 ** r.uniform(-2.5, 0.3, 3)
    bcs = {s: abi.BC_PERIODIC for s in (abi.XLO, abi.XHI, abi.YLO, abi.YHI)}
    grid = abi.make_grid(N, N, hi=(float(N), float(N), 1.0),
                         bcs=bcs | {abi.ZLO: abi.BC_SLIP_WALL, abi.ZHI: abi.BC_SLIP_WALL})
    params = abi.make_params(cfl=0.4, r_gas=1.0, reconstruction=recon, flux_scheme=abi.FLUX_HLLC_TEXTBOOK,
                             fixed_dt=r.uniform(0.1, 0.9))
    return grid, params, cases.prim_to_cons(rho, ux, 0.0, p)


def physical(u):
    p = 0.4 * (u[..., 4] - 0.5 * (u[..., 1] ** 2 + u[..., 2] ** 2) / u[..., 0])
    return bool(np.all(u[..., 0] > 0.0) and np.all(p > 0.0))


# the RK stage (None: no stage) whose output alone is non-physical in the CPU oracle, with
# |rho| and |p| of every cell and stage at least 0.04, far above the forms' differences
CASES = [(0, 10), (0, 11), (0, 15), (1, 329), (1, 506), (1, 541), (2, 658), (2, 780), (2, 855), (None, 1), (None, 2)]


@pytest.mark.parametrize("stage,seed", CASES)
def test_one_stage_alone_is_reported(stage, seed):
    from dev_field_efvm_b200.device import Context, EfvmError

    grid, params, u = case(seed)
    whole, parts = Context(grid, params), Context(grid, params)
    assert whole.stage_kernel()[0] == abi.KERNEL_FACES
    whole.upload(u)
    parts.upload(u)
    for k in range(3):
        parts.substep()
        assert physical(parts.download()) == (k != stage), k
    if stage is None:
        whole.step(1)
        assert parts.solver_state().step == 1
    else:
        with pytest.raises(EfvmError) as e:
            whole.step(3)  # the next step's set-up stops the run
        assert e.value.code == abi.ERR_NONPHYSICAL
        with pytest.raises(EfvmError):
            parts.solver_state()
    assert np.array_equal(whole.download(), parts.download())
