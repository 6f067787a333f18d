"""The work that users of this library have it do, as timed cases.

Each case goes through the public Python API (``dev_field_efvm_b200.device``):
a context, batch or network is created and loaded once, and a pass advances it
and reads the result back, as a driver does between two outputs.

    listed()            the cases
    draw(rng)           one more case from the same ranges
    prepare(case, seed) the loaded context, batch or network
    run(state)          one pass
    work(case)          bytes and floating-point operations a pass cannot do without
    exact(case, seed)   what a pass on a fresh state returns, in 64 bits, in plain torch

A case is a dict; ``kind`` selects the workload:

    vortex     isentropic vortex on the periodic [0,10]^2 box
    riemann    four-quadrant Riemann problem, transmissive sides, the state
               uploaded from host memory and downloaded again on every pass
    cylinder   the DFG 2D-1 channel: immersed cylinder, viscous terms, parabolic
               inlet, outlet sponge; the force of every substage is read
    tube       a 3-D periodic box: the vortex along z, carried through z
    sphere     resolved sphere drag: 3-D, viscous, immersed sphere, sponge
    batch      many independent small cases advanced together (FP32 fluxes)
    train      one training step of the flux-correction network
    corrected  a periodic flow advanced with the trained flux correction
"""
from __future__ import annotations

import math

import numpy as np
import torch

from dev_field_efvm_b200 import abi, cases, learned

GAMMA = 1.4
N_MARKERS = 2000  # on a sphere


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one step of a small grid at a time, as a driver that couples other
        # physics after every step runs it: latency and launches
        {"name": "vortex_64_step", "kind": "vortex", "nx": 64, "ny": 64, "precision": "fp64", "limiter": "minmod",
         "order": "muscl", "steps": 1},
        # the convergence-study vortex: a small grid over many steps
        {"name": "vortex_128", "kind": "vortex", "nx": 128, "ny": 128, "precision": "fp64", "limiter": "minmod",
         "order": "muscl", "steps": 64},
        # the headline grid between two outputs, in both precisions
        {"name": "vortex_4096", "kind": "vortex", "nx": 4096, "ny": 4096, "precision": "fp64", "limiter": "minmod",
         "order": "muscl", "steps": 50},
        {"name": "vortex_4096_fp32flux", "kind": "vortex", "nx": 4096, "ny": 4096, "precision": "fp32_flux",
         "limiter": "minmod", "order": "muscl", "steps": 50},
        # an odd-sized grid with shocks and open sides whose state lives on the
        # host: uploaded, advanced, downloaded
        {"name": "riemann_1003x777", "kind": "riemann", "nx": 1003, "ny": 777, "precision": "fp64", "limiter": "mc",
         "order": "muscl", "steps": 10},
        # the published drag run (first order) and the finer MUSCL one
        {"name": "cylinder_440x82", "kind": "cylinder", "nx": 440, "ny": 82, "precision": "fp64",
         "limiter": "minmod", "order": "first", "steps": 100},
        {"name": "cylinder_1100x205", "kind": "cylinder", "nx": 1100, "ny": 205, "precision": "fp64",
         "limiter": "minmod", "order": "muscl", "steps": 100},
        # 3-D: the periodic vortex tube, and the published sphere drag run
        {"name": "tube_128", "kind": "tube", "n": 128, "nz": 128, "limiter": "minmod", "steps": 20},
        {"name": "sphere_144x72x72", "kind": "sphere", "nx": 144, "ny": 72, "nz": 72, "order": "first", "steps": 20},
        # an ensemble: 48 grids of 32^2 to 512^2, vortices and Riemann problems
        {"name": "batch_48", "kind": "batch", "cases": 48, "n_max": 512, "steps": 32},
        # the learned correction: a training step of the shipped configuration, and
        # the corrected solver on the coarse grid it was trained for
        {"name": "train_64_b32", "kind": "train", "n": 64, "batch": 32},
        {"name": "corrected_64", "kind": "corrected", "n": 64, "precision": "fp64", "steps": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vortex", "vortex", "riemann", "cylinder", "cylinder", "tube", "sphere", "batch", "train",
                       "corrected"])
    c = {"kind": kind}
    if kind in ("vortex", "riemann"):
        c["nx"], c["ny"] = _log(rng, 40, 3000), _log(rng, 40, 3000)
        c["precision"] = rng.choice(["fp64", "fp64", "fp32_flux"])
        c["limiter"] = rng.choice(["minmod", "mc"])
        c["order"] = rng.choice(["muscl", "muscl", "muscl", "first"])
        c["steps"] = rng.choice([1, 4, 16]) if kind == "vortex" else rng.choice([2, 10])
    elif kind == "cylinder":
        c["nx"] = _log(rng, 330, 1500)
        c["ny"] = max(62, int(c["nx"] * rng.uniform(0.18, 0.2)))
        c["precision"] = rng.choice(["fp64", "fp64", "fp32_flux"])
        c["limiter"] = rng.choice(["minmod", "mc"])
        c["order"] = rng.choice(["muscl", "muscl", "first"])
        c["steps"] = 40
    elif kind == "tube":
        c["n"], c["nz"] = _log(rng, 24, 160), _log(rng, 8, 160)
        c["limiter"] = rng.choice(["minmod", "mc"])
        c["steps"] = 10
    elif kind == "sphere":
        s = rng.uniform(0.6, 1.2)
        c["nx"], c["ny"], c["nz"] = int(144 * s), int(72 * s), int(72 * s)
        c["order"] = rng.choice(["first", "muscl"])
        c["steps"] = 10
    elif kind == "batch":
        c["cases"], c["n_max"], c["steps"] = rng.randint(6, 48), _log(rng, 100, 512), 32
    elif kind == "train":
        c["n"], c["batch"] = 8 * rng.randint(2, 12), rng.randint(1, 40)
    else:
        c["n"], c["precision"], c["steps"] = 8 * rng.randint(3, 32), rng.choice(["fp64", "fp32_flux"]), 16
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _muscl(case):
    return case.get("order", "muscl") == "muscl"


def _limiter(case):
    return abi.LIMITER_MC if case.get("limiter") == "mc" else abi.LIMITER_MINMOD


def _precision(case):
    return abi.PREC_FP32_FLUX if case.get("precision") == "fp32_flux" else abi.PREC_FP64


def _setup(case, seed):
    """(grid, params, extras) of a flow case; extras hold its bodies and vortex."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    recon = abi.RECON_MUSCL if _muscl(case) else abi.RECON_FIRST_ORDER
    if kind == "vortex":
        nx, ny = case["nx"], case["ny"]
        per = abi.BC_PERIODIC
        bcs = {abi.XLO: per, abi.XHI: per, abi.YLO: per, abi.YHI: per,
               abi.ZLO: abi.BC_SLIP_WALL, abi.ZHI: abi.BC_SLIP_WALL}
        grid = abi.make_grid(nx, ny, hi=(10.0, 10.0, 10.0 / nx), bcs=bcs)
        params = abi.make_params(cfl=0.4, reconstruction=recon, limiter=_limiter(case), precision=_precision(case))
        v = abi.make_vortex(beta=rng.uniform(1.0, 5.0), cx0=rng.uniform(3.0, 7.0), cy0=rng.uniform(3.0, 7.0),
                            mean_u=1.0, mean_v=1.0, min_image=True)
        return grid, params, {"vortex": v}
    if kind == "riemann":
        nx, ny = case["nx"], case["ny"]
        grid = abi.make_grid(nx, ny, hi=(1.0, ny / nx, 1.0 / nx),
                             bcs={abi.ZLO: abi.BC_SLIP_WALL, abi.ZHI: abi.BC_SLIP_WALL})
        params = abi.make_params(cfl=0.4, reconstruction=recon, limiter=_limiter(case), precision=_precision(case))
        split = (rng.uniform(0.3, 0.7), rng.uniform(0.3, 0.7) * ny / nx)
        quads = [(rng.uniform(0.1, 2.0), rng.uniform(-1.0, 1.0), rng.uniform(-1.0, 1.0), rng.uniform(0.1, 2.0))
                 for _ in range(4)]
        x, y = cases.centroids(grid)
        return grid, params, {"u": cases.riemann4_state(x, y, split, quads)}
    if kind == "cylinder":
        if _muscl(case):
            grid, params, u, ex = cases.cylinder_baseline_case(case["nx"], case["ny"], limiter=_limiter(case),
                                                               precision=_precision(case))
        else:
            grid, params, u, ex = cases.cylinder_case(case["nx"], case["ny"], precision=_precision(case))
        x, y = cases.centroids(grid)
    elif kind == "tube":
        grid, params, u, ex = cases.vortex_tube_case(
            case["n"], case["nz"], limiter=_limiter(case), beta=rng.uniform(1.0, 5.0),
            centre=(rng.uniform(3.0, 7.0), rng.uniform(3.0, 7.0)))
        ex["u"] = u
        return grid, params, ex
    elif kind == "sphere":
        grid, params, u, ex = cases.sphere_drag_case(case["nx"], case["ny"], case["nz"], muscl=_muscl(case),
                                                     n_markers=N_MARKERS)
        x, y = cases.centroids(grid)
    elif kind == "corrected":
        net, dt = learned.load_trained()
        grid, params = learned.grid_params(case["n"], dt * 64.0 / case["n"])
        params.precision = _precision(case)
        return grid, params, {"u": learned.family_state(case["n"], seed), "net": net}
    else:
        raise ValueError(kind)
    # the two drag cases start from their uniform stream with a small smooth
    # velocity disturbance of the seed's own
    k, ph, amp = rng.integers(1, 5, 2), rng.uniform(0.0, 2.0 * np.pi, 2), rng.uniform(0.002, 0.01)
    d = 1.0 + amp * np.sin(k[0] * 7.0 * x[None, :] + ph[0]) * np.cos(k[1] * 20.0 * y[:, None] + ph[1])
    ke0 = 0.5 * (u[..., 1] ** 2 + u[..., 2] ** 2) / u[..., 0]
    u[..., 1] *= d
    u[..., 4] += 0.5 * (u[..., 1] ** 2 + u[..., 2] ** 2) / u[..., 0] - ke0
    ex["u"] = u
    return grid, params, ex


def _ensemble_sizes(case):
    """The grid sizes of a batch, log-uniform in [32, n_max]; the case's own, whatever the seed."""
    rng = np.random.default_rng(case["cases"])
    return [int(round(math.exp(rng.uniform(math.log(32), math.log(case["n_max"]))))) for _ in range(case["cases"])]


def _ensemble(case, seed):
    """Grids, shared settings and states: even cases vortices, odd ones Riemann problems."""
    rng = np.random.default_rng(seed)
    params = abi.make_params(cfl=0.4, reconstruction=abi.RECON_MUSCL, precision=abi.PREC_FP32_FLUX)
    grids, states = [], []
    for k, n in enumerate(_ensemble_sizes(case)):
        if k % 2 == 0:
            grid, _, u, _ = cases.vortex_case(n, periodic=True, muscl=True, mean=(1.0, 1.0),
                                              beta=rng.uniform(1.0, 5.0),
                                              centre=(rng.uniform(3.0, 7.0), rng.uniform(3.0, 7.0)))
        else:
            grid, _, ex = _setup({"kind": "riemann", "nx": n, "ny": n}, int(rng.integers(1 << 30)))
            u = ex["u"]
        grids.append(grid)
        states.append(u)
    return grids, params, states


def _train_inputs(case, seed):
    net, _ = learned.load_trained()
    n, b = case["n"], case["batch"]
    dx = learned.L / n
    s = np.stack([np.moveaxis(learned.family_state(n, 1000 * seed + k)[..., [0, 1, 2, 4]], -1, 0) for k in range(b)])
    r = np.random.default_rng(seed).standard_normal(s.shape) * (net.out_scale() / dx)
    w = 1.0 / np.mean(r ** 2, axis=(0, 2, 3))
    return net, s, r, dx, w / w.sum() * 4.0


def prepare(case, seed):
    from dev_field_efvm_b200.device import Batch, Context

    kind = case["kind"]
    if kind == "batch":
        grids, params, states = _ensemble(case, seed)
        b = Batch(grids, params)
        for k, u in enumerate(states):
            b.upload(k, u)
        return {"kind": kind, "batch": b, "n": case["cases"], "steps": case["steps"]}
    if kind == "train":
        net, s, r, dx, w = _train_inputs(case, seed)
        return {"kind": kind, "net": net, "s": torch.tensor(s, device="cuda"), "r": torch.tensor(r, device="cuda"),
                "dx": dx, "w": w, "grad": torch.zeros(net.P, dtype=torch.float32, device="cuda")}
    grid, params, ex = _setup(case, seed)
    ctx = Context(grid, params)
    shape = (grid.ny, grid.nx, 5) if grid.nz == 1 else (grid.nz, grid.ny, grid.nx, 5)
    state = {"kind": kind, "ctx": ctx, "steps": case["steps"],
             "out": torch.zeros(shape, dtype=torch.float64, pin_memory=True)}
    if "cylinders" in ex:
        ctx.set_cylinders(ex["cylinders"], ex["freestream"])
    if "spheres" in ex:
        ctx.set_spheres(ex["spheres"], ex["freestream"], ex["n_markers"])
    if kind == "corrected":
        ctx.set_flux_correction(ex["net"])
    if kind == "vortex":
        ctx.init_vortex(ex["vortex"])
    elif kind == "riemann":
        state["u"] = torch.tensor(ex["u"]).pin_memory()
    else:
        ctx.upload(ex["u"])
    return state


def run(state):
    kind = state["kind"]
    if kind == "batch":
        b = state["batch"]
        res = b.run(1.0e9, max_steps=state["steps"])
        return {"u": [b.download(k) for k in range(state["n"])], "time": np.array([r.time for r in res])}
    if kind == "train":
        net = state["net"]
        loss = net.loss_grad(state["s"], state["r"], state["dx"], state["dx"], state["w"], state["grad"])
        net.adam(1.0e-3)
        return {"loss": loss, "grad": state["grad"]}
    ctx, out = state["ctx"], state["out"]
    if kind in ("cylinder", "sphere"):
        info, force = ctx.step(state["steps"], history=True)
        ctx.download(out.numpy())
        return {"u": out, "time": info.time, "force": force}
    if kind == "riemann":
        ctx.upload(state["u"].numpy())
    info = ctx.step(state["steps"])
    ctx.download(out.numpy())
    return {"u": out, "time": info.time}


# Floating-point operations of one cell and one RK stage, the fewest with which
# the method can be written down: per face a limited slope for each variable on
# both sides, two primitive states, the Thornber blend and one HLLC flux, and per
# cell the divergence and the RK combination.
def _stage_flops(axes, muscl, viscous):
    nv = 2 + axes
    face = 90 + 22 * axes + (9 * nv if muscl else 0)
    return axes * face + 8 * nv + (40 * axes if viscous else 0)


def work(case):
    kind = case["kind"]
    if kind == "train":
        b, n = case["batch"], case["n"]
        faces = 2.0 * b * n * n
        macs = 100 * 32 + 32 * 32 + 32 * 4
        # states and residuals in, the gradient out; forward, and backward's two products per layer
        # (none towards the inputs)
        return {"bytes": 2 * 4 * 8.0 * b * n * n + 4 * learned_params(), "flops": faces * 2.0 * (3 * macs - 100 * 32)}
    if kind == "batch":
        cells, axes = float(sum(n * n for n in _ensemble_sizes(case))), 2
    elif kind in ("tube", "sphere"):
        cells, axes = float(case["n"] ** 2 * case["nz"] if kind == "tube" else case["nx"] * case["ny"] * case["nz"]), 3
    else:
        cells, axes = float(case["n"] ** 2 if kind == "corrected" else case["nx"] * case["ny"]), 2
    # a step's stages read U^n and the stage input and write the stage output: 8 states
    # per cell; the result leaves as 5 doubles per cell (and arrives, where it is uploaded)
    state = 8.0 * (2 + axes)
    steps = case["steps"]
    transfers = (2 if kind == "riemann" else 1) * (40.0 + state)
    viscous = kind in ("cylinder", "sphere")
    flops = 3.0 * _stage_flops(axes, _muscl(case), viscous)
    if kind == "corrected":
        flops += 3.0 * 2 * 2 * (100 * 32 + 32 * 32 + 32 * 4)
    return {"bytes": cells * (steps * 8 * state + transfers), "flops": cells * steps * flops}


def learned_params():
    return 32 * 112 + 32 * 32 + 4 * 32 + 32 + 32 + 4


# ---------------------------------------------------------------------------
# The same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
class _Flow:
    """SSP-RK3 of the compressible equations on a uniform box, MUSCL or first
    order, HLLC with the Thornber blend; states are [2 + axes, (nz,) ny, nx]."""

    def __init__(self, grid, params, ex, dev):
        self.axes = 3 if grid.nz > 1 else 2
        self.n = [grid.nx, grid.ny, grid.nz][:self.axes]
        self.h = [(grid.hi[a] - grid.lo[a]) / [grid.nx, grid.ny, grid.nz][a] for a in range(3)]
        self.lo = [grid.lo[a] for a in range(3)]
        self.bc = [grid.bc[s] for s in range(6)]
        self.p, self.g, self.dev = params, params.gamma, dev
        self.muscl = params.reconstruction == abi.RECON_MUSCL
        self.t, self.net, self.solid, self.force = 0.0, None, None, []
        if "net" in ex:
            self.net = _Net(ex["net"], dev)
        self.x = [self.lo[a] + (torch.arange(self.n[a], dtype=torch.float64, device=dev) + 0.5) * self.h[a]
                  for a in range(self.axes)]

    # -- gas model
    def prim(self, u):
        v = u[1:-1] / u[0]
        p = (self.g - 1.0) * (u[-1] - 0.5 * u[0] * (v * v).sum(0))
        return v, p

    def cons(self, r, v, p):
        return torch.cat([r[None], r * v, (p / (self.g - 1.0) + 0.5 * r * (v * v).sum(0))[None]])

    # -- two ghost layers along one axis
    def ghosts(self, u, a):
        d = u.dim() - 1 - a
        n = u.shape[d]
        cut = lambda q, i, m=1: q.narrow(d, i, m)  # noqa: E731
        if self.bc[2 * a].kind == abi.BC_PERIODIC:
            return torch.cat([cut(u, n - 2, 2), u, cut(u, 0, 2)], d)
        out = []
        for side, edge in ((2 * a, cut(u, 0)), (2 * a + 1, cut(u, n - 1))):
            b, q = self.bc[side], edge.clone()
            if b.kind in (abi.BC_SLIP_WALL, abi.BC_SYMMETRY):
                q[1 + a] = -q[1 + a]
            elif b.kind == abi.BC_NO_SLIP_WALL:
                q[1:-1] = -q[1:-1]
            elif b.kind == abi.BC_PRESSURE_OUTLET:
                v, _ = self.prim(edge)
                q = self.cons(edge[0], v, torch.full_like(edge[0], b.p))
            elif b.kind == abi.BC_SUBSONIC_INFLOW:
                _, p = self.prim(edge)
                v = torch.stack([torch.full_like(p, w) for w in (b.u, b.v, b.w)[:self.axes]])
                q = self.cons(torch.full_like(p, b.rho), v, p)
            elif b.kind != abi.BC_SUPERSONIC_OUTFLOW:
                raise ValueError(b.kind)
            if side == 0 and self.p.parabolic_inflow:
                _, p = self.prim(edge)
                hh, um = self.p.inflow_height, self.p.inflow_u_max
                v = torch.zeros_like(edge[1:-1])
                v[0] = (4.0 * um * self.x[1] * (hh - self.x[1]) / (hh * hh))[:, None]
                q = self.cons(torch.full_like(p, self.p.inflow_rho), v, p)
            out.append(q)
        lo, hi = out
        return torch.cat([lo, lo, u, hi, hi], d)

    # -- one numerical flux
    def flux(self, ul, ur, a):
        (vl, pl), (vr, pr) = self.prim(ul), self.prim(ur)
        rl, rr = ul[0], ur[0]
        al, ar = (self.g * pl / rl).sqrt(), (self.g * pr / rr).sqrt()
        z = (torch.maximum((vl * vl).sum(0), (vr * vr).sum(0)).sqrt() / torch.maximum(al, ar)).clamp(max=1.0)
        avg, dv = 0.5 * (vl + vr), 0.5 * z * (vl - vr)
        vl, vr = avg + dv, avg - dv
        ul, ur = self.cons(rl, vl, pl), self.cons(rr, vr, pr)
        sl, sr = torch.minimum(vl[a] - al, vr[a] - ar), torch.maximum(vl[a] + al, vr[a] + ar)
        fl, fr = rl * (sl - vl[a]), rr * (sr - vr[a])
        ss = (pr - pl + fl * vl[a] - fr * vr[a]) / (fl - fr)
        left = (sl >= 0) | (ss >= 0)
        pick = lambda x, y: torch.where(left, x, y)  # noqa: E731
        r, v, p, u, s, f = pick(rl, rr), pick(vl, vr), pick(pl, pr), pick(ul, ur), pick(sl, sr), pick(fl, fr)
        out = u * v[a]
        out[1 + a] += p
        out[-1] += p * v[a]
        rs = f / (s - ss)
        vs = v.clone()
        vs[a] = ss
        es = u[-1] / r + (ss - v[a]) * (ss + p / f)
        star = torch.cat([rs[None], rs * vs, (rs * es)[None]])
        inside = (sl < 0) & (sr >= 0)
        return torch.where(inside, out + s * (star - u), out)

    def slopes(self, w, d):
        n = w.shape[d]
        b, f = w.narrow(d, 1, n - 2) - w.narrow(d, 0, n - 2), w.narrow(d, 2, n - 2) - w.narrow(d, 1, n - 2)
        if self.p.limiter == abi.LIMITER_MC:
            s = torch.minimum(torch.minimum(2 * f.abs(), 2 * b.abs()), 0.5 * (f + b).abs()) * f.sign()
        else:
            s = torch.where(f.abs() < b.abs(), f, b)
        return torch.where(f * b <= 0, torch.zeros_like(s), s)

    def faces(self, u, a):
        """Fluxes of the n + 1 faces along axis a."""
        w, d, n = self.ghosts(u, a), u.dim() - 1 - a, self.n[a]
        l, r = w.narrow(d, 1, n + 1), w.narrow(d, 2, n + 1)
        if self.muscl:
            s = 0.5 * self.slopes(w, d)  # cells -1 .. n
            sl, sr = s.narrow(d, 0, n + 1).clone(), s.narrow(d, 1, n + 1).clone()
            per = self.bc[2 * a].kind == abi.BC_PERIODIC
            true_seam = per and self.p.periodic_seam == abi.SEAM_TRUE_PERIODIC
            if not true_seam:  # the halo side of an edge face is not reconstructed
                sl.narrow(d, 0, 1).zero_()
                sr.narrow(d, n, 1).zero_()
            if not per:
                sl.narrow(d, n, 1).zero_()
                sr.narrow(d, 0, 1).zero_()
            l, r = l + sl, r - sr
        return self.flux(l, r, a)

    def rhs(self, u):
        out = torch.zeros_like(u)
        corr = self.net.corrections(u[None], 0.2)[0] if self.net else None
        for a in range(self.axes):
            f, d, n = self.faces(u, a), u.dim() - 1 - a, self.n[a]
            out -= (f.narrow(d, 1, n) - f.narrow(d, 0, n)) / self.h[a]
            if corr is not None:
                out -= (corr[a].roll(-1, d) - corr[a]) / self.h[a]
        if self.p.viscous:
            self.viscous(u, out)
        if self.solid is not None:
            out[:, self.solid] = 0.0
        return out

    def viscous(self, u, out):
        mu = self.p.mu
        kappa = mu * self.g * self.p.r_gas / (self.g - 1.0) / 0.72

        def vt(q):
            v, p = self.prim(q)
            return torch.cat([v, (p / (q[0] * self.p.r_gas))[None]])

        c = vt(u)
        lap = torch.zeros_like(c)
        for a in range(self.axes):
            d, n = u.dim() - 1 - a, self.n[a]
            w = vt(self.ghosts(u, a))
            for k in (1, 3):
                nb = w.narrow(d, k, n).clone()
                if self.solid is not None:
                    wall = torch.zeros_like(self.solid)
                    m = self.solid.roll(1 if k == 1 else -1, d - 1)
                    wall.narrow(d - 1, 1 if k == 1 else 0, n - 1).copy_(m.narrow(d - 1, 1 if k == 1 else 0, n - 1))
                    nb[:-1, wall] = 0.0
                    nb[-1] = torch.where(wall, c[-1], nb[-1])
                lap += (nb - c) / self.h[a] ** 2
        f = mu * lap[:-1]
        out[1:-1] += f
        out[-1] += (c[:-1] * f).sum(0) + kappa * lap[-1]

    def dt(self, u):
        if self.p.fixed_dt > 0:
            return self.p.fixed_dt
        v, p = self.prim(u)
        a = (self.g * p / u[0]).sqrt()
        lam = a * sum(1.0 / h for h in self.h) + sum(v[k].abs() / self.h[k] for k in range(self.axes))
        if self.p.viscous:
            lam = lam + 2.0 * self.p.mu / u[0] * sum(1.0 / (h * h) for h in self.h)
        return self.p.cfl / float(lam.max())

    # -- immersed body: a circle or a sphere at rest
    def body(self, centre, radius, markers, freestream, shallow):
        ax, dev = self.axes, self.dev
        mesh = torch.meshgrid(*[x for x in reversed(self.x)], indexing="ij")[::-1]
        rel = torch.stack([m - c for m, c in zip(mesh, centre)])
        sd = (rel * rel).sum(0).sqrt() - radius
        self.solid = sd < 0
        mirrored = self.solid
        if shallow:  # only cells with a fluid face neighbour
            buried = self.solid.clone()
            for d in range(ax):
                for s in (1, -1):
                    buried &= self.solid.roll(s, d)
            mirrored = self.solid & ~buried
        self.cells = mirrored.nonzero(as_tuple=True)
        q = rel[(slice(None),) + self.cells]
        r = (q * q).sum(0).sqrt()
        nrm = torch.where(r < 1e-12, torch.tensor([1.0] + [0.0] * (ax - 1), device=dev,
                                                  dtype=torch.float64)[:, None], q / r)
        at = torch.stack([m[self.cells] for m in mesh])
        self.image = self.locate(at + 2.0 * (radius - r) * nrm)
        k = torch.arange(markers, dtype=torch.float64, device=dev)
        if ax == 2:
            th = 2.0 * math.pi * (k + 0.5) / markers
            self.normal = torch.stack([th.cos(), th.sin()])
            self.area = 2.0 * math.pi * radius * self.h[2] / markers
        else:
            z = 1.0 - 2.0 * (k + 0.5) / markers
            rr, phi = (1.0 - z * z).clamp(min=0).sqrt(), math.pi * (3.0 - math.sqrt(5.0)) * k
            self.normal = torch.stack([rr * phi.cos(), rr * phi.sin(), z])
            self.area = 4.0 * math.pi * radius ** 2 / markers
        c = torch.tensor(centre[:ax], device=dev, dtype=torch.float64)[:, None]
        self.probe = self.locate(c + (radius + self.h[0]) * self.normal)
        fs = torch.tensor(freestream, device=dev, dtype=torch.float64)
        self.stagnant = torch.zeros(2 + ax, device=dev, dtype=torch.float64)
        self.stagnant[0], self.stagnant[-1] = fs[0], fs[4] - 0.5 * float((fs[1:4] ** 2).sum()) / fs[0]

    def locate(self, pts):
        """Corner indices and weights of the block of cell centres around each
        point, solid corners left out (the bodies stay clear of the sides)."""
        f = torch.stack([(pts[a] - self.lo[a]) / self.h[a] - 0.5 for a in range(self.axes)])
        lo = f.floor()
        t = f - lo
        corners = []
        for m in range(2 ** self.axes):
            o = [(m >> a) & 1 for a in range(self.axes)]
            idx = tuple((lo[a] + o[a]).long() for a in reversed(range(self.axes)))
            w = torch.ones_like(t[0])
            for a in range(self.axes):
                w = w * (t[a] if o[a] else 1.0 - t[a])
            corners.append((idx, torch.where(self.solid[idx], torch.zeros_like(w), w)))
        return corners

    def sample(self, u, corners):
        acc, total = 0.0, 0.0
        for idx, w in corners:
            q = u[(slice(None),) + idx]
            v, p = self.prim(q)
            acc = acc + w * torch.cat([q[0][None], v, p[None]])
            total = total + w
        return acc / total, total >= 1e-12

    def mirror(self, u):
        s, ok = self.sample(u, self.image)
        q = self.cons(s[0], -s[1:-1], s[-1])
        at = (slice(None),) + self.cells
        u[at] = torch.where(ok, q, u[at])

    def marker_force(self, u):
        s, _ = self.sample(u, self.probe)
        v = s[1:-1]
        vt = v - (v * self.normal).sum(0) * self.normal
        out = torch.zeros(6, dtype=torch.float64, device=self.dev)
        out[:self.axes] = (-s[-1] * self.normal * self.area).sum(1)
        out[3:3 + self.axes] = (self.p.mu * vt / self.h[0] * self.area).sum(1)
        self.force.append(out)

    def sponge(self, u, dt):
        p = self.p
        s = ((self.x[0] - p.sponge_x_start) / (p.sponge_x_end - p.sponge_x_start)).clamp(0.0, 1.0)
        f = (p.sponge_sigma * s * s * dt).clamp(max=1.0)
        v = torch.zeros_like(u[1:-1])
        if self.axes == 2:
            hh = p.sponge_height
            v[0] = (4.0 * p.sponge_u_max * self.x[1] * (hh - self.x[1]) / (hh * hh))[:, None]
        else:
            v[0] = p.sponge_u_max
        r = torch.full_like(u[0], p.sponge_rho)
        return u + f * (self.cons(r, v, torch.full_like(r, p.sponge_p)) - u)

    def step(self, u, dt):
        if self.solid is not None:
            self.mirror(u)
        u0 = u
        for w0, w1 in ((0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)):
            if self.solid is not None and w0:
                self.mirror(u)
            v = u + dt * self.rhs(u)
            u = w0 * u0 + w1 * v if w0 else v
            if self.p.sponge and w0 == 1.0 / 3.0:
                u = self.sponge(u, dt)
            if self.solid is not None:
                self.marker_force(u)
        return u

    def advance(self, u, steps):
        dt = self.dt(u)  # the first step's CFL precedes the geometry
        if self.solid is not None:
            u[:, self.solid] = self.stagnant[:, None]
        for _ in range(steps):
            u = self.step(u, dt)
            self.t += dt
            dt = self.dt(u)
        return u


class _Net:
    """The correction network (100-32-32-4 per face, ReLU) without its BF16 roundings."""

    def __init__(self, net, dev):
        self.p = torch.tensor(net.params(), device=dev, dtype=torch.float64)
        self.scale = net.out_scale()

    def corrections(self, u, sensor=0.0):
        """[B, 2, 4, ny, nx] of states [B, 4, ny, nx], grid frame."""
        w1, w2, w3 = self.p[:3584].reshape(32, 112)[:, :100], self.p[3584:4608].reshape(32, 32), \
            self.p[4608:4736].reshape(4, 32)
        b1, b2, b3 = self.p[4736:4768], self.p[4768:4800], self.p[4800:4804]
        r, vx, vy = u[:, 0], u[:, 1] / u[:, 0], u[:, 2] / u[:, 0]
        p = (GAMMA - 1.0) * (u[:, 3] - 0.5 * r * (vx * vx + vy * vy))
        out = []
        for o in range(2):
            q = torch.stack([r - 1.0, vx if o == 0 else vy, vy if o == 0 else vx, p - 1.0], -1)
            feats = []
            for c in range(-2, 3):
                for a in range(-3, 2):
                    sx, sy = (a, c) if o == 0 else (c, a)
                    feats.append(q.roll((-sy, -sx), (1, 2)))
            h = torch.relu(torch.cat(feats, -1) @ w1.T + b1)
            y = (torch.relu(h @ w2.T + b2) @ w3.T + b3) * self.scale
            if sensor > 0:
                pl = p.roll(1, 2 if o == 0 else 1)
                y = torch.where(((p - pl).abs() > sensor * torch.minimum(p, pl))[..., None], torch.zeros_like(y), y)
            out.append(torch.stack([y[..., 0], y[..., 1 + o], y[..., 2 - o], y[..., 3]], 1))
        return torch.stack(out, 1)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _planes(u, dev):
    """[..., 5] conserved states as [nv, ...], without rho_w on a 2-D grid."""
    q = torch.as_tensor(np.ascontiguousarray(np.moveaxis(u, -1, 0)), device=dev)
    return q if q.dim() == 4 else q[[0, 1, 2, 4]]


def _cells(q):
    """The layout of a downloaded state."""
    if q.shape[0] == 4:
        q = torch.stack([q[0], q[1], q[2], torch.zeros_like(q[0]), q[3]])
    return q.movedim(0, -1).contiguous().cpu()


def _vortex_planes(v, flow, dev):
    X, Y = flow.x[0][None, :], flow.x[1][:, None]
    dx, dy = X - v.cx0, Y - v.cy0
    dx, dy = dx - v.len_x * (dx / v.len_x).round(), dy - v.len_y * (dy / v.len_y).round()
    r2 = dx * dx + dy * dy
    f = v.beta / (2.0 * math.pi) * (0.5 * (1.0 - r2)).exp()
    temp = 1.0 - (GAMMA - 1.0) * v.beta ** 2 / (8.0 * GAMMA * math.pi ** 2) * (1.0 - r2).exp()
    r = temp ** (1.0 / (GAMMA - 1.0))
    return flow.cons(r, torch.stack([v.mean_u - f * dy, v.mean_v + f * dx]), r ** GAMMA)


def exact(case, seed):
    dev, kind = _device(), case["kind"]
    if kind == "train":
        net, s, r, dx, w = _train_inputs(case, seed)
        n = _Net(net, dev)
        n.p.requires_grad_(True)
        c = n.corrections(torch.tensor(s, device=dev))
        div = (c[:, 0].roll(-1, 3) - c[:, 0]) / dx + (c[:, 1].roll(-1, 2) - c[:, 1]) / dx
        e = torch.tensor(r, device=dev) + div
        loss = (torch.tensor(w, device=dev) * (e * e).mean((0, 2, 3))).sum()
        loss.backward()
        return {"loss": float(loss.detach()), "grad": n.p.grad}
    if kind == "batch":
        grids, params, states = _ensemble(case, seed)
        out, times = [], []
        for k, (g, u) in enumerate(zip(grids, states)):
            f = _Flow(g, params, {}, dev)
            # the small grids would take as long as the large ones: some of each size stand for all
            out.append(_cells(f.advance(_planes(u, dev), case["steps"])) if k % 4 == 0 else None)
            times.append(f.t)
        return {"u": out, "time": None}
    grid, params, ex = _setup(case, seed)
    f = _Flow(grid, params, ex, dev)
    if "cylinders" in ex:
        cx, cy, r = ex["cylinders"][0]
        f.body((cx, cy), r, 64, ex["freestream"], False)
    if "spheres" in ex:
        s = ex["spheres"][0]
        f.body((s.cx, s.cy, s.cz), s.radius, ex["n_markers"], ex["freestream"], True)
    u = _vortex_planes(ex["vortex"], f, dev) if kind == "vortex" else _planes(ex["u"], dev)
    out = {"u": _cells(f.advance(u, case["steps"])), "time": f.t}
    if f.force:
        out["force"] = torch.stack(f.force).cpu()
    return out
