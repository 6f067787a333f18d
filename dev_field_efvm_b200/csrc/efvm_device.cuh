// efvm_device.cuh — device helpers of the 2-D kernels: cell indexing, programmatic
// launch ordering, the gas model's rounding wrappers, boundary ghosts, the
// wave speed, MUSCL face states and warp shuffles of states.  Included inside
// each translation unit that defines 2-D kernels.
#pragma once

#include <cuda_runtime.h>

#include "efvm_internal.h"
#include "efvm_math.cuh"

namespace efvm {

namespace {

__device__ __forceinline__ long long cidx(const Geometry& g, int i, int j) {
    return (long long)(YO + j) * g.pitch + (XO + i);
}

// Programmatic dependent launch.  The kernels of a step are launched with
// programmatic stream serialization, so a kernel's blocks may be scheduled while
// its predecessor is still draining.  Each such kernel waits for the predecessor
// to complete (and its writes to become visible) before it reads anything, then
// lets its own successor launch.  Without the launch attribute both are no-ops.
__device__ __forceinline__ void pdl_wait_then_release() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Cell centre lo + (i + 0.5) h with one rounding per operation, as the host
// computes it (no FMA), so geometry tests agree bit for bit.
__device__ __forceinline__ double centre(double lo, double h, int i) {
    return __dadd_rn(lo, __dmul_rn((double)i + 0.5, h));
}

// ---- 2-D conserved state in the grid frame ---------------------------------
struct U4 {
    double r, mx, my, E;
};

__device__ __forceinline__ U4 load4(const double* q, long long plane, long long o) {
    return U4{q[o], q[plane + o], q[2 * plane + o], q[3 * plane + o]};
}
// Loads of a stage's inputs.  CG: through L2 only (ld.global.cg), for the
// persistent batch kernel, whose inputs were written earlier in the same launch
// by other blocks (an L1 line of this SM could still hold an older value).
template <bool CG>
__device__ __forceinline__ double gld(const double* p) {
    if constexpr (CG) return __ldcg(p);
    else return *p;
}
template <bool CG>
__device__ __forceinline__ U4 load4g(const double* q, long long plane, long long o) {
    return U4{gld<CG>(q + o), gld<CG>(q + plane + o), gld<CG>(q + 2 * plane + o), gld<CG>(q + 3 * plane + o)};
}
__device__ __forceinline__ void store4(double* q, long long plane, long long o, const U4& u) {
    q[o] = u.r;
    q[plane + o] = u.mx;
    q[2 * plane + o] = u.my;
    q[3 * plane + o] = u.E;
}

// The helpers below (pressure, prim_to_cons, the boundary ghosts, the wave
// speed) are evaluated in more than one kernel on the same state: the stage
// epilogue refills ghosts and takes the CFL maximum, and the stand-alone ghost
// fill and CFL pass do the same after an upload.  A restart must see identical
// values from both, so these round every operation explicitly (no FMA
// contraction, whose choice may differ between inlined copies).
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add_(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub_(double a, double b) { return __dsub_rn(a, b); }

// IdealGas::pressure, crates/cfd_eos/src/lib.rs:61-64 (w = 0)
__device__ __forceinline__ double pressure_d(const U4& u, double gm1) {
    return mul_(gm1, sub_(u.E, mul_(0.5, add_(mul_(u.mx, u.mx), mul_(u.my, u.my))) / u.r));
}

// IdealGas::prim_to_cons (2-D, w = 0), crates/cfd_eos/src/lib.rs:55-59
__device__ __forceinline__ U4 prim_to_cons(double rho, double u, double v, double p, double gm1) {
    const double ke = mul_(mul_(0.5, rho), add_(mul_(u, u), mul_(v, v)));
    return U4{rho, mul_(rho, u), mul_(rho, v), add_(p / gm1, ke)};
}

// Viscosity::mu, crates/cfd_eos/src/lib.rs:108-117 (Sutherland :75-80)
__device__ __forceinline__ double viscosity(const Physics& ph, double t) {
    if (ph.viscosity_model == EFVM_VISC_CONSTANT) return ph.mu;
    const double MU_REF = 1.827e-5, T_REF = 291.15, S = 120.0;
    return MU_REF * pow(t / T_REF, 1.5) * (T_REF + S) / (t + S);
}

// One boundary ghost from its interior neighbour (BoundaryCondition::ghost_at),
// crates/cfd_boundary/src/lib.rs:172-362.  side = 0..3 (XLO, XHI, YLO, YHI).
__device__ __forceinline__ U4 bc_ghost(const DevBC& bc, int side, const U4& in, double gm1) {
    switch (bc.kind) {
        case EFVM_BC_SLIP_WALL:
        case EFVM_BC_SYMMETRY: {
            const double n0 = side < 2 ? (side == 1 ? 1.0 : -1.0) : 0.0;
            const double n1 = side >= 2 ? (side == 3 ? 1.0 : -1.0) : 0.0;
            const double mn = add_(mul_(in.mx, n0), mul_(in.my, n1));
            U4 g = in;
            g.mx = sub_(in.mx, mul_(mul_(2.0, mn), n0));
            g.my = sub_(in.my, mul_(mul_(2.0, mn), n1));
            return g;
        }
        case EFVM_BC_NO_SLIP_WALL:
            return U4{in.r, -in.mx, -in.my, in.E};
        case EFVM_BC_SUPERSONIC_INFLOW: {
            const double ke = mul_(mul_(0.5, bc.rho), add_(add_(mul_(bc.u, bc.u), mul_(bc.v, bc.v)), mul_(bc.w, bc.w)));
            return U4{bc.rho, mul_(bc.rho, bc.u), mul_(bc.rho, bc.v), add_(bc.p / gm1, ke)};
        }
        case EFVM_BC_SUBSONIC_INFLOW: {
            const double p_in = pressure_d(in, gm1);
            const double ke = mul_(mul_(0.5, bc.rho), add_(add_(mul_(bc.u, bc.u), mul_(bc.v, bc.v)), mul_(bc.w, bc.w)));
            return U4{bc.rho, mul_(bc.rho, bc.u), mul_(bc.rho, bc.v), add_(p_in / gm1, ke)};
        }
        case EFVM_BC_PRESSURE_OUTLET: {
            const double inv = 1.0 / in.r;
            const double u = mul_(in.mx, inv), v = mul_(in.my, inv);
            return prim_to_cons(in.r, u, v, bc.p, gm1);
        }
        default:
            return in;
    }
}

// Boundary-ghost refill for the cell (i, j) whose new value is `u`: the Halo
// (periodic wrap) and Boundary phases of the next substage, done by the thread
// that owns the interior source cell (each ghost has exactly one writer).
// PXY: both axes are known to be periodic at compile time (the TMA-fed form
// of fully periodic cases), so the boundary-condition paths are not compiled.
template <bool PXY = false>
__device__ __forceinline__ void write_ghosts(const Geometry& g, const Physics& ph, double* q, int i, int j,
                                             const U4& u) {
    const long long P = g.plane;
    const double gm1 = ph.gamma - 1.0;
    if (PXY || ph.periodic_x) {
        if (i >= g.nx - NG) store4(q, P, cidx(g, i - g.nx, j), u);
        if (i < NG) store4(q, P, cidx(g, i + g.nx, j), u);
    } else {
        if (i == 0) {
            store4(q, P, cidx(g, -1, j), bc_ghost(ph.bc[0], 0, u, gm1));
            if (ph.parabolic_inflow) {
                // parabolic_inflow_system, examples/cylinder_drag_validation/main.rs:151-177
                const double y = centre(g.lo[1], g.h[1], j + g.j_off);
                const double um = ph.inflow_u_max, hh = ph.inflow_height, rho = ph.inflow_rho;
                const double uy = mul_(mul_(mul_(4.0, um), y), sub_(hh, y)) / mul_(hh, hh);
                const double p_in = pressure_d(u, gm1);
                const U4 c = prim_to_cons(rho, uy, 0.0, p_in, gm1);
                store4(q, P, cidx(g, -1, j), c);
                store4(q, P, cidx(g, -2, j), c);
            }
        }
        if (i == g.nx - 1) store4(q, P, cidx(g, g.nx, j), bc_ghost(ph.bc[1], 1, u, gm1));
    }
    if (PXY || ph.periodic_y) {
        if (j >= g.ny - NG) store4(q, P, cidx(g, i, j - g.ny), u);
        if (j < NG) store4(q, P, cidx(g, i, j + g.ny), u);
    } else {
        // a side that faces another slab is filled by the caller's halo exchange
        if (j == 0 && !ph.halo_ylo) store4(q, P, cidx(g, i, -1), bc_ghost(ph.bc[2], 2, u, gm1));
        if (j == g.ny - 1 && !ph.halo_yhi) store4(q, P, cidx(g, i, g.ny), bc_ghost(ph.bc[3], 3, u, gm1));
    }
}

// A slab's two rows next to a side with a halo peer go straight into the
// peer's ghost rows of the same stage's output: rows 0, 1 become the lower
// slab's rows ny_lo, ny_lo + 1, and rows ny - 2, ny - 1 the upper slab's rows
// -2, -1 (the peers share this slab's nx, hence its pitch).  The exchange that
// halo_exchange_forward_all does between stages then happens as the stage
// writes, on this GPU's peer memory path (another slab's buffer on the same
// GPU, or a peer GPU's buffer over NVLink).  Batch cases have no peers.
__device__ __forceinline__ void peer_rows(const StageArgs& a, const Geometry& g, int i, int j, const U4& u) {
    if (a.peer_out[0] && j < NG)
        store4(a.peer_out[0], a.peer_plane[0], (long long)(YO + a.peer_ny[0] + j) * g.pitch + (XO + i), u);
    if (a.peer_out[1] && j >= g.ny - NG)
        store4(a.peer_out[1], a.peer_plane[1], (long long)(YO + j - g.ny) * g.pitch + (XO + i), u);
    // a peer on another GPU reads these rows after the stage: make them visible system-wide
    if ((a.peer_out[0] && j < NG) || (a.peer_out[1] && j >= g.ny - NG)) __threadfence_system();
}
template <class A>
__device__ __forceinline__ void peer_rows(const A&, const Geometry&, int, int, const U4&) {}

// The wave-speed accumulator of the current step: the context's own double
// buffer, or the external slot that slabs max-reduce across GPUs.
__device__ __forceinline__ unsigned long long* lam_slot(DevState* st) {
    return st->ext_lam ? &st->lam_ext : &st->lam[st->lam_idx];
}
// The same slot, its selectors read coherently (the persistent batch kernel).
__device__ __forceinline__ unsigned long long* lam_slot_v(DevState* st) {
    const volatile DevState* v = st;
    return v->ext_lam ? &st->lam_ext : &st->lam[v->lam_idx];
}

// Local max wave speed of cfl_system, crates/cfd_solver/src/lib.rs:647-669.
// The divisions of the reference's formula (by rho, by dx/dy/dz, by R) are taken
// as products with reciprocals (1 / rho once per cell, the others once per
// mesh): the wave speed differs from the reference's by a few ulps, and so
// does dt, far below the step's own error.  The stage epilogue and the
// stand-alone CFL pass both call this function, so they agree bit for bit.
__device__ __forceinline__ double wave_speed(const Geometry& g, const Physics& ph, const U4& u) {
    if (!(u.r > 0.0)) return 0.0;
    const double gm1 = ph.gamma - 1.0;
    const double inv = 1.0 / u.r;
    const double vx = mul_(u.mx, inv), vy = mul_(u.my, inv);
    const double ke = mul_(mul_(0.5, u.r), add_(mul_(vx, vx), mul_(vy, vy)));
    const double p = mul_(gm1, sub_(u.E, ke));
    const double a = sqrt(mul_(mul_(ph.gamma, p), inv));
    double lam = add_(add_(mul_(add_(fabs(vx), a), g.inv_h[0]), mul_(add_(fabs(vy), a), g.inv_h[1])),
                      mul_(add_(0.0, a), g.inv_h[2]));
    if (ph.viscous) {
        const double t = mul_(mul_(p, inv), ph.inv_r_gas);
        const double nu = mul_(viscosity(ph, t), inv);
        lam = add_(lam, mul_(mul_(2.0, nu), ph.cfl_visc_sum));
    }
    return lam;
}

// outlet_sponge_system, examples/cylinder_drag_validation/main.rs:186-229, on one cell.
__device__ __forceinline__ void sponge_2d(const Geometry& g, const Physics& ph, int i, int j, double dt, U4& nw) {
    const double cx = centre(g.lo[0], g.h[0], i);
    if (cx < ph.sponge_x_start) return;
    const double cy = centre(g.lo[1], g.h[1], j + g.j_off);
    const double s = fmin(fmax((cx - ph.sponge_x_start) * ph.sponge_inv_w, 0.0), 1.0);
    const double f = fmin(ph.sponge_sigma * s * s * dt, 1.0);
    const double hh = ph.sponge_height;
    const double uy = 4.0 * ph.sponge_u_max * cy * (hh - cy) / (hh * hh);
    // prim_to_cons(rho, uy, 0, p) with p / (gamma - 1) formed on the host
    const double rho_s = ph.sponge_rho;
    const double ke = mul_(mul_(0.5, rho_s), add_(mul_(uy, uy), mul_(0.0, 0.0)));
    const U4 tg{rho_s, mul_(rho_s, uy), mul_(rho_s, 0.0), add_(ph.sponge_e0, ke)};
    nw.r += f * (tg.r - nw.r);
    nw.mx += f * (tg.mx - nw.mx);
    nw.my += f * (tg.my - nw.my);
    nw.E += f * (tg.E - nw.E);
}

// Flags a non-physical state (rho <= 0, p <= 0, NaN).  p > 0 with rho > 0 is
// 2 E rho > m^2 (no division); a NaN in any component fails one of the two
// tests, so the NaN bit is only looked at once a test has failed.
__device__ __forceinline__ void flag_nonphysical(int* flags, const U4& nw) {
    int bad = 0;
    if (!(nw.r > 0.0)) bad |= 1;
    if (!(2.0 * nw.E * nw.r > nw.mx * nw.mx + nw.my * nw.my)) bad |= 2;
    if (bad) {
        if (nw.r != nw.r || nw.mx != nw.mx || nw.my != nw.my || nw.E != nw.E) bad |= 4;
        atomicOr(flags, bad);
    }
}

// Per-step Setup: dt from the wave-speed max (cfl_system's final lines,
// crates/cfd_solver/src/lib.rs:671-676) or fixed_dt, and the stop test of the
// case drivers' `if t >= T_FINAL break`.
// The stop rule of step_setup: a non-physical state or t >= t_stop ends the run.
template <class S>
__device__ __forceinline__ bool step_stops(S* st) {
    return st->nonphysical || (st->stop_at_t && st->time >= st->t_stop);
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The step's dt: cfl / max wave speed (cfl_system, crates/cfd_solver/src/lib.rs:647-669).
template <class S>
__device__ __forceinline__ double step_dt(const Physics& ph, const S* st) {
    if (ph.fixed_dt > 0.0) return ph.fixed_dt;
    const unsigned long long bits = st->ext_lam ? st->lam_ext : st->lam[st->lam_idx];
    const double lam = __longlong_as_double((long long)bits);
    return lam > 0.0 ? ph.cfl / lam : INFINITY;
}
// The switch of the wave-speed buffer that the step's last stage accumulates into.
template <class S>
__device__ __forceinline__ void switch_lam(S* st) {
    if (st->ext_lam) {  // the slot starts this step's accumulation from zero
        st->lam_ext = 0ull;
        return;
    }
    const int nxt = st->lam_idx ^ 1;
    st->lam[nxt] = 0ull;
    st->lam_idx = nxt;
}

// Per-step set-up (one thread): stop check, dt and the wave-speed buffer.
// S = DevState, or volatile DevState where other blocks of the same launch
// write the state (the persistent batch kernel).
template <class S>
__device__ __forceinline__ void step_setup(const Physics& ph, S* st) {
    if (step_stops(st)) {
        st->active = 0;
        st->done_ns = global_ns();
        return;
    }
    st->dt = step_dt(ph, st);
    st->step_par = (int)(st->step & 1ull);
    switch_lam(st);
}

__device__ __forceinline__ void block_max_atomic(double v, unsigned long long* target) {
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    const int nw = (blockDim.x * blockDim.y + 31) / 32;
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    if (tid < 32) {
        double w = tid < nw ? red[tid] : 0.0;
        for (int o = 16; o > 0; o >>= 1) w = fmax(w, __shfl_xor_sync(0xffffffffu, w, o));
        if (tid == 0 && w > 0.0 && w == w) atomicMax(target, (unsigned long long)__double_as_longlong(w));
    }
}

// A conserved state in the reconstruction precision R, grid frame.
template <class R>
struct V4 {
    R r, mx, my, E;
};
template <class R>
__device__ __forceinline__ V4<R> toR(const U4& u) {
    return V4<R>{R(u.r), R(u.mx), R(u.my), R(u.E)};
}
__device__ __forceinline__ U4 toU4(const V4<double>& u) { return U4{u.r, u.mx, u.my, u.E}; }
__device__ __forceinline__ U4 toU4(const V4<float>& u) { return U4{u.r, u.mx, u.my, u.E}; }
// The state in the frame of an x-face (normal x) or a y-face (normal y).
template <class R>
__device__ __forceinline__ Q4<R> xq(const V4<R>& u) {
    return Q4<R>{u.r, u.mx, u.my, u.E};
}
template <class R>
__device__ __forceinline__ Q4<R> yq(const V4<R>& u) {
    return Q4<R>{u.r, u.my, u.mx, u.E};
}

// The two face states c + s/2 (toward the next cell) and c - s/2 (toward the
// previous one) of a cell, s = lim(p - c, c - m) per conserved variable
// (limited_slope_cons and reconstruct_to_face, crates/cfd_solver/src/lib.rs:199-211,273-286);
// m/c/p are the previous/own/next cells along the face normal.  The FP32 path
// takes the differences in FP32.
//
// fp and fm scale the slope of the two states: 0.5 where the face on that side
// reconstructs this cell, 0 where it takes the cell value itself (a first-order
// side on the domain edge), so the edge faces need no select of whole states.
// c + s fp and c - s fm are each one multiply-add; with fp = fm = 0.5 the
// product is exact, so they are the bits of c + (s/2) and c - (s/2), and with 0
// they are c.
template <class R>
__device__ __forceinline__ R half_slope(int limiter, R m, R c, R p) {
    return limit<R>(limiter, p - c, c - m) * R(0.5);
}
__device__ __forceinline__ double fma_(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fma_(float a, float b, float c) { return fmaf(a, b, c); }
template <class R>
__device__ __forceinline__ void slope_faces(int limiter, const V4<R>& m, const V4<R>& c, const V4<R>& p, R fp, R fm,
                                            V4<R>& plus, V4<R>& minus) {
    const R sr = limit<R>(limiter, p.r - c.r, c.r - m.r), sx = limit<R>(limiter, p.mx - c.mx, c.mx - m.mx);
    const R sy = limit<R>(limiter, p.my - c.my, c.my - m.my), se = limit<R>(limiter, p.E - c.E, c.E - m.E);
    plus = V4<R>{fma_(sr, fp, c.r), fma_(sx, fp, c.mx), fma_(sy, fp, c.my), fma_(se, fp, c.E)};
    minus = V4<R>{fma_(-sr, fm, c.r), fma_(-sx, fm, c.mx), fma_(-sy, fm, c.my), fma_(-se, fm, c.E)};
}
__device__ __forceinline__ void slope_pair(int limiter, double m, double c, double p, double fp, double fm, double& plus,
                                           double& minus) {
    double s, f, g;
    const double fwd = p - c, bwd = c - m;
    limited_slope(limiter, fwd, bwd, fp, s, f);
    limited_slope(limiter, fwd, bwd, fm, s, g);
    plus = fma(s, f, c);
    minus = fma(-s, g, c);
}
template <>
__device__ __forceinline__ void slope_faces<double>(int limiter, const V4<double>& m, const V4<double>& c,
                                                    const V4<double>& p, double fp, double fm, V4<double>& plus,
                                                    V4<double>& minus) {
    slope_pair(limiter, m.r, c.r, p.r, fp, fm, plus.r, minus.r);
    slope_pair(limiter, m.mx, c.mx, p.mx, fp, fm, plus.mx, minus.mx);
    slope_pair(limiter, m.my, c.my, p.my, fp, fm, plus.my, minus.my);
    slope_pair(limiter, m.E, c.E, p.E, fp, fm, plus.E, minus.E);
}
// The same two states with both factors 0.5, as c + h and c - h of one half
// slope h = s/2: the same bits as the factor form.  The FP32-flux forms and
// the batch kernels use this one (the factor form raised their spills).
template <class R>
__device__ __forceinline__ void slope_faces_half(int limiter, const V4<R>& m, const V4<R>& c, const V4<R>& p,
                                                 V4<R>& plus, V4<R>& minus) {
    const R hr = half_slope(limiter, m.r, c.r, p.r), hx = half_slope(limiter, m.mx, c.mx, p.mx);
    const R hy = half_slope(limiter, m.my, c.my, p.my), he = half_slope(limiter, m.E, c.E, p.E);
    plus = V4<R>{c.r + hr, c.mx + hx, c.my + hy, c.E + he};
    minus = V4<R>{c.r - hr, c.mx - hx, c.my - hy, c.E - he};
}
// The slope factor of a side that a face does (0.5) or does not (0) reconstruct.
template <class R>
__device__ __forceinline__ R rec_factor(bool rec) {
    return rec ? R(0.5) : R(0);
}

template <class R>
__device__ __forceinline__ V4<R> shfl_up_v(const V4<R>& u, int d) {
    return V4<R>{__shfl_up_sync(0xffffffffu, u.r, d), __shfl_up_sync(0xffffffffu, u.mx, d),
                 __shfl_up_sync(0xffffffffu, u.my, d), __shfl_up_sync(0xffffffffu, u.E, d)};
}
template <class R>
__device__ __forceinline__ V4<R> shfl_down_v(const V4<R>& u, int d) {
    return V4<R>{__shfl_down_sync(0xffffffffu, u.r, d), __shfl_down_sync(0xffffffffu, u.mx, d),
                 __shfl_down_sync(0xffffffffu, u.my, d), __shfl_down_sync(0xffffffffu, u.E, d)};
}

template <class R>
__device__ __forceinline__ Q4<R> shfl_up_q(const Q4<R>& u, int d) {
    return Q4<R>{__shfl_up_sync(0xffffffffu, u.r, d), __shfl_up_sync(0xffffffffu, u.mn, d),
                 __shfl_up_sync(0xffffffffu, u.mt, d), __shfl_up_sync(0xffffffffu, u.E, d)};
}
template <class R>
__device__ __forceinline__ Q4<R> shfl_down_q(const Q4<R>& u, int d) {
    return Q4<R>{__shfl_down_sync(0xffffffffu, u.r, d), __shfl_down_sync(0xffffffffu, u.mn, d),
                 __shfl_down_sync(0xffffffffu, u.mt, d), __shfl_down_sync(0xffffffffu, u.E, d)};
}

// Primitive (u, v, T) of a state given 1/rho (cons_to_prim, crates/cfd_eos/src/lib.rs:44-53).
__device__ __forceinline__ void prim_uvt(const U4& u, double inv, double gm1, double inv_r_gas, double& vu, double& vv,
                                         double& t) {
    vu = u.mx * inv;
    vv = u.my * inv;
    const double ke = 0.5 * u.r * (vu * vu + vv * vv);
    t = gm1 * (u.E - ke) * inv * inv_r_gas;  // T = p / (rho R), the division by R as a product
}

constexpr int STRIP = 31;  // cells a warp owns per row (lane 31 supplies the right face)
constexpr int WPB = 4;     // warps per block

}  // namespace

}  // namespace efvm
