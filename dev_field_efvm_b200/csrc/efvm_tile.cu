// efvm_tile.cu — the face-parallel stage kernel: one RK substage of a 2-D FP64 case
// with one face per lane.
//
// A block of 2 R + 1 warps covers 31 columns x R rows.  Warps 0 .. R-1 form the
// x faces of one row each (lane l the face on the left of column i0 + l, lane 31
// the last cell's right face), warps R .. 2R the y faces below rows jb .. jb + R.
// Both run the same code: a face reads the four cells along its normal (stride 1
// or one row), limits the two slopes, evaluates one flux and leaves it in shared
// memory.  After one block barrier the x warps own a row of cells each: the
// flux divergence, viscous terms, body force, RK combination and, on a step's
// last stage, the sponge, the ghost refill and the wave-speed maximum, as the
// strip kernel does.
//
// Against the strip form (efvm_kernels.cu), where a lane marches the rows of its
// column and forms both faces of every cell in turn, the chain of dependent FP64
// operations a stage waits for is one face and one epilogue instead of two
// faces per row for three or more rows, which is what bounds grids that do not
// fill the GPU many times over.  Nothing is carried from row to row, so there are
// no shuffles, no halo lanes and no carry to store, and the x and y faces share
// one copy of the flux code; the price is (R + 1) / R y faces per row and a memory
// latency and a barrier per tile, which lose to the TMA-fed form where the grid
// is many waves of tiles (the rule: efvm_plan.h).  us per step, strip or TMA form -> this kernel:
// vortex 64^2 22.6 -> 12.3, 128^2 24.4 -> 14.4, 512^2 57.7 -> 53.7, 768^2 95.7 -> 106;
// cylinder 440x82 first order 42.5 -> 26.7, 1100x205 MUSCL 77.7 -> 68.5, 2200x410
// 203 -> 203.  (Persistent blocks with double-buffered TMA tiles measured 18.5 us at
// 128^2, 69.5 at 1100x205 and 129 at 1003x777, and won only on large viscous grids,
// 4400x820 744 -> 709: dropped.)
//
// R = 3 rows and four resident blocks (28 warps per SM, 72 registers) measured
// fastest over 128^2 to 1100x205 among R = 2 .. 7 and 18 to 30 warps: 1100x205
// 72.6 us per step (the force history included) against 73.4 at R = 4 with 27
// warps, 79.5 at R = 5 with 22 and 92 at R = 4 with 18.
#include <cuda_runtime.h>

#include <algorithm>

#include "efvm_internal.h"
#include "efvm_math.cuh"
#include "efvm_device.cuh"

namespace efvm {

namespace {

// FULL: immersed bodies, body force and sponge compiled in; PXY: fully periodic
// at compile time; LIM: the limiter (MUSCL).
template <int SCHEME, int RECON, bool VISC, bool FULL, bool CORR, int LIM, bool PXY, int R, int MINB>
__global__ void __launch_bounds__(32 * (2 * R + 1), MINB) tile_stage_kernel(const __grid_constant__ StageArgs a) {
    constexpr bool MUSCL = RECON == EFVM_RECON_MUSCL;
    constexpr int W = 2 * R + 1;
    __shared__ double flux[4][W][32];
    // viscous: u, v, T of the tile's cells and the ring around them, row jb - 1 + r, column i0 - 1 + c
    __shared__ double prim[VISC ? 3 : 1][VISC ? R + 2 : 1][VISC ? 34 : 1];
    const Geometry& g = a.g;
    const Physics& ph = a.ph;
    pdl_wait_then_release();
    // read ahead of the state's loads, tested after them: a whole stage of a small
    // grid is a few memory latencies and one chain of arithmetic
    // (the viscous forms have no registers to spare and keep the set-up launch)
    const bool fold = !VISC && a.fold_setup;
    const bool setup = fold && a.stage == 0;
    const int active = a.st->active && !(setup && step_stops(a.st));
    const double dt = setup ? step_dt(ph, a.st) : a.st->dt;
    const long long P = g.plane;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i0 = blockIdx.x * STRIP, jb = blockIdx.y * R;
    if (fold && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        // The step's set-up (step_setup) without a launch of its own.  In stage 1 every
        // block forms dt and the stop decision from fields that this launch does not
        // change -- its own non-physical bits go to flags0 -- and this thread records
        // them; stage 2 merges the bits and switches the wave-speed buffer, which no
        // block of it reads.
        DevState* st = a.st;
        if (setup) {
            if (active) {
                st->dt = dt;
                st->step_par = (int)(st->step & 1ull);
            } else if (st->active) {
                st->active = 0;
                st->done_ns = global_ns();
            }
        } else if (a.stage == 1 && active) {
            if (st->flags0) {
                atomicOr(&st->nonphysical, st->flags0);
                st->flags0 = 0;
            }
            switch_lam(st);
        }
    }
    if (active && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        // RK state machine and clock of update_system, crates/cfd_solver/src/lib.rs:607-621
        DevState* st = a.st;
        if (a.stage >= 2) {
            st->rk_stage = 0;
            st->completed = 1;
            st->step += 1;
            st->time += st->dt;
            if (a.defer_forces) st->forces_pending = 1;
        } else {
            st->rk_stage = a.stage + 1;
            st->completed = 0;
        }
    }
    const bool isx = w < R;                     // warp-uniform
    const int j = jb + (isx ? w : w - R);       // the row, or the row above the y face
    const int i = i0 + lane;
    const double gm1 = ph.gamma - 1.0;
    const bool todo = j < g.ny + (isx ? 0 : 1);  // warp-uniform
    const bool owner = isx && todo && lane < STRIP && i < g.nx;
    const long long o = cidx(g, i, j);
    U4 uc{0.0, 0.0, 0.0, 0.0};                  // x warps: the state of cell (i, j)
    U4 u0{0.0, 0.0, 0.0, 0.0};                  // and U^n there (RK stages 2 and 3)
    bool solid = false, sn[4] = {false, false, false, false};  // the cell, its +x, -x, +y, -y neighbours
    const bool with_u0 = a.stage == 1 || a.stage == 2;
    Q4<double> fx{0.0, 0.0, 0.0, 0.0};
    if (todo) {
        // the last columns' idle lanes repeat a cell inside the ghost ring
        const int il = min(i, isx ? g.nx : g.nx + NG - 1);
        const double* __restrict__ p = a.uin + cidx(g, il, j);
        // cells 0, 1 | 2, 3 about the face, in its frame
        Q4<double> c0{0.0, 0.0, 0.0, 0.0}, c1, c2, c3 = c0;
        if (isx) {
            auto ld = [&](int d) { return Q4<double>{p[d], p[P + d], p[2 * P + d], p[3 * P + d]}; };
            c1 = ld(-1);
            c2 = ld(0);
            if (MUSCL) {
                c0 = ld(-2);
                c3 = ld(1);
            }
        } else {
            auto ld = [&](const double* q) { return Q4<double>{q[0], q[2 * P], q[P], q[3 * P]}; };
            c1 = ld(p - g.pitch);
            c2 = ld(p);
            if (MUSCL) {
                c0 = ld(p - 2 * g.pitch);
                c3 = ld(p + g.pitch);
            }
        }
        if (owner) {
            if (with_u0) u0 = load4(a.u0, P, o);
            if (FULL && a.mask) {
                solid = a.mask[o];
                if (VISC) {
                    sn[0] = a.mask[o + 1];
                    sn[1] = a.mask[o - 1];
                    sn[2] = a.mask[o + g.pitch];
                    sn[3] = a.mask[o - g.pitch];
                }
            }
        }
        Q4<double> L = c1, Rr = c2;
        if constexpr (MUSCL) {
            // Sides on the domain edge that take the cell value (efvm_kernels.cu):
            // the whole edge without a periodic wrap, the far side of the seam
            // unless it is reconstructed; an edge between slabs is interior.
            double fl = 0.5, fr = 0.5;
            const int n = isx ? g.nx : g.ny, k = isx ? il : j;
            if (k == 0 || k == n) {
                const bool per = isx ? (PXY || ph.periodic_x) : (PXY || ph.periodic_y || ph.seam_ylo || ph.seam_yhi);
                const double in = per ? 0.5 : 0.0;
                const double far = per && ph.periodic_seam == EFVM_SEAM_TRUE_PERIODIC ? 0.5 : 0.0;
                if (k == 0 && (isx || !ph.halo_ylo || ph.seam_ylo)) {
                    fl = far;
                    fr = in;
                } else if (k == n && (isx || !ph.halo_yhi || ph.seam_yhi)) {
                    fl = in;
                    fr = far;
                }
            }
            auto face = [&](double q0, double q1, double q2, double q3, double& l, double& r) {
                const double d1 = __dsub_rn(q1, q0), d2 = __dsub_rn(q2, q1), d3 = __dsub_rn(q3, q2);
                double sl, f;
                limited_slope(LIM, d2, d1, fl, sl, f);
                l = __fma_rn(sl, f, q1);
                limited_slope(LIM, d3, d2, fr, sl, f);
                r = __fma_rn(-sl, f, q2);
            };
            face(c0.r, c1.r, c2.r, c3.r, L.r, Rr.r);
            face(c0.mn, c1.mn, c2.mn, c3.mn, L.mn, Rr.mn);
            face(c0.mt, c1.mt, c2.mt, c3.mt, L.mt, Rr.mt);
            face(c0.E, c1.E, c2.E, c3.E, L.E, Rr.E);
        }
        if constexpr (VISC) {
            // u, v, T of the cells the viscous stencil reads: y warp w the row below its
            // face (the last one also the row above), lane 0 of an x warp the cell
            // left of the tile; columns past the grid repeat the last ghost.
            auto put = [&](const U4& u, int r, int c) {
                double vu, vv, t;
                prim_uvt(u, rcp_(u.r), gm1, ph.inv_r_gas, vu, vv, t);
                prim[0][r][c] = vu;
                prim[1][r][c] = vv;
                prim[2][r][c] = t;
            };
            if (!isx) {
                put(U4{c1.r, c1.mt, c1.mn, c1.E}, w - R, lane + 1);
                // the row above the last face of the tile or of the grid
                if (w == 2 * R || j == g.ny) put(U4{c2.r, c2.mt, c2.mn, c2.E}, w - R + 1, lane + 1);
            } else if (lane == 0) {
                put(U4{c1.r, c1.mn, c1.mt, c1.E}, w + 1, 0);
            }
        }
        fx = face_flux<SCHEME, double>(L, Rr, ph.gamma, gm1);
        flux[0][w][lane] = fx.r;
        flux[1][w][lane] = fx.mn;
        flux[2][w][lane] = fx.mt;
        flux[3][w][lane] = fx.E;
        if (isx) uc = U4{c2.r, c2.mn, c2.mt, c2.E};
    }
    __syncthreads();
    if (!isx || !active) return;
    double lam = 0.0;
    if (owner) {
        const double fl[4] = {fx.r, fx.mn, fx.mt, fx.E};
        constexpr int Y[4] = {0, 2, 1, 3};  // plane v of a y flux in its face frame
        double rhs[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            // (F_left - F_right) / dx + (G_below - G_above) / dy, as the strip kernel forms it
            const double part = __dmul_rn(__dsub_rn(fl[v], flux[v][w][lane + 1]), g.inv_x);
            rhs[v] = __fma_rn(__dsub_rn(flux[Y[v]][R + w][lane], flux[Y[v]][R + w + 1][lane]), g.inv_y, part);
        }
        if constexpr (CORR) {
            // learned corrections of the four faces (periodic grid): the
            // x face on the left of a cell, the y face below it
            const long long n = (long long)g.nx * g.ny, c = (long long)j * g.nx + i;
            const long long cr = (long long)j * g.nx + (i + 1 == g.nx ? 0 : i + 1);
            const long long ct = (long long)(j + 1 == g.ny ? 0 : j + 1) * g.nx + i;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const float* cx = a.corr + v * n;
                const float* cy = a.corr + (4 + v) * n;
                rhs[v] += ((double)cx[c] - (double)cx[cr]) * g.inv_x + ((double)cy[c] - (double)cy[ct]) * g.inv_y;
            }
        }
        if (VISC && !solid) {
            // viscous_system, crates/cfd_solver/src/lib.rs:514-557 (z terms vanish in 2-D);
            // a solid neighbour takes (0, 0, T of the cell)
            auto at = [&](int v, int dr, int dc) { return prim[v][w + 1 + dr][lane + 1 + dc]; };
            const double us = at(0, 0, 0), vs = at(1, 0, 0), ts = at(2, 0, 0);
            double lap[3] = {0.0, 0.0, 0.0};
            const double y_im = a.yw[j], y_ip = a.yw[g.ny + j], y_is = a.yw[2 * g.ny + j];
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                const double c = v == 0 ? us : (v == 1 ? vs : ts), wall = v == 2 ? ts : 0.0;
                const double xp = sn[0] ? wall : at(v, 0, 1), xm = sn[1] ? wall : at(v, 0, -1);
                const double yp = sn[2] ? wall : at(v, 1, 0), ym = sn[3] ? wall : at(v, -1, 0);
                lap[v] = (xp - 2.0 * c + xm) * ph.dx_inv2 + ((yp - c) * y_ip - (c - ym) * y_im) * y_is;
            }
            const double mu = viscosity(ph, ts);
            const double kappa = mu * ph.cp_pr;  // thermal_conductivity mu cp / Pr, crates/cfd_eos/src/lib.rs:83-87
            const double fxv = mu * lap[0], fyv = mu * lap[1];
            rhs[1] += fxv;
            rhs[2] += fyv;
            rhs[3] += us * fxv + vs * fyv + kappa * lap[2];
        }
        if (solid) rhs[0] = rhs[1] = rhs[2] = rhs[3] = 0.0;  // zero_solid_rhs, crates/cfd_ibm/src/lib.rs:293-301
        if (FULL && ph.body_force_x != 0.0) {  // crates/cfd_solver/tests/poiseuille_channel_validation.rs:100-118
            rhs[1] += uc.r * ph.body_force_x;
            rhs[3] += ph.body_force_x * uc.mx;
        }
        // Rk3Integrator / EulerIntegrator::substep, crates/cfd_solver/src/integrate.rs:48-101
        const double ucv[4] = {uc.r, uc.mx, uc.my, uc.E};
        double un[4];
        if (with_u0) {
            const double w0 = a.stage == 1 ? 0.75 : (1.0 / 3.0), w1 = a.stage == 1 ? 0.25 : (2.0 / 3.0);
            const double u0v[4] = {u0.r, u0.mx, u0.my, u0.E};
#pragma unroll
            for (int v = 0; v < 4; ++v)
                un[v] = __fma_rn(w1, __fma_rn(rhs[v], dt, ucv[v]), __dmul_rn(w0, u0v[v]));
        } else {
#pragma unroll
            for (int v = 0; v < 4; ++v) un[v] = __fma_rn(rhs[v], dt, ucv[v]);
        }
        U4 nw{un[0], un[1], un[2], un[3]};
        if (FULL && a.completes_step && ph.sponge) sponge_2d(g, ph, i, j, dt, nw);
        if constexpr (CORR) {
            // the network's inputs of this cell for the next stage (nn_prims_kernel forms
            // them only after the state was replaced): a launch less per stage
            const double pu = nw.mx / nw.r, pv = nw.my / nw.r;
            const double pp = (a.prim_gamma - 1.0) * (nw.E - 0.5 * nw.r * (pu * pu + pv * pv));
            a.prims[(long long)j * g.nx + i] = make_float4((float)nw.r - 1.0f, (float)pu, (float)pv, (float)pp - 1.0f);
        }
        store4(a.uout, P, o, nw);
        if (i < NG || i >= g.nx - NG || j < NG || j >= g.ny - NG) {
            write_ghosts<PXY>(g, ph, a.uout, i, j, nw);
            peer_rows(a, g, i, j, nw);
        }
        flag_nonphysical(setup ? &a.st->flags0 : &a.st->nonphysical, nw);
        if (a.completes_step && a.want_cfl) lam = wave_speed(g, ph, nw);
    }
    // wave-speed max for the next step's CFL dt: one atomic per warp
    if (a.completes_step && a.want_cfl) {
        for (int d = 16; d > 0; d >>= 1) lam = fmax(lam, __shfl_xor_sync(0xffffffffu, lam, d));
        if (lane == 0 && lam > 0.0 && lam == lam)
            atomicMax(lam_slot(a.st), (unsigned long long)__double_as_longlong(lam));
    }
}

template <int SCHEME, int RECON, bool VISC, bool FULL, bool CORR, int LIM, bool PXY>
void launch_k(const StageArgs& a, bool pdl, cudaStream_t s) {
    static_assert(TILE_COLS == STRIP, "the launch rule counts the kernel's tiles");
    constexpr int R = TILE_ROWS, MINB = TILE_BLOCKS;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((a.g.nx + STRIP - 1) / STRIP, (a.g.ny + R - 1) / R);
    cfg.blockDim = dim3(32 * (2 * R + 1));
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, tile_stage_kernel<SCHEME, RECON, VISC, FULL, CORR, LIM, PXY, R, MINB>, a);
}

template <int SCHEME, int RECON, int LIM>
void launch_l(const StageArgs& a, bool pdl, cudaStream_t s) {
    const bool full = a.mask != nullptr || a.ph.sponge || a.ph.body_force_x != 0.0;
    const bool pxy = a.ph.periodic_x && a.ph.periodic_y;
    if (a.ph.viscous) launch_k<SCHEME, RECON, true, true, false, LIM, false>(a, pdl, s);
    else if (full) launch_k<SCHEME, RECON, false, true, false, LIM, false>(a, pdl, s);
    else if (pxy) launch_k<SCHEME, RECON, false, false, false, LIM, true>(a, pdl, s);
    else launch_k<SCHEME, RECON, false, false, false, LIM, false>(a, pdl, s);
}

template <int SCHEME>
void launch_s(const StageArgs& a, bool pdl, cudaStream_t s) {
    if (a.ph.reconstruction != EFVM_RECON_MUSCL) launch_l<SCHEME, EFVM_RECON_FIRST_ORDER, EFVM_LIMITER_MINMOD>(a, pdl, s);
    else if (a.ph.limiter == EFVM_LIMITER_MC) launch_l<SCHEME, EFVM_RECON_MUSCL, EFVM_LIMITER_MC>(a, pdl, s);
    else launch_l<SCHEME, EFVM_RECON_MUSCL, EFVM_LIMITER_MINMOD>(a, pdl, s);
}

}  // namespace

int launch_stage_tile(const StageArgs& a, bool pdl, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (a.corr) {  // the learned correction runs with MUSCL + HLLC on periodic grids (checked when it is attached)
        if (a.ph.limiter == EFVM_LIMITER_MC)
            launch_k<EFVM_FLUX_HLLC, EFVM_RECON_MUSCL, false, true, true, EFVM_LIMITER_MC, true>(a, pdl, s);
        else
            launch_k<EFVM_FLUX_HLLC, EFVM_RECON_MUSCL, false, true, true, EFVM_LIMITER_MINMOD, true>(a, pdl, s);
        return 1;
    }
    switch (a.ph.flux_scheme) {
        case EFVM_FLUX_RUSANOV: launch_s<EFVM_FLUX_RUSANOV>(a, pdl, s); break;
        case EFVM_FLUX_HLLC_TEXTBOOK: launch_s<EFVM_FLUX_HLLC_TEXTBOOK>(a, pdl, s); break;
        default: launch_s<EFVM_FLUX_HLLC>(a, pdl, s);
    }
    return 1;
}

}  // namespace efvm
