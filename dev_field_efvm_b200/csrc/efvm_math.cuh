// efvm_math.cuh — the gas model, numerical fluxes and limiters on the device,
// templated on the arithmetic type R (double for the plain path, float for the
// FP32-flux path).  Each function restates the reference routine it cites
// (crates/cfd_eos/src/lib.rs, crates/cfd_riemann/src/lib.rs,
// crates/cfd_solver/src/lib.rs) with the same evaluation order; the compiler
// may fuse a multiply and an add into one FMA, which moves results by at most
// an ulp per operation.
//
// 2-D specialisation: states carry (rho, m_n, m_t, E) in the frame of the face
// normal; rho_w and w are identically zero, so every `+ w*w` / `+ rho_w^2`
// term of the 3-D formulas adds an exact zero and is dropped.
#pragma once

#include <cuda_runtime.h>

namespace efvm {

template <class R>
struct Q4 {
    R r, mn, mt, E;
};

__device__ __forceinline__ double sqrt_(double x) { return sqrt(x); }
__device__ __forceinline__ float sqrt_(float x) { return sqrtf(x); }
__device__ __forceinline__ double fmax_(double a, double b) { return fmax(a, b); }
__device__ __forceinline__ float fmax_(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double fmin_(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ float fmin_(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ double fabs_(double a) { return fabs(a); }
__device__ __forceinline__ float fabs_(float a) { return fabsf(a); }

// Reciprocal from the PTX approximate reciprocal rcp.approx.ftz.f64 (a seed r0
// with relative error e = 1 - b r0 of about 2^-22) and one third-order step of
// the series 1/b = r0 / (1 - e) = r0 (1 + e + e^2 + ...): r0 + r0 (e + e^2)
// leaves a relative error of e^3 (about 2^-66) before the final rounding, the
// accuracy of two Newton steps at one operation less.  Branch-free; denormals
// flush to zero (the flow states here are far from that range).
__device__ __forceinline__ double rcp_(double b) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    const double e = fma(-b, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
// FP32: the library functions, which also take subnormal arguments: thin gases reach
// them (den X in hllc_flux is about 4 rho^3 a^4).  The .ftz instructions give the same
// bits for normal arguments but infinity below them; used throughout they ran 4 %
// faster (FP32-flux step at 4096^2: 1.380 against 1.437 ms).  Taking them first and repeating a flux
// that is not finite with these functions was no faster (1.436 to 1.496 ms).
__device__ __forceinline__ float rcp_(float b) { return __fdividef(1.0f, b); }
// 1/sqrt(x) from the PTX approximate rsqrt.approx.ftz.f64 seed y0 and one
// third-order step of the binomial series 1/sqrt(x) = y0 (1 - e)^(-1/2) with
// e = 1 - x y0^2: y0 + y0 e (1/2 + 3e/8), relative error about 5e^3/16 before
// rounding (the seed's e is about 2^-21), as accurate as two Newton steps.
__device__ __forceinline__ double rsqrt_(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}
__device__ __forceinline__ float rsqrt_(float x) { return rsqrtf(x); }
// 1/sqrt(x) of a normal x >= normal_min: the instruction (the guarded product of
// hllc_flux; 440x82 cylinder with FP32 fluxes 45.2 -> 44.0 us per step).
__device__ __forceinline__ float rsqrt_normal(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// The smallest normal value: the .ftz seeds of the FP64 functions flush anything
// below it to zero (and return infinity for it).
template <class R>
__device__ __forceinline__ R normal_min();
template <>
__device__ __forceinline__ double normal_min<double>() { return 2.2250738585072014e-308; }
template <>
__device__ __forceinline__ float normal_min<float>() { return 1.17549435e-38f; }

// Gas-dynamic quantities of one face state, each computed once per face side:
// 1/rho, normal and tangential velocity, |v|^2, pressure and sound speed
// (IdealGas::cons_to_prim / pressure / sound_speed, crates/cfd_eos/src/lib.rs:44-68,
// with the kinetic energy taken from the velocities and one reciprocal of rho).
template <class R>
struct Side {
    R inv, un, ut, q, p, a;
};
template <class R>
__device__ __forceinline__ Side<R> side_with(const Q4<R>& u, R inv, R gamma, R gm1) {
    Side<R> s;
    s.inv = inv;
    s.un = u.mn * s.inv;
    s.ut = u.mt * s.inv;
    s.q = s.un * s.un + s.ut * s.ut;
    s.p = gm1 * (u.E - R(0.5) * u.r * s.q);
    const R a2 = gamma * s.p * s.inv;
    s.a = a2 * rsqrt_(a2);  // sqrt(a2); NaN for a non-physical p <= 0, which the stage flags
    return s;
}
// Both sides of a face, with 1/rho_L = rho_R w and 1/rho_R = rho_L w from one
// reciprocal w = 1/(rho_L rho_R) (a few ulps from the two separate reciprocals).
template <class R>
__device__ __forceinline__ void sides_of(const Q4<R>& L, const Q4<R>& Rr, R gamma, R gm1, Side<R>& l, Side<R>& r) {
    const R w = rcp_(L.r * Rr.r);
    l = side_with(L, Rr.r * w, gamma, gm1);
    r = side_with(Rr, L.r * w, gamma, gm1);
}

// physical_flux_inline along the face normal for a state with known normal
// velocity and pressure, crates/cfd_riemann/src/lib.rs:21-43.
template <class R>
__device__ __forceinline__ Q4<R> physical_flux(R rho, R un, R ut, R E, R p) {
    const R m = rho * un;
    Q4<R> f;
    f.r = m;
    f.mn = m * un + p;
    f.mt = (rho * ut) * un;
    f.E = (E + p) * un;
    return f;
}

// ---- FP64 fluxes ------------------------------------------------------------
// Every operation of the FP64 fluxes is rounded explicitly (the compiler neither
// fuses nor splits them), so a face formed by different kernels, or by two
// warps of one, has the same bits whatever code surrounds it.
struct SideD {
    double un, ut, q, p, a2, a;
};
__device__ __forceinline__ SideD side_d(const Q4<double>& u, double inv, double gamma, double gm1) {
    SideD s;
    s.un = __dmul_rn(u.mn, inv);
    s.ut = __dmul_rn(u.mt, inv);
    s.q = __fma_rn(s.un, s.un, __dmul_rn(s.ut, s.ut));
    s.p = __dmul_rn(gm1, __fma_rn(__dmul_rn(-0.5, u.r), s.q, u.E));
    s.a2 = __dmul_rn(__dmul_rn(gamma, s.p), inv);
    s.a = __dmul_rn(s.a2, rsqrt_(s.a2));  // NaN for a non-physical p <= 0, which the stage flags
    return s;
}
__device__ __forceinline__ void sides_d(const Q4<double>& L, const Q4<double>& R, double gamma, double gm1, SideD& l,
                                        SideD& r) {
    const double w = rcp_(__dmul_rn(L.r, R.r));
    l = side_d(L, __dmul_rn(R.r, w), gamma, gm1);
    r = side_d(R, __dmul_rn(L.r, w), gamma, gm1);
}
// physical_flux_inline, crates/cfd_riemann/src/lib.rs:21-43
__device__ __forceinline__ Q4<double> physical_flux_d(double rho, double un, double ut, double E, double p) {
    Q4<double> f;
    f.r = __dmul_rn(rho, un);
    f.mn = __fma_rn(f.r, un, p);
    f.mt = __dmul_rn(f.r, ut);
    f.E = __dmul_rn(__dadd_rn(E, p), un);
    return f;
}
// Rusanov::flux_inline, crates/cfd_riemann/src/lib.rs:222-240
__device__ __forceinline__ Q4<double> rusanov_flux_d(const Q4<double>& L, const Q4<double>& R, double gamma,
                                                     double gm1) {
    SideD l, r;
    sides_d(L, R, gamma, gm1, l, r);
    const Q4<double> fl = physical_flux_d(L.r, l.un, l.ut, L.E, l.p);
    const Q4<double> fr = physical_flux_d(R.r, r.un, r.ut, R.E, r.p);
    const double hl = __dmul_rn(-0.5, fmax(__dadd_rn(fabs(l.un), l.a), __dadd_rn(fabs(r.un), r.a)));
    auto mix = [&](double a, double b, double ul, double ur) {
        return __fma_rn(hl, __dsub_rn(ur, ul), __dmul_rn(0.5, __dadd_rn(a, b)));
    };
    return Q4<double>{mix(fl.r, fr.r, L.r, R.r), mix(fl.mn, fr.mn, L.mn, R.mn), mix(fl.mt, fr.mt, L.mt, R.mt),
                      mix(fl.E, fr.E, L.E, R.E)};
}
// Hllc::flux_with_thornber + thornber_reconstruct + star_state,
// crates/cfd_riemann/src/lib.rs:395-506,619-644, in an equivalent form:
//  * the Thornber blend keeps rho and the internal energy, hence p and a (the
//    reference's cached path relies on the same identity, :586-588), and the
//    blended velocities are used directly;
//  * the upwind side K (left for s_l >= 0 or s_* >= 0, else right) is selected
//    first.  In the star regions the flux is the star state's physical flux,
//    which equals F_K + s_K (U*_K - U_K): with f_K = rho_K (s_K - u_K),
//    rho* = f_K / (s_K - s_*), m = rho* s_*, p* = p_K + f_K (s_* - u_K),
//    E* = ((s_K - u_K) E_K - p_K u_K + p* s_*) / (s_K - s_*),
//    F = (m, m s_* + p*, m t_K, (E* + p*) s_*);
//  * s_* = n/d and 1/(s_K - s_*) = d/(s_K d - n) come from one reciprocal of
//    d (s_K d - n), and only in the star regions: elsewhere the sign of s_* is
//    read from the sign of n d;
//  * a_max^2 is the larger a^2, a side without a positive one left out (as the
//    maximum of the sound speeds leaves out a NaN).
template <bool THORNBER>
__device__ __forceinline__ Q4<double> hllc_flux_d(const Q4<double>& L, const Q4<double>& R, double gamma, double gm1) {
    SideD l, r;
    sides_d(L, R, gamma, gm1, l, r);
    double lcn = l.un, lct = l.ut, rcn = r.un, rct = r.ut, ELc = L.E, ERc = R.E;
    if (THORNBER) {
        // z = min(|v|max / a_max, 1) as vmax2 / sqrt(vmax2 a_max^2): one reciprocal square
        // root.  Where vmax2 a_max^2 is below the normal range (round-off velocities
        // near 1e-157 in still gas), z is taken as 0: the reference's z there is
        // about 1e-160 and scales velocity differences of the same size, far below
        // any representable change of the flux.
        const double vmax2 = l.q > r.q ? l.q : r.q;
        const double amax2 = l.a2 > r.a2 ? l.a2 : r.a2;
        const double prod = __dmul_rn(vmax2, amax2);
        double hz = __dmul_rn(__dmul_rn(0.5, vmax2), rsqrt_(prod));
        hz = prod >= normal_min<double>() ? hz : 0.0;
        hz = vmax2 >= amax2 && amax2 > 0.0 ? 0.5 : hz;
        const double avgn = __dmul_rn(0.5, __dadd_rn(l.un, r.un)), avgt = __dmul_rn(0.5, __dadd_rn(l.ut, r.ut));
        const double dun = __dsub_rn(l.un, r.un), dut = __dsub_rn(l.ut, r.ut);
        lcn = __fma_rn(hz, dun, avgn);
        lct = __fma_rn(hz, dut, avgt);
        rcn = __fma_rn(-hz, dun, avgn);
        rct = __fma_rn(-hz, dut, avgt);
        ELc = __fma_rn(__dmul_rn(0.5, L.r), __fma_rn(lcn, lcn, __fma_rn(lct, lct, -l.q)), L.E);
        ERc = __fma_rn(__dmul_rn(0.5, R.r), __fma_rn(rcn, rcn, __fma_rn(rct, rct, -r.q)), R.E);
    }
    const double s_l = fmin(__dsub_rn(lcn, l.a), __dsub_rn(rcn, r.a));
    const double s_r = fmax(__dadd_rn(lcn, l.a), __dadd_rn(rcn, r.a));
    const double fac_l = __dmul_rn(L.r, __dsub_rn(s_l, lcn));
    const double fac_r = __dmul_rn(R.r, __dsub_rn(s_r, rcn));
    const double num = __fma_rn(-fac_r, rcn, __fma_rn(fac_l, lcn, __dsub_rn(r.p, l.p)));
    const double den = __dsub_rn(fac_l, fac_r);
    // s_* = num / den >= 0 without the division (false for den = 0 or NaN)
    const bool star_nonneg = __dmul_rn(num, den) >= 0.0 && den != 0.0;
    const bool useL = (s_l >= 0.0) || star_nonneg;
    const double uK = useL ? lcn : rcn;
    const double tK = useL ? lct : rct;
    const double EK = useL ? ELc : ERc;
    const double pK = useL ? l.p : r.p;
    if (s_l < 0.0 && (star_nonneg || s_r >= 0.0)) {  // one of the two star regions
        const double sK = useL ? s_l : s_r;
        const double facK = useL ? fac_l : fac_r;
        const double Y = __fma_rn(sK, den, -num);
        const double w = rcp_(__dmul_rn(den, Y));
        const double s_star = __dmul_rn(num, __dmul_rn(Y, w));
        const double inv = __dmul_rn(den, __dmul_rn(den, w));  // 1 / (s_K - s_*)
        const double pS = __fma_rn(facK, __dsub_rn(s_star, uK), pK);
        Q4<double> f;
        f.r = __dmul_rn(__dmul_rn(facK, inv), s_star);
        f.mn = __fma_rn(f.r, s_star, pS);
        f.mt = __dmul_rn(f.r, tK);
        const double eS = __fma_rn(pS, s_star, __fma_rn(__dsub_rn(sK, uK), EK, -__dmul_rn(pK, uK)));
        f.E = __dmul_rn(__fma_rn(eS, inv, pS), s_star);
        return f;
    }
    return physical_flux_d(useL ? L.r : R.r, uK, tK, EK, pK);
}

// Rusanov::flux_inline, crates/cfd_riemann/src/lib.rs:222-240
template <class R>
__device__ __forceinline__ Q4<R> rusanov_flux(const Q4<R>& L, const Q4<R>& Rr, R gamma, R gm1) {
    Side<R> l, r;
    sides_of(L, Rr, gamma, gm1, l, r);
    const Q4<R> fl = physical_flux(L.r, l.un, l.ut, L.E, l.p);
    const Q4<R> fr = physical_flux(Rr.r, r.un, r.ut, Rr.E, r.p);
    const R hl = R(0.5) * fmax_(fabs_(l.un) + l.a, fabs_(r.un) + r.a);
    Q4<R> f;
    f.r = R(0.5) * (fl.r + fr.r) - hl * (Rr.r - L.r);
    f.mn = R(0.5) * (fl.mn + fr.mn) - hl * (Rr.mn - L.mn);
    f.mt = R(0.5) * (fl.mt + fr.mt) - hl * (Rr.mt - L.mt);
    f.E = R(0.5) * (fl.E + fr.E) - hl * (Rr.E - L.E);
    return f;
}

// Hllc::flux_with_thornber + thornber_reconstruct + star_state,
// crates/cfd_riemann/src/lib.rs:395-506,619-644, in an equivalent form that
// evaluates each quantity once:
//  * the Thornber blend keeps rho and the internal energy, hence p and a, so
//    the pressures and sound speeds of the blended states are those of the
//    inputs (the reference's cached path relies on the same identity, :586-588);
//  * the blended normal/tangential velocities are used directly instead of
//    re-dividing the rebuilt momenta by rho;
//  * the upwind side K (left for s_l >= 0 or s_* >= 0, else right) is selected
//    first and one star state is built, F = F(U_K) + s_K (U*_K - U_K), with
//    rho_* = f_K/(s_K - s_*) and p_K/(rho_K (s_K - u_K)) = p_K/f_K where
//    f_K = rho_K (s_K - u_K) is the same factor that enters s_*;
//  * s_* = n/d is only formed on the faces that need its value (the star
//    regions); elsewhere its sign is read from the signs of n and d.  Where it
//    is formed, s_* and 1/(f_K (s_K - s_*)) = d/(f_K (s_K d - n)) come from one
//    reciprocal of d f_K (s_K d - n).
// The results agree with the literal evaluation to a few ulps.
template <class R, bool THORNBER>
__device__ __forceinline__ Q4<R> hllc_flux(const Q4<R>& L, const Q4<R>& Rr, R gamma, R gm1) {
    Side<R> l, r;
    sides_of(L, Rr, gamma, gm1, l, r);
    R lcn = l.un, lct = l.ut, rcn = r.un, rct = r.ut, ELc = L.E, ERc = Rr.E;
    if (THORNBER) {
        const R vmax2 = fmax_(l.q, r.q);
        const R amax = fmax_(l.a, r.a);
        // z = min(|v|max / a_max, 1) as vmax2 / sqrt(vmax2 a_max^2): one reciprocal square
        // root.  Where vmax2 a_max^2 is below the normal range (round-off velocities
        // near 1e-157 in still gas), z is taken as 0: the reference's z there is
        // about 1e-160 and scales velocity differences of the same size, far below
        // any representable change of the flux.
        const R amax2 = amax * amax;
        const R prod = vmax2 * amax2;
        const R z = (vmax2 >= amax2) ? R(1) : (prod >= normal_min<R>() ? vmax2 * rsqrt_normal(prod) : R(0));
        const R avgn = R(0.5) * (l.un + r.un), avgt = R(0.5) * (l.ut + r.ut);
        const R hz = R(0.5) * z;
        const R dvn = hz * (l.un - r.un), dvt = hz * (l.ut - r.ut);
        lcn = avgn + dvn;
        lct = avgt + dvt;
        rcn = avgn - dvn;
        rct = avgt - dvt;
        ELc = L.E + R(0.5) * L.r * ((lcn * lcn + lct * lct) - l.q);
        ERc = Rr.E + R(0.5) * Rr.r * ((rcn * rcn + rct * rct) - r.q);
    }
    const R s_l = fmin_(lcn - l.a, rcn - r.a);
    const R s_r = fmax_(lcn + l.a, rcn + r.a);
    const R fac_l = L.r * (s_l - lcn);
    const R fac_r = Rr.r * (s_r - rcn);
    const R num = (r.p - l.p) + fac_l * lcn - fac_r * rcn;
    const R den = fac_l - fac_r;
    // s_* = num / den >= 0 without the division (false for den = 0 or NaN)
    const bool star_nonneg = den > R(0) ? num >= R(0) : (den < R(0) ? num <= R(0) : false);
    const bool useL = (s_l >= R(0)) || star_nonneg;
    const R rK = useL ? L.r : Rr.r;
    const R uK = useL ? lcn : rcn;
    const R tK = useL ? lct : rct;
    const R EK = useL ? ELc : ERc;
    const R pK = useL ? l.p : r.p;
    const R iK = useL ? l.inv : r.inv;
    Q4<R> f = physical_flux(rK, uK, tK, EK, pK);
    if (s_l < R(0) && (star_nonneg || s_r >= R(0))) {  // one of the two star regions
        const R sK = useL ? s_l : s_r;
        const R facK = useL ? fac_l : fac_r;
        // s_* = num/den and inv = 1/(f_K d_K), d_K = s_K - s_*, from one reciprocal;
        // rho_* = f_K / d_K and p_K / f_K follow from inv
        const R X = facK * (sK * den - num);
        const R w = rcp_(den * X);
        const R s_star = num * (X * w);
        const R dK = sK - s_star;
        const R inv = den * den * w;
        const R rho_star = facK * facK * inv;
        const R e_star = EK * iK + (s_star - uK) * (s_star + pK * dK * inv);
        f.r = f.r + sK * (rho_star - rK);
        f.mn = f.mn + sK * (rho_star * s_star - rK * uK);
        f.mt = f.mt + sK * (rho_star * tK - rK * tK);
        f.E = f.E + sK * (rho_star * e_star - EK);
    }
    return f;
}

template <int SCHEME, class R>
__device__ __forceinline__ Q4<R> face_flux(const Q4<R>& L, const Q4<R>& Rr, R gamma, R gm1) {
    if constexpr (sizeof(R) == sizeof(double)) {
        if (SCHEME == EFVM_FLUX_RUSANOV) return rusanov_flux_d(L, Rr, gamma, gm1);
        return hllc_flux_d<SCHEME != EFVM_FLUX_HLLC_TEXTBOOK>(L, Rr, gamma, gm1);
    } else {
        if (SCHEME == EFVM_FLUX_RUSANOV) return rusanov_flux(L, Rr, gamma, gm1);
        return hllc_flux<R, SCHEME != EFVM_FLUX_HLLC_TEXTBOOK>(L, Rr, gamma, gm1);
    }
}

// ---- 3-D: states (rho, m_n, m_t, m_s, E) in the frame of the face normal,
// with two tangential momenta.  The same forms as the FP64 functions above,
// with the second tangential velocity in |v|^2, the Thornber blend and the
// star state.
struct Q5 {
    double r, mn, mt, ms, E;
};
struct Side5 {
    double un, ut, us, q, p, a2, a;
};
__device__ __forceinline__ Side5 side5(const Q5& u, double inv, double gamma, double gm1) {
    Side5 s;
    s.un = __dmul_rn(u.mn, inv);
    s.ut = __dmul_rn(u.mt, inv);
    s.us = __dmul_rn(u.ms, inv);
    s.q = __fma_rn(s.un, s.un, __fma_rn(s.ut, s.ut, __dmul_rn(s.us, s.us)));
    s.p = __dmul_rn(gm1, __fma_rn(__dmul_rn(-0.5, u.r), s.q, u.E));
    s.a2 = __dmul_rn(__dmul_rn(gamma, s.p), inv);
    s.a = __dmul_rn(s.a2, rsqrt_(s.a2));
    return s;
}
__device__ __forceinline__ void sides5(const Q5& L, const Q5& R, double gamma, double gm1, Side5& l, Side5& r) {
    const double w = rcp_(__dmul_rn(L.r, R.r));
    l = side5(L, __dmul_rn(R.r, w), gamma, gm1);
    r = side5(R, __dmul_rn(L.r, w), gamma, gm1);
}
// physical_flux_inline along the face normal, crates/cfd_riemann/src/lib.rs:21-43
__device__ __forceinline__ Q5 physical_flux5(double rho, double un, double ut, double us, double E, double p) {
    Q5 f;
    f.r = __dmul_rn(rho, un);
    f.mn = __fma_rn(f.r, un, p);
    f.mt = __dmul_rn(f.r, ut);
    f.ms = __dmul_rn(f.r, us);
    f.E = __dmul_rn(__dadd_rn(E, p), un);
    return f;
}
// Rusanov::flux_inline, crates/cfd_riemann/src/lib.rs:222-240
__device__ __forceinline__ Q5 rusanov_flux5(const Q5& L, const Q5& R, double gamma, double gm1) {
    Side5 l, r;
    sides5(L, R, gamma, gm1, l, r);
    const Q5 fl = physical_flux5(L.r, l.un, l.ut, l.us, L.E, l.p);
    const Q5 fr = physical_flux5(R.r, r.un, r.ut, r.us, R.E, r.p);
    const double hl = __dmul_rn(-0.5, fmax(__dadd_rn(fabs(l.un), l.a), __dadd_rn(fabs(r.un), r.a)));
    auto mix = [&](double a, double b, double ul, double ur) {
        return __fma_rn(hl, __dsub_rn(ur, ul), __dmul_rn(0.5, __dadd_rn(a, b)));
    };
    return Q5{mix(fl.r, fr.r, L.r, R.r), mix(fl.mn, fr.mn, L.mn, R.mn), mix(fl.mt, fr.mt, L.mt, R.mt),
              mix(fl.ms, fr.ms, L.ms, R.ms), mix(fl.E, fr.E, L.E, R.E)};
}
// Hllc::flux_with_thornber + thornber_reconstruct + star_state,
// crates/cfd_riemann/src/lib.rs:395-506,619-644, in the equivalent form of
// hllc_flux_d above (Thornber over all three velocity components).
template <bool THORNBER>
__device__ __forceinline__ Q5 hllc_flux5(const Q5& L, const Q5& R, double gamma, double gm1) {
    Side5 l, r;
    sides5(L, R, gamma, gm1, l, r);
    double lcn = l.un, lct = l.ut, lcs = l.us, rcn = r.un, rct = r.ut, rcs = r.us, ELc = L.E, ERc = R.E;
    if (THORNBER) {
        const double vmax2 = l.q > r.q ? l.q : r.q;
        const double amax2 = l.a2 > r.a2 ? l.a2 : r.a2;
        const double prod = __dmul_rn(vmax2, amax2);  // below the normal range: z = 0, as in hllc_flux_d
        double hz = __dmul_rn(__dmul_rn(0.5, vmax2), rsqrt_(prod));
        hz = prod >= normal_min<double>() ? hz : 0.0;
        hz = vmax2 >= amax2 && amax2 > 0.0 ? 0.5 : hz;
        auto blend = [&](double a, double b, double& x, double& y) {
            const double avg = __dmul_rn(0.5, __dadd_rn(a, b)), d = __dsub_rn(a, b);
            x = __fma_rn(hz, d, avg);
            y = __fma_rn(-hz, d, avg);
        };
        blend(l.un, r.un, lcn, rcn);
        blend(l.ut, r.ut, lct, rct);
        blend(l.us, r.us, lcs, rcs);
        ELc = __fma_rn(__dmul_rn(0.5, L.r), __fma_rn(lcn, lcn, __fma_rn(lct, lct, __fma_rn(lcs, lcs, -l.q))), L.E);
        ERc = __fma_rn(__dmul_rn(0.5, R.r), __fma_rn(rcn, rcn, __fma_rn(rct, rct, __fma_rn(rcs, rcs, -r.q))), R.E);
    }
    const double s_l = fmin(__dsub_rn(lcn, l.a), __dsub_rn(rcn, r.a));
    const double s_r = fmax(__dadd_rn(lcn, l.a), __dadd_rn(rcn, r.a));
    const double fac_l = __dmul_rn(L.r, __dsub_rn(s_l, lcn));
    const double fac_r = __dmul_rn(R.r, __dsub_rn(s_r, rcn));
    const double num = __fma_rn(-fac_r, rcn, __fma_rn(fac_l, lcn, __dsub_rn(r.p, l.p)));
    const double den = __dsub_rn(fac_l, fac_r);
    const bool star_nonneg = __dmul_rn(num, den) >= 0.0 && den != 0.0;
    const bool useL = (s_l >= 0.0) || star_nonneg;
    const double uK = useL ? lcn : rcn;
    const double tK = useL ? lct : rct;
    const double wK = useL ? lcs : rcs;
    const double EK = useL ? ELc : ERc;
    const double pK = useL ? l.p : r.p;
    if (s_l < 0.0 && (star_nonneg || s_r >= 0.0)) {
        const double sK = useL ? s_l : s_r;
        const double facK = useL ? fac_l : fac_r;
        const double Y = __fma_rn(sK, den, -num);
        const double w = rcp_(__dmul_rn(den, Y));
        const double s_star = __dmul_rn(num, __dmul_rn(Y, w));
        const double inv = __dmul_rn(den, __dmul_rn(den, w));  // 1 / (s_K - s_*)
        const double pS = __fma_rn(facK, __dsub_rn(s_star, uK), pK);
        Q5 f;
        f.r = __dmul_rn(__dmul_rn(facK, inv), s_star);
        f.mn = __fma_rn(f.r, s_star, pS);
        f.mt = __dmul_rn(f.r, tK);
        f.ms = __dmul_rn(f.r, wK);
        const double eS = __fma_rn(pS, s_star, __fma_rn(__dsub_rn(sK, uK), EK, -__dmul_rn(pK, uK)));
        f.E = __dmul_rn(__fma_rn(eS, inv, pS), s_star);
        return f;
    }
    return physical_flux5(useL ? L.r : R.r, uK, tK, wK, EK, pK);
}
template <int SCHEME>
__device__ __forceinline__ Q5 face_flux5(const Q5& L, const Q5& R, double gamma, double gm1) {
    if (SCHEME == EFVM_FLUX_RUSANOV) return rusanov_flux5(L, R, gamma, gm1);
    return hllc_flux5<SCHEME != EFVM_FLUX_HLLC_TEXTBOOK>(L, R, gamma, gm1);
}

// minmod / monotonized_central, crates/cfd_solver/src/lib.rs:170-192.  (Deciding
// the sign test and the magnitude comparison on the bit patterns, to spare the
// FP64 pipe, measured 4 % slower at 4096^2: the 64-bit integer work costs more.)
template <class R>
__device__ __forceinline__ bool opposite_or_zero(R a, R b) { return a * b <= R(0); }
template <class R>
__device__ __forceinline__ bool smaller_magnitude(R a, R b) { return fabs_(a) < fabs_(b); }

template <class R>
__device__ __forceinline__ R minmod(R a, R b) {
    if (opposite_or_zero(a, b)) return R(0);
    return smaller_magnitude(a, b) ? a : b;
}
template <class R>
__device__ __forceinline__ R monotonized_central(R a, R b) {
    if (opposite_or_zero(a, b)) return R(0);
    const R s = a > R(0) ? R(1) : R(-1);
    return s * fmin_(fmin_(R(2) * fabs_(a), R(2) * fabs_(b)), R(0.5) * fabs_(a + b));
}
template <class R>
__device__ __forceinline__ R limit(int limiter, R fwd, R bwd) {
    return limiter == EFVM_LIMITER_MC ? monotonized_central(fwd, bwd) : minmod(fwd, bwd);
}

// The limited slope for the FP64 forms that apply it as c +- s f: s is the
// limiter's value as if the differences had the same sign, and f is `factor` (0.5,
// or 0 on a first-order side) or 0 where they have opposite signs.  The sign
// test is one bit operation on the high words instead of a product and a
// comparison, and the zero of the limiter costs one select of f's high word (the
// low word of 0.5 and 0 is zero) instead of two of s.  The states have the bits
// of c +- limit() / 2, except where a difference product underflows (|a b| <
// 1e-308), whose slope is kept instead of dropped.
__device__ __forceinline__ void limited_slope(int limiter, double fwd, double bwd, double factor, double& s, double& f) {
    const bool opposite = (__double2hiint(fwd) ^ __double2hiint(bwd)) < 0;
    f = __hiloint2double(opposite ? 0 : __double2hiint(factor), 0);
    if (limiter == EFVM_LIMITER_MC) {
        const double a = fabs(fwd), b = fabs(bwd), h = __dmul_rn(0.5, fabs(__dadd_rn(fwd, bwd)));
        const double m = __dmul_rn(2.0, a < b ? a : b);
        s = copysign(m < h ? m : h, fwd);
    } else {
        s = fabs(fwd) < fabs(bwd) ? fwd : bwd;
    }
}

}  // namespace efvm
