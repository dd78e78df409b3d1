// physics.cuh -- device-side pointwise physics of the per-step Godunov update.
//
// Every function follows the Fortran routine it cites with the same operation order (Fortran
// evaluates `a*b*c` as (a*b)*c and `a/b*c` as (a/b)*c), so the FP64 build compiled without FMA
// contraction reproduces the CPU oracle bit for bit.  The mixed-precision build instantiates
// the same templates with float.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "fp64.cuh"

namespace shark {

// 1/x for the mixed path: the FP32 reciprocal refined by one FP64 Newton step, relative error
// ~1e-14, for x within FP32 range (a handful of FP64 operations instead of a division).
__device__ __forceinline__ double rcp_refined(double x) {
    const double r = widen(1.0f / narrow(x));
    return r * (2.0 - x * r);
}

template <typename R> __device__ __forceinline__ R sq(R x) { return x * x; }
// gfortran MAX/MIN on non-NaN operands
template <typename R> __device__ __forceinline__ R fmax2(R a, R b) { return a > b ? a : b; }
template <typename R> __device__ __forceinline__ R fmin2(R a, R b) { return a < b ? a : b; }

// slope_limit (src/solver/slope_limiters.f90:5-37): FP32 forms of the three limiters for the mixed
// path, with single FMNMX min/max and copysign instead of a sign multiply:
//   minmod: 0 if l*r < 0, else the argument of smaller modulus (the right one on ties)
//   van Leer (harmonic): 0 if l*r <= 0, else 2 l r / (l + r)
//   MC(1.5): 0 if l*r <= 0, else sign(l+r) min(1.5 min(|l|,|r|), |l+r|/2)
__device__ __forceinline__ float limit_minmod_f(float l, float r) {
    const float m = fabsf(r) < fabsf(l) ? r : l;
    return l * r < 0.f ? 0.f : m;
}
__device__ __forceinline__ float limit_vl_f(float l, float r) {
    const float p = l * r;
    return p <= 0.f ? 0.f : 2.f * p / (l + r);
}
// min(|a|, |b|) carrying the sign sign(a) xor sign(b): >= 0 exactly when a and b have the same
// sign (or one is zero)
__device__ __forceinline__ float min_xorsign_abs_f(float a, float b) {
    float d;
    asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}
// MC: sign(s) min(1.5 min(|l|, |r|), |s|/2) when l r > 0, else 0; with m = max(min.xorsign.abs(l, r), 0)
// (0 unless l and r have the same sign) it is min.xorsign.abs(1.5 m, s/2)
__device__ __forceinline__ float limit_mc_f(float l, float r) {
    // 1.5 max(mx, 0) = 0.75 (mx + |mx|) exactly (one rounding of 1.5 mx, or 0): an add with an
    // operand modifier in place of a max
    const float mx = min_xorsign_abs_f(l, r);
    return min_xorsign_abs_f(0.75f * (mx + fabsf(mx)), 0.5f * (l + r));
}

// FP64 forms of the limiters, bit for bit those of slope_limiters.f90's operations with fewer FP64
// instructions (but where the product of the slopes underflows, below 1e-162 each: its sign decides here,
// there the zero that it rounds to):
// compares and sign choices on the bit patterns, 1.5 min(|l|, |r|) for the smaller of the two
// products (rounding keeps their order), one division by half the sum for 2 l r / (l + r).  What is
// not a number comes out as those operations leave it.
__device__ __forceinline__ double limit_minmod_d(double l, double r) {
    const double s = abs_less(r, l) ? r : l;
    return is_nan(l) || is_nan(r) ? l : signs_differ(l, r) ? 0.0 : s;
}
__device__ __forceinline__ double limit_vl_d(double l, double r) {
    const double b = 0.5 * (l + r), a = l * r;
    const double s = div64_const(a, b, rcp64(b));   // a is zero where b is below the normal range
    return is_zero(a) || is_neg(a) ? 0.0 : s;
}
__device__ __forceinline__ double limit_mc_d(double l, double r) {
    const double c = 0.5 * (l + r);
    const double m = 1.5 * abs64(abs_less(r, l) ? r : l);
    const double s = abs_less(m, c) ? m : c;
    return is_nan(c) ? c : no_common_sign(l, r) ? 0.0 : with_sign(s, c);
}

// Compile-time limiter choice (0 = first order) for kernels specialised per configuration.
template <int ST, typename R>
__device__ __forceinline__ R slope_limit_t(R l, R r) {
    if constexpr (ST == 0) return R(0);
    else if constexpr (std::is_same<R, float>::value) {
        if constexpr (ST == 1) return limit_minmod_f(l, r);
        else if constexpr (ST == 2) return limit_vl_f(l, r);
        else return limit_mc_f(l, r);
    } else if constexpr (ST == 1) return limit_minmod_d(l, r);
    else if constexpr (ST == 2) return limit_vl_d(l, r);
    else return limit_mc_d(l, r);
}

// inside (FP64 solvers, WHERE = TRIED): the solver's denominators lay inside div64_const's range.
template <typename R> struct GasFlux { R rho, mn, mt, mz, e; bool inside = true; };
template <typename R> struct DustFlux { R rho, mn, mt, mz; bool inside = true; };

// solver_llf (src/solver/solvers.f90:4-155), non-MHD
template <typename R>
__device__ __forceinline__ GasFlux<R> gas_llf(R gamma, R rho_lft, R u_lft, R v_lft, R w_lft, R P_lft,
                                              R rho_rgt, R u_rgt, R v_rgt, R w_rgt, R P_rgt, R csl, R csr) {
    const R half = R(0.5);
    R mom_u_rgt = rho_rgt * u_rgt, mom_u_lft = rho_lft * u_lft;
    R E_rgt = P_rgt / (gamma - R(1)) + half * rho_rgt * sq(u_rgt);
    R E_lft = P_lft / (gamma - R(1)) + half * rho_lft * sq(u_lft);
    R mom_v_rgt = rho_rgt * v_rgt, mom_v_lft = rho_lft * v_lft;
    E_rgt = E_rgt + half * rho_rgt * sq(v_rgt);
    E_lft = E_lft + half * rho_lft * sq(v_lft);
    R mom_w_rgt = rho_rgt * w_rgt, mom_w_lft = rho_lft * w_lft;
    E_rgt = E_rgt + half * rho_rgt * sq(w_rgt);
    E_lft = E_lft + half * rho_lft * sq(w_lft);
    R flx_rho_rgt = rho_rgt * u_rgt, flx_rho_lft = rho_lft * u_lft;
    R flx_mom_u_rgt = (rho_rgt * sq(u_rgt) + P_rgt), flx_mom_u_lft = (rho_lft * sq(u_lft) + P_lft);
    R flx_mom_v_rgt = rho_rgt * u_rgt * v_rgt, flx_mom_v_lft = rho_lft * u_lft * v_lft;
    R flx_mom_w_rgt = rho_rgt * u_rgt * w_rgt, flx_mom_w_lft = rho_lft * u_lft * w_lft;
    R flx_P_rgt = (E_rgt + P_rgt) * u_rgt, flx_P_lft = (E_lft + P_lft) * u_lft;
    R lam = fmax2(R(fabs(u_lft)) + csl, R(fabs(u_rgt)) + csr);
    GasFlux<R> f;
    f.rho = half * (flx_rho_lft + flx_rho_rgt) - half * lam * (rho_rgt - rho_lft);
    f.mn = half * (flx_mom_u_lft + flx_mom_u_rgt) - half * lam * (mom_u_rgt - mom_u_lft);
    f.mt = half * (flx_mom_v_lft + flx_mom_v_rgt) - half * lam * (mom_v_rgt - mom_v_lft);
    f.mz = half * (flx_mom_w_lft + flx_mom_w_rgt) - half * lam * (mom_w_rgt - mom_w_lft);
    f.e = half * (flx_P_lft + flx_P_rgt) - half * lam * (E_rgt - E_lft);
    return f;
}

// solver_dust_Huang_Bai (src/solver/solvers.f90:506-698): pressureless upwind, 4 cases (:654-694):
// both velocities > 0 -> left flux; both < 0 -> right flux; converging (u_l > 0 > u_r) -> sum;
// diverging or any exactly-zero velocity -> 0.  Written branch-free: the left flux enters when
// u_l > 0 and u_r != 0, the right flux when u_r < 0 and u_l != 0 (same cases, same sums).
// FP32, with selects only (mixed path).
__device__ __forceinline__ DustFlux<float> dust_hb_f(float rho_lft, float u_lft, float v_lft, float w_lft,
                                                     float rho_rgt, float u_rgt, float v_rgt, float w_rgt) {
    const bool takeL = (u_lft > 0.f) && (u_rgt != 0.f);
    const bool takeR = (u_rgt < 0.f) && (u_lft != 0.f);
    const float ml = takeL ? rho_lft * u_lft : 0.f;
    const float mr = takeR ? rho_rgt * u_rgt : 0.f;
    DustFlux<float> f;
    f.rho = ml + mr;
    f.mn = ml * u_lft + mr * u_rgt;
    f.mt = ml * v_lft + mr * v_rgt;
    f.mz = ml * w_lft + mr * w_rgt;
    return f;
}

// solver_dust_llf (src/solver/solvers.f90:840-1001), non-MHD
template <typename R>
__device__ __forceinline__ DustFlux<R> dust_llf(R rho_lft, R u_lft, R v_lft, R w_lft,
                                                R rho_rgt, R u_rgt, R v_rgt, R w_rgt) {
    const R half = R(0.5);
    R lam = fmax2(R(fabs(u_lft)), R(fabs(u_rgt)));
    DustFlux<R> f;
    f.rho = half * (rho_lft * u_lft + rho_rgt * u_rgt) - half * lam * (rho_rgt - rho_lft);
    f.mn = half * (rho_lft * sq(u_lft) + rho_rgt * sq(u_rgt)) - half * lam * (rho_rgt * u_rgt - rho_lft * u_lft);
    f.mt = half * (rho_lft * u_lft * v_lft + rho_rgt * u_rgt * v_rgt) - half * lam * (rho_rgt * v_rgt - rho_lft * v_lft);
    f.mz = half * (rho_lft * u_lft * w_lft + rho_rgt * u_rgt * w_rgt) - half * lam * (rho_rgt * w_rgt - rho_lft * w_lft);
    return f;
}

// solver_dust_hll (src/solver/solvers.f90:1010-1194), non-MHD
template <typename R>
__device__ __forceinline__ DustFlux<R> dust_hll(R rho_lft, R u_lft, R v_lft, R w_lft,
                                                R rho_rgt, R u_rgt, R v_rgt, R w_rgt) {
    R S_lft = fmin2(fmin2(u_lft, u_rgt), R(0));
    R S_rgt = fmax2(fmax2(u_lft, u_rgt), R(0));
    DustFlux<R> f{R(0), R(0), R(0), R(0)};
    if (S_rgt - S_lft != R(0)) {
        f.rho = (S_rgt * (rho_lft * u_lft) - S_lft * (rho_rgt * u_rgt) + S_rgt * S_lft * (rho_rgt - rho_lft)) / (S_rgt - S_lft);
        f.mn = (S_rgt * (rho_lft * sq(u_lft)) - S_lft * (rho_rgt * sq(u_rgt)) + S_rgt * S_lft * (rho_rgt * u_rgt - rho_lft * u_lft)) / (S_rgt - S_lft);
        f.mt = (S_rgt * (rho_lft * u_lft * v_lft) - S_lft * (rho_rgt * u_rgt * v_rgt) + S_rgt * S_lft * (rho_rgt * v_rgt - rho_lft * v_lft)) / (S_rgt - S_lft);
        f.mz = (S_rgt * (rho_lft * u_lft * w_lft) - S_lft * (rho_rgt * u_rgt * w_rgt) + S_rgt * S_lft * (rho_rgt * w_rgt - rho_lft * w_lft)) / (S_rgt - S_lft);
    }
    return f;
}

// FP64 forms of the solvers, rounding as the reference's operations do with fewer FP64 instructions: one
// reciprocal for the quotients of a denominator, minima, maxima and case choices on the bit patterns, and
// the HLLC's energy and star state for the sampled side only.  y1 = rcp64 of gamma - 1.
__device__ __forceinline__ double gas_energy_d(double g1, double y1, double rho, double u, double v, double w, double P) {
    const double hr = 0.5 * rho;
    return div64_const(P, g1, y1) + hr * sq(u) + hr * sq(v) + hr * sq(w);
}
__device__ __forceinline__ GasFlux<double> gas_llf_d(double gamma, double y1, double rl, double ul, double vl, double wl,
                                                     double Pl, double rr, double ur, double vr, double wr, double Pr,
                                                     double csl, double csr) {
    const double El = gas_energy_d(gamma - 1.0, y1, rl, ul, vl, wl, Pl), Er = gas_energy_d(gamma - 1.0, y1, rr, ur, vr, wr, Pr);
    const double ml = rl * ul, mr = rr * ur;
    const double hl = 0.5 * max64(abs64(ul) + csl, abs64(ur) + csr);
    GasFlux<double> f;
    f.rho = 0.5 * (ml + mr) - hl * (rr - rl);
    f.mn = 0.5 * ((rl * sq(ul) + Pl) + (rr * sq(ur) + Pr)) - hl * (mr - ml);
    f.mt = 0.5 * (ml * vl + mr * vr) - hl * (rr * vr - rl * vl);
    f.mz = 0.5 * (ml * wl + mr * wr) - hl * (rr * wr - rl * wl);
    f.e = 0.5 * ((El + Pl) * ul + (Er + Pr) * ur) - hl * (Er - El);
    return f;
}
// solver_hll (src/solver/solvers.f90:157-306), non-MHD
template <int WHERE>
__device__ __forceinline__ GasFlux<double> gas_hll_d(double gamma, double y1, double rl, double ul, double vl, double wl,
                                                     double Pl, double rr, double ur, double vr, double wr, double Pr,
                                                     double csl, double csr) {
    const double El = gas_energy_d(gamma - 1.0, y1, rl, ul, vl, wl, Pl), Er = gas_energy_d(gamma - 1.0, y1, rr, ur, vr, wr, Pr);
    const double ml = rl * ul, mr = rr * ur, cm = max64(csl, csr);
    const double Sl = min64_0(min64(ul, ur) - cm), Sr = max64_0(max64(ul, ur) + cm);
    const double ss = Sr * Sl;
    const Over<double, WHERE> by_b(Sr - Sl);
    GasFlux<double> f;
    f.inside = by_b.inside();
    f.rho = Sr * ml - Sl * mr + ss * (rr - rl);
    f.mn = Sr * (rl * sq(ul) + Pl) - Sl * (rr * sq(ur) + Pr) + ss * (mr - ml);
    f.mt = Sr * (ml * vl) - Sl * (mr * vr) + ss * (rr * vr - rl * vl);
    f.mz = Sr * (ml * wl) - Sl * (mr * wr) + ss * (rr * wr - rl * wl);
    f.e = Sr * ((El + Pl) * ul) - Sl * ((Er + Pr) * ur) + ss * (Er - El);
    by_b.all(f.rho, f.mn, f.mt, f.mz, f.e);
    return f;
}
// solver_hllc (src/solver/solvers.f90:308-500): RAMSES-style HLLC with the wave speeds clipped to
// include 0 (:435-436), Lagrangian star state (:450-463), sampling at x/t = 0 (:466-486) and the
// passive transverse momenta upwinded on the sign of u* (:491-497).
template <int WHERE>
__device__ __forceinline__ GasFlux<double> gas_hllc_d(double gamma, double y1, double rl, double ul, double vl, double wl,
                                                      double Pl, double rr, double ur, double vr, double wr, double Pr,
                                                      double csl, double csr) {
    const double cm = max64(csl, csr);
    const double Sl = min64_0(min64(ul, ur) - cm), Sr = max64_0(max64(ul, ur) + cm);
    const double hl = rl * (ul - Sl), hr = rr * (Sr - ur);
    const Over<double, WHERE> by_b(hr + hl);
    double us = hr * ur + hl * ul + (Pl - Pr), Ps = hr * Pl + hl * Pr + hl * hr * (ul - ur);
    by_b.all(us, Ps);
    bool inside = by_b.inside();
    const bool left = is_pos(us);
    const double S = left ? Sl : Sr, rho = left ? rl : rr, u = left ? ul : ur, v = left ? vl : vr, w = left ? wl : wr;
    const double P = left ? Pl : Pr;
    const double E = gas_energy_d(gamma - 1.0, y1, rho, u, v, w, P);
    double ro = rho, uo = u, Po = P, eo = E;
    if (left || is_pos(Sr)) {   // Sl is at most 0, so the left state itself is never sampled
        const double d = S - u;
        const Over<double, WHERE> by_c(S - us);
        ro = rho * d;
        uo = us;
        Po = Ps;
        eo = d * E - P * u + Ps * us;
        by_c.all(ro, eo);
        inside = inside && by_c.inside();
    }
    GasFlux<double> f;
    f.inside = inside;
    f.rho = ro * uo;
    f.mn = f.rho * uo + Po;
    f.e = (eo + Po) * uo;
    f.mt = f.rho * v;
    f.mz = f.rho * w;
    return f;
}
__device__ __forceinline__ DustFlux<double> dust_hb_d(double rl, double ul, double vl, double wl, double rr, double ur,
                                                      double vr, double wr) {
    const bool takeL = is_pos(ul) && !is_zero(ur), takeR = is_neg(ur) && !is_zero(ul);
    const double rho = takeL ? rl : rr, u = takeL ? ul : ur, v = takeL ? vl : vr, w = takeL ? wl : wr;
    const bool any = takeL || takeR;
    const double m = any ? rho * u : 0.0;
    DustFlux<double> f{m, any ? rho * sq(u) : 0.0, m * v, m * w};
    if (takeL && takeR) {   // converging: the right side's flux on top
        const double mr = rr * ur;
        f.rho = f.rho + mr;
        f.mn = f.mn + rr * sq(ur);
        f.mt = f.mt + mr * vr;
        f.mz = f.mz + mr * wr;
    }
    return f;
}
__device__ __forceinline__ DustFlux<double> dust_llf_d(double rl, double ul, double vl, double wl, double rr, double ur,
                                                       double vr, double wr) {
    const double hl = 0.5 * max64(abs64(ul), abs64(ur)), ml = rl * ul, mr = rr * ur;
    DustFlux<double> f;
    f.rho = 0.5 * (ml + mr) - hl * (rr - rl);
    f.mn = 0.5 * (rl * sq(ul) + rr * sq(ur)) - hl * (mr - ml);
    f.mt = 0.5 * (ml * vl + mr * vr) - hl * (rr * vr - rl * vl);
    f.mz = 0.5 * (ml * wl + mr * wr) - hl * (rr * wr - rl * wl);
    return f;
}
template <int WHERE>
__device__ __forceinline__ DustFlux<double> dust_hll_d(double rl, double ul, double vl, double wl, double rr, double ur,
                                                       double vr, double wr) {
    const double Sl = min64_0(min64(ul, ur)), Sr = max64_0(max64(ul, ur)), b = Sr - Sl;
    DustFlux<double> f{0.0, 0.0, 0.0, 0.0};
    if (!is_zero(b)) {
        const Over<double, WHERE> by_b(b);
        const double ss = Sr * Sl, ml = rl * ul, mr = rr * ur;
        f.inside = by_b.inside();
        f.rho = Sr * ml - Sl * mr + ss * (rr - rl);
        f.mn = Sr * (rl * sq(ul)) - Sl * (rr * sq(ur)) + ss * (mr - ml);
        f.mt = Sr * (ml * vl) - Sl * (mr * vr) + ss * (rr * vr - rl * vl);
        f.mz = Sr * (ml * wl) - Sl * (mr * wr) + ss * (rr * wr - rl * wl);
        by_b.all(f.rho, f.mn, f.mt, f.mz);
    }
    return f;
}
template <int WHERE>
__device__ __forceinline__ DustFlux<double> dust_hllc_d(double rl, double ul, double vl, double wl, double rr, double ur,
                                                        double vr, double wr, double csl, double csr) {
    const double cm = max64(csl, csr);
    const double Sl = min64_0(min64(ul, ur) - cm), Sr = max64_0(max64(ul, ur) + cm);
    const double hl = rl * (ul - Sl), hr = rr * (Sr - ur);
    const Over<double, WHERE> by_b(hr + hl);
    double us = hr * ur + hl * ul, Ps = hl * hr * (ul - ur);
    by_b.all(us, Ps);
    bool inside = by_b.inside();
    const bool left = is_pos(us);
    const double S = left ? Sl : Sr, rho = left ? rl : rr, u = left ? ul : ur, v = left ? vl : vr, w = left ? wl : wr;
    double ro = rho, uo = u, Po = 0.0;
    if (left || is_pos(Sr)) {
        const Over<double, WHERE> by_c(S - us);
        ro = by_c(rho * (S - u));
        uo = us;
        Po = Ps;
        inside = inside && by_c.inside();
    }
    DustFlux<double> f;
    f.inside = inside;
    f.rho = ro * uo;
    f.mn = f.rho * uo + Po;
    f.mt = f.rho * v;
    f.mz = f.rho * w;
    return f;
}

// solver_hllc_dust (src/solver/solvers.f90:704-836): the gas HLLC with zero pressure on one
// pressureless species, signal speeds bounded by the gas sound speeds csl, csr of the face (the
// reference's operation order; the energies it forms do not enter the flux).
template <typename R>
__device__ __forceinline__ DustFlux<R> dust_hllc(R rho_lft, R u_lft, R v_lft, R w_lft, R rho_rgt, R u_rgt, R v_rgt,
                                                 R w_rgt, R csl, R csr) {
    const R P_rgt = R(0), P_lft = R(0);
    const R cm = fmax2(csl, csr);
    const R S_lft = fmin2(fmin2(u_lft, u_rgt) - cm, R(0));
    const R S_rgt = fmax2(fmax2(u_lft, u_rgt) + cm, R(0));
    const R hllc_l = rho_lft * (u_lft - S_lft);
    const R hllc_r = rho_rgt * (S_rgt - u_rgt);
    const R ustar = (hllc_r * u_rgt + hllc_l * u_lft + (P_lft - P_rgt)) / (hllc_r + hllc_l);
    const R Pstar = (hllc_r * P_lft + hllc_l * P_rgt + hllc_l * hllc_r * (u_lft - u_rgt)) / (hllc_r + hllc_l);
    R r_o, u_o, P_o;
    if (S_lft > R(0)) { r_o = rho_lft; u_o = u_lft; P_o = P_lft; }
    else if (ustar > R(0)) { r_o = rho_lft * (S_lft - u_lft) / (S_lft - ustar); u_o = ustar; P_o = Pstar; }
    else if (S_rgt > R(0)) { r_o = rho_rgt * (S_rgt - u_rgt) / (S_rgt - ustar); u_o = ustar; P_o = Pstar; }
    else { r_o = rho_rgt; u_o = u_rgt; P_o = P_rgt; }
    DustFlux<R> f;
    f.rho = r_o * u_o;
    f.mn = r_o * u_o * u_o + P_o;
    const bool lft = ustar > R(0);
    f.mt = r_o * u_o * (lft ? v_lft : v_rgt);
    f.mz = r_o * u_o * (lft ? w_lft : w_rgt);
    return f;
}

}  // namespace shark
