// flux_line.cuh -- the flux kernels' shared pieces (setup forces, solver choice) and K1 for 1D grids.
//
// K1 in 1D: one warp per 32 columns of one species (lane = column; lanes 0, 1, 30, 31 are the
// halo, 28 columns are updated).  A lane converts its cell to primitives (ctoprim, solve.f90:195-253),
// forms its limited slopes and half-step face states from its neighbours' values by shuffle
// (predictor, godunov.f90:7-629), solves its left face and updates its cell with both faces' fluxes
// (add_delta_u, godunov.f90:659-750; kick, force_kicks.f90:2-41).  No shared memory, no barrier.
//
// A 1D grid of a few thousand cells leaves most of the GPU idle whatever the split: what counts is
// the length of one warp's instruction chain, in FP64 at 64 clocks an instruction.  One warp per
// 28 cells and species gives every warp an SM partition of its own, and the FP64 operations are
// those of fp64.cuh.  Sod, 1000 cells, FP64: 0.055 ms as 128-cell shared-memory tiles, 0.016 ms
// so; dusty wave, 2048 x 4: 0.050 -> 0.015 ms.  FP64 rounds as the oracle's operation order does;
// FP32 is the mixed path's form (flux_strip.cuh).
#pragma once

#include <type_traits>

namespace shark {

// Force of the setup on a gas (s == 0) or dust (s > 0) element with primitive velocities
// (vx, vy, vz) at column ix: update_force_setup of SI (src/setups/SI/setup.f90:335-368) and of
// the polar disk (point-mass gravity -Mstar/r^2, disk_polar/setup.f90:358-366, no planet or
// self-gravity).  SOD and DUSTYWAVE have no force.  `drag` is on for every configuration that
// uses the force (the !drag extra terms are rejected at init).
template <typename R>
__device__ __forceinline__ void setup_force(const KParams<R>& p, int s, int ix, long long cell, R vx, R vz, R& f1,
                                            R& f2, R& f3) {
    if (p.setup == SHARK_SETUP_SI) {
        const R qs = prm<R>(p.si_q, p.f_si_q), om = prm<R>(p.si_om, p.f_si_om);
        const R xc = p.xpos[ix] - prm<R>(R(0.5) * R(p.box_l), p.f_half_box_l);
        if (s == 0)
            f1 = R(2) * qs * sq(om) * xc - R(2) * om * vz - R(2) * prm<R>(p.si_r0, p.f_si_r0) * om * prm<R>(p.si_eta, p.f_si_eta);
        else
            f1 = R(2) * qs * sq(om) * xc - R(2) * om * vz;
        f2 = R(0);
        f3 = R(2) * om * vx;
    } else if (p.setup == SHARK_SETUP_DISK_POLAR) {
        f1 = p.fgrav[ix];
        f2 = f3 = R(0);
    } else if (p.setup == SHARK_SETUP_DISK_CART) {   // the star's softened gravity (disk/setup.f90)
        f1 = p.cfx[cell];
        f2 = p.cfy[cell];
        f3 = R(0);
    } else {
        f1 = f2 = f3 = R(0);
    }
}

// HLLC with one reciprocal for the star state and one for the sampled star side (mixed path).
__device__ __forceinline__ GasFlux<float> gas_hllc_fast(float inv_g1, float rho_lft, float u_lft, float v_lft,
                                                        float w_lft, float P_lft, float rho_rgt, float u_rgt,
                                                        float v_rgt, float w_rgt, float P_rgt, float csl, float csr) {
    const float E_rgt = P_rgt * inv_g1 + 0.5f * rho_rgt * (u_rgt * u_rgt + v_rgt * v_rgt + w_rgt * w_rgt);
    const float E_lft = P_lft * inv_g1 + 0.5f * rho_lft * (u_lft * u_lft + v_lft * v_lft + w_lft * w_lft);
    const float cmax = fmaxf(csl, csr);
    const float S_lft = fminf(fminf(u_lft, u_rgt) - cmax, 0.f);
    const float S_rgt = fmaxf(fmaxf(u_lft, u_rgt) + cmax, 0.f);
    const float hllc_l = rho_lft * (u_lft - S_lft);
    const float hllc_r = rho_rgt * (S_rgt - u_rgt);
    const float inv = 1.0f / (hllc_r + hllc_l);
    const float ustar = (hllc_r * u_rgt + hllc_l * u_lft + (P_lft - P_rgt)) * inv;
    const float Pstar = (hllc_r * P_lft + hllc_l * P_rgt + hllc_l * hllc_r * (u_lft - u_rgt)) * inv;
    float r_o, u_o, P_o, e_o;
    if (S_lft > 0.f) {
        r_o = rho_lft; u_o = u_lft; P_o = P_lft; e_o = E_lft;
    } else if (S_rgt <= 0.f) {
        r_o = rho_rgt; u_o = u_rgt; P_o = P_rgt; e_o = E_rgt;
    } else {
        // star side chosen by the sign of u* (solvers.f90:469-481)
        const bool left = ustar > 0.f;
        const float S = left ? S_lft : S_rgt, rho = left ? rho_lft : rho_rgt, u = left ? u_lft : u_rgt;
        const float P = left ? P_lft : P_rgt, E = left ? E_lft : E_rgt;
        const float a = 1.0f / (S - ustar);
        r_o = rho * (S - u) * a;
        u_o = ustar;
        P_o = Pstar;
        e_o = ((S - u) * E - P * u + Pstar * ustar) * a;
    }
    GasFlux<float> f;
    f.rho = r_o * u_o;
    f.mn = r_o * u_o * u_o + P_o;
    f.e = (e_o + P_o) * u_o;
    if (ustar > 0.f) { f.mt = r_o * u_o * v_lft; f.mz = r_o * u_o * w_lft; }
    else { f.mt = r_o * u_o * v_rgt; f.mz = r_o * u_o * w_rgt; }
    return f;
}

// HLL with one reciprocal (mixed path).
__device__ __forceinline__ GasFlux<float> gas_hll_fast(float inv_g1, float rho_lft, float u_lft, float v_lft,
                                                       float w_lft, float P_lft, float rho_rgt, float u_rgt,
                                                       float v_rgt, float w_rgt, float P_rgt, float csl, float csr) {
    const float E_rgt = P_rgt * inv_g1 + 0.5f * rho_rgt * (u_rgt * u_rgt + v_rgt * v_rgt + w_rgt * w_rgt);
    const float E_lft = P_lft * inv_g1 + 0.5f * rho_lft * (u_lft * u_lft + v_lft * v_lft + w_lft * w_lft);
    const float cmax = fmaxf(csl, csr);
    const float S_lft = fminf(fminf(u_lft, u_rgt) - cmax, 0.f);
    const float S_rgt = fmaxf(fmaxf(u_lft, u_rgt) + cmax, 0.f);
    const float inv = 1.0f / (S_rgt - S_lft);
    const float ss = S_rgt * S_lft;
    const float ml = rho_lft * u_lft, mr = rho_rgt * u_rgt;
    GasFlux<float> f;
    f.rho = (S_rgt * ml - S_lft * mr + ss * (rho_rgt - rho_lft)) * inv;
    f.mn = (S_rgt * (ml * u_lft + P_lft) - S_lft * (mr * u_rgt + P_rgt) + ss * (mr - ml)) * inv;
    f.mt = (S_rgt * ml * v_lft - S_lft * mr * v_rgt + ss * (rho_rgt * v_rgt - rho_lft * v_lft)) * inv;
    f.mz = (S_rgt * ml * w_lft - S_lft * mr * w_rgt + ss * (rho_rgt * w_rgt - rho_lft * w_lft)) * inv;
    f.e = (S_rgt * (E_lft + P_lft) * u_lft - S_lft * (E_rgt + P_rgt) * u_rgt + ss * (E_rgt - E_lft)) * inv;
    return f;
}

// Compile-time solver choice (solve_wrapper, godunov.f90:768-833) for specialised kernels.
template <int SOLVER, int WHERE, typename R>
__device__ __forceinline__ GasFlux<R> gas_flux_t(R gamma, R inv_g1, R rl, R ul, R vl, R wl, R pl, R rr, R ur, R vr,
                                                 R wr, R pr, R csl, R csr) {
    if constexpr (std::is_same<R, float>::value) {
        if constexpr (SOLVER == 2) return gas_hllc_fast(inv_g1, rl, ul, vl, wl, pl, rr, ur, vr, wr, pr, csl, csr);
        else if constexpr (SOLVER == 1) return gas_hll_fast(inv_g1, rl, ul, vl, wl, pl, rr, ur, vr, wr, pr, csl, csr);
        else return gas_llf(gamma, rl, ul, vl, wl, pl, rr, ur, vr, wr, pr, csl, csr);
    } else {
        if constexpr (SOLVER == 2) return gas_hllc_d<WHERE>(gamma, inv_g1, rl, ul, vl, wl, pl, rr, ur, vr, wr, pr, csl, csr);
        else if constexpr (SOLVER == 1) return gas_hll_d<WHERE>(gamma, inv_g1, rl, ul, vl, wl, pl, rr, ur, vr, wr, pr, csl, csr);
        else return gas_llf_d(gamma, inv_g1, rl, ul, vl, wl, pl, rr, ur, vr, wr, pr, csl, csr);
    }
}

// csl, csr: the gas sound speeds of the face (used by the HLLC dust solver only).
template <int SOLVERDUST, int WHERE, typename R>
__device__ __forceinline__ DustFlux<R> dust_flux_t(R rl, R ul, R vl, R wl, R rr, R ur, R vr, R wr, R csl, R csr) {
    if constexpr (SOLVERDUST == 0 && std::is_same<R, float>::value) return dust_hb_f(rl, ul, vl, wl, rr, ur, vr, wr);
    else if constexpr (std::is_same<R, double>::value) {
        if constexpr (SOLVERDUST == 0) return dust_hb_d(rl, ul, vl, wl, rr, ur, vr, wr);
        else if constexpr (SOLVERDUST == 1) return dust_llf_d(rl, ul, vl, wl, rr, ur, vr, wr);
        else if constexpr (SOLVERDUST == 2) return dust_hll_d<WHERE>(rl, ul, vl, wl, rr, ur, vr, wr);
        else return dust_hllc_d<WHERE>(rl, ul, vl, wl, rr, ur, vr, wr, csl, csr);
    }
    else if constexpr (SOLVERDUST == 1) return dust_llf(rl, ul, vl, wl, rr, ur, vr, wr);
    else if constexpr (SOLVERDUST == 2) return dust_hll(rl, ul, vl, wl, rr, ur, vr, wr);
    else return dust_hllc(rl, ul, vl, wl, rr, ur, vr, wr, csl, csr);
}

constexpr int LINE_UX = 28;   // columns updated per warp

// One species of one strip.  ST: slope limiter (0..3).  WHERE = TRIED (FP64): false where a denominator of
// the strip lies outside div64_const's range; what it stored is then to be written over.
template <typename R, bool IS_GAS, int ST, int WHERE>
__device__ __forceinline__ bool flux_line(const KParams<R>& p, int s) {
    constexpr bool FAST = std::is_same<R, float>::value;
    constexpr int NV = IS_GAS ? 5 : 4;
    const int N = p.ndust, lane = threadIdx.x & 31;
    const int gx = p.ng + blockIdx.x * LINE_UX - 2 + lane;
    const int gxc = min(gx, p.nx_max - 1), gxl = max(gxc - 1, 0), gxr = min(gxc + 1, p.nx_max - 1);
    const R dt = step_dt(p), half = R(0.5), hdt = half * dt;
    const R gamma = prm<R>(p.gamma, p.f_gamma), smallP = prm<R>(p.smallp, p.f_smallp), smallR = prm<R>(p.smallr, p.f_smallr);
    const bool iso = p.iso == 1, fk = (p.flags & SHARK_FLAG_FORCE_KICK) != 0;
    auto up = [](R x) { return __shfl_up_sync(0xffffffffu, x, 1); };
    auto dn = [](R x) { return __shfl_down_sync(0xffffffffu, x, 1); };

    R uu[NV], q[NV], cs = p.cs[gxc];
#pragma unroll
    for (int k = 0; k < NV; ++k) uu[k] = p.u_cur[svar(s, k, N) * p.plane + gxc];
    const Over<R, WHERE> by_rho(uu[0]);
    bool inside = by_rho.inside();
    q[0] = uu[0];
    if constexpr (FAST) {
        const R ir = R(1) / uu[0];
        q[1] = uu[1] * ir; q[2] = uu[2] * ir; q[3] = uu[3] * ir;
    } else {
        q[1] = by_rho(uu[1]); q[2] = by_rho(uu[2]); q[3] = by_rho(uu[3]);
    }
    if constexpr (IS_GAS) {
        if constexpr (FAST) {
            const R P = fmax2((gamma - R(1)) * (uu[4] - half * (uu[1] * q[1] + uu[2] * q[2] + uu[3] * q[3])), smallP);
            q[0] = fmax2(uu[0], smallR);
            if (!iso) { cs = sqrt(gamma * P / q[0]); q[4] = P; }
            else q[4] = uu[0] * sq(cs);
        } else {
            q[0] = max64_pos(uu[0], smallR);
            if (iso) {
                q[4] = uu[0] * sq(cs);
            } else {
                const R hr = half * uu[0];
                q[4] = max64_pos((gamma - R(1)) * (uu[4] - (hr * sq(q[1]) + hr * sq(q[2]) + hr * sq(q[3]))), smallP);
                cs = sqrt(Over<R, WHERE>(q[0])(gamma * q[4]));
            }
        }
    }
    // limited slopes
    const R dx1 = p.dx1[gxc];
    const R bl = half * (dx1 + p.dx1[gxl]), br = half * (p.dx1[gxr] + dx1);   // 2 d / (dx + dx') = d / ((dx + dx') / 2)
    const R sfl = p.sfx[gxc], sfr = p.sfx[gxr];
    const Over<R, CONSTANT> by_l(bl), by_r(br);
    R dq[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        dq[k] = R(0);
        if (IS_GAS && k == 4 && iso) continue;   // isothermal: rho's slope times cs^2
        const R dl = q[k] - up(q[k]), dr = dn(q[k]) - q[k];
        if constexpr (ST > 0) {
            if constexpr (FAST) dq[k] = slope_limit_t<ST>(dl * sfl, dr * sfr);
            else dq[k] = slope_limit_t<ST>(by_l(dl), by_r(dr));
        }
    }
    // half-step face states of the cell: qm its right face, qp its left one
    R u = q[1], v = q[2], w = q[3], f1 = R(0), f2 = R(0), f3 = R(0);
    if (fk) {
        if (gx >= p.ng && gx < p.ng + p.nx) setup_force(p, s, gxc, gxc, u, w, f1, f2, f3);   // ghost cells: no force
        u = u + f1 * hdt;
        v = v + f2 * hdt;
        w = w + f3 * hdt;
    }
    const R hdx = half * dx1;
    R qm[NV], qp[NV];
    R b[NV];
    b[0] = q[0] + hdt * (-u * dq[0] - dq[1] * q[0]);
    b[2] = v + hdt * (-u * dq[2]);
    b[3] = w + hdt * (-u * dq[3]);
    if constexpr (IS_GAS) {
        if (iso) { q[4] = q[0] * sq(cs); dq[4] = dq[0] * sq(cs); }
        R dp_r;
        if constexpr (FAST) dp_r = dq[4] * (R(1) / q[0]);
        else {
            const Over<R, WHERE> by_q(q[0]);
            dp_r = by_q(dq[4]);
            inside = inside && by_q.inside();
        }
        b[1] = u + hdt * (-u * dq[1] - dp_r);
        b[4] = q[4] + hdt * (-u * dq[4] - dq[1] * gamma * q[4]);
    } else {
        b[1] = u + hdt * (-u * dq[1]);
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        qm[k] = b[k] + hdx * dq[k];
        qp[k] = b[k] - hdx * dq[k];
    }
    // left face: qm of the left neighbour, qp of this cell
    R fl[NV];
    if constexpr (IS_GAS) {
        if (iso) {
            qm[4] = sq(cs) * qm[0];
            qp[4] = sq(cs) * qp[0];
        } else if constexpr (FAST) {
            qm[4] = fmaxf(qm[4], smallP);
            qp[4] = fmaxf(qp[4], smallP);
        } else {
            qm[4] = max64_pos(qm[4], smallP);
            qp[4] = max64_pos(qp[4], smallP);
        }
    }
    R ql[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) ql[k] = up(qm[k]);
    if constexpr (IS_GAS) {
        R csl = up(cs), csr = cs;
        if (!iso) {
            if constexpr (FAST) { csl = sqrt(gamma * ql[4] / ql[0]); csr = sqrt(gamma * qp[4] / qp[0]); }
            else {
                const Over<R, WHERE> by_ql(ql[0]), by_qp(qp[0]);
                csl = sqrt(by_ql(gamma * ql[4]));
                csr = sqrt(by_qp(gamma * qp[4]));
                inside = inside && by_ql.inside() && by_qp.inside();
            }
        }
        R g1;   // 1/(gamma - 1)
        if constexpr (FAST) g1 = p.f_inv_g1;
        else g1 = rcp64(gamma - R(1));
        GasFlux<R> g;
        if (p.solver == 2) g = gas_flux_t<2, WHERE>(gamma, g1, ql[0], ql[1], ql[2], ql[3], ql[4], qp[0], qp[1], qp[2], qp[3], qp[4], csl, csr);
        else if (p.solver == 1) g = gas_flux_t<1, WHERE>(gamma, g1, ql[0], ql[1], ql[2], ql[3], ql[4], qp[0], qp[1], qp[2], qp[3], qp[4], csl, csr);
        else g = gas_flux_t<0, WHERE>(gamma, g1, ql[0], ql[1], ql[2], ql[3], ql[4], qp[0], qp[1], qp[2], qp[3], qp[4], csl, csr);
        fl[0] = g.rho; fl[1] = g.mn; fl[2] = g.mt; fl[3] = g.mz; fl[4] = g.e;
        inside = inside && g.inside;
    } else {
        // the HLLC dust solver's gas sound speeds (isothermal gas: per column, godunov.f90:675-677)
        const R csl = up(cs);
        DustFlux<R> d;
        if (p.solverdust == 0) d = dust_flux_t<0, WHERE>(ql[0], ql[1], ql[2], ql[3], qp[0], qp[1], qp[2], qp[3], csl, cs);
        else if (p.solverdust == 1) d = dust_flux_t<1, WHERE>(ql[0], ql[1], ql[2], ql[3], qp[0], qp[1], qp[2], qp[3], csl, cs);
        else if (p.solverdust == 2) d = dust_flux_t<2, WHERE>(ql[0], ql[1], ql[2], ql[3], qp[0], qp[1], qp[2], qp[3], csl, cs);
        else d = dust_flux_t<3, WHERE>(ql[0], ql[1], ql[2], ql[3], qp[0], qp[1], qp[2], qp[3], csl, cs);
        fl[0] = d.rho; fl[1] = d.mn; fl[2] = d.mt; fl[3] = d.mz;
        inside = inside && d.inside;
    }
    // kick(1.0) (force_kicks.f90:2-41), then the flux difference
    if (fk) {
        const R rdt = uu[0] * dt;
        R eo = R(0);
        auto kinetic = [&]() -> R {
            if constexpr (FAST) return half * (sq(uu[1]) + sq(uu[2]) + sq(uu[3])) * (R(1) / uu[0]);
            else return by_rho(half * sq(uu[1])) + by_rho(half * sq(uu[2])) + by_rho(half * sq(uu[3]));
        };
        if constexpr (IS_GAS) eo = kinetic();
        uu[1] = uu[1] + rdt * f1;
        uu[2] = uu[2] + rdt * f2;
        uu[3] = uu[3] + rdt * f3;
        if constexpr (IS_GAS) uu[4] = uu[4] + (kinetic() - eo);
    }
    const R s1 = p.surf1[gxc], vol = p.vol[gxc];
    const Over<R, CONSTANT> by_vol(vol);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const R a = fl[k] * s1, ar = dn(a);   // the right face is the right neighbour's left one
        if constexpr (FAST) uu[k] = uu[k] + (a - ar) * (dt * p.rvol[gxc]);
        else uu[k] = uu[k] + by_vol(a - ar) * dt;
        if (lane >= 2 && lane <= 29 && gx < p.ng + p.nx) p.u_next[svar(s, k, N) * p.plane + gx] = uu[k];
    }
    return FAST || WHERE != TRIED || __all_sync(0xffffffffu, inside);
}

// The strip with a denominator outside the range, out of line: the kernel keeps to the registers (72) and
// the code of the other form.
template <typename R, bool IS_GAS, int ST>
static __device__ __noinline__ void flux_line_wide(const KParams<R>& p, int s) { flux_line<R, IS_GAS, ST, ANYWHERE>(p, s); }

template <typename R, int ST>
__global__ void __launch_bounds__(32, 28) k_flux_line(const __grid_constant__ KParams<R> p) {
    chain_begin();
    if (blockIdx.y == 0) {
        if (!flux_line<R, true, ST, TRIED>(p, 0)) flux_line_wide<R, true, ST>(p, 0);
    } else {
        if (!flux_line<R, false, ST, TRIED>(p, blockIdx.y)) flux_line_wide<R, false, ST>(p, blockIdx.y);
    }
}

}  // namespace shark
