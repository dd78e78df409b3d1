// charge.cuh -- K5: grain charging, Marchand et al. (2021) Newton on the reduced grain potential
// psi per cell (src/chemistry/ionisation.f90:4-214), optionally seeded by the charging network.
//
// One thread per cell over every cell of the grid, ghosts included (the reference's active-cell
// test is commented out).  The cell's inputs come from the conserved state at the start of the
// step through the setup's map (host-built tables):
//   nH   = rho/hs * unit_nH                  hs = sqrt(2 pi) H for the 2D polar disk, else 1
//   n_k  = rho_k/hs * unit_d / (m_k unit_m)  m_k = 4/3 pi rhograin s_k^3
//   T    = per temperature row (one row, or one per column for the disk), with the T-only
//          constants sigmav_ie, vi, tau_k, alpha_k tabulated on the host
//   zeta = chg_x, attenuated by exp(-Sigma unit_d unit_l/chg_sigma_att) for the disk.
// R = double runs in FP64; R = float (mixed precision) runs the cold part of the iteration in FP32
// and finishes it in FP64.  Outputs: psi_old (FP64, the warm start of the
// next call), zd (N planes), ni, ne, and with SHARK_CHARGE_RESISTIVITIES eta_o/H/a and gamma_d,
// plus the per-call histogram of Newton iteration counts.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/shark_gpu.h"
#include "physics.cuh"

namespace shark {

constexpr int CHARGE_HIST = SHARK_CHARGE_HIST;   // histogram bins: iterations 0..62, the last >= 63

template <typename R>
struct ChargeParams {
    const R* u;                  // state (variable planes, pitch layout)
    long long plane;
    int pitch, nx_max, ny_max, ndust, nvar;
    int t_per_col;               // 1: temperature tables per column (disk), 0: one row
    int res;                     // compute the resistivities
    int use_seed;                // 0 none, 1 seed where psi_old == 0, 2 seed always
    const double* hs;            // [nx_max] column-to-midplane factor (nullptr: 1)
    const double* trow;          // [rows][8]: T, sigmav_ie, vi, cs_T, c_el, c_ions, sigmav_el, sigmav_ions
    // per species and temperature row, element k * rows + row
    const double* tau;
    const double* alpha;
    const double* ptau;          // pi l_k^2 / tau_k
    const double* ntau;          // nfac_k tau_k
    int rows;
    // per species
    const double* l2;            // grain radius^2 (cm^2)
    const double* mkum;          // grain mass (g)
    const double* nfac;          // unit_d / m_k (g): n_k = rho_k / hs * nfac_k
    const double* npl;           // nfac_k pi l_k^2
    const double* wk;            // sqrt(pi gamma/8) rhograin_cgs l_k / m_k: stopping time over mass, times rho_cgs cs
    const float4* tf;            // (alpha, 1/tau, pi l^2/tau, tau) at (2 k) * rows + row and (unit_d/m, pi l^2, 1/m,
                                 // sqrt(pi gamma/8) rhograin l) at (2 k + 1) * rows + row, FP32 (mixed path)
    double unH, ud, ul, x0, sig_att;
    double thetai, th2, th3, psi0, eps, B0, mu_ions;
    int nitermax;
    double* psi_old;             // [plane] FP64
    R* zd;                       // [N][plane]
    R* ni;                       // [plane]
    R* ne;
    R* eta;                      // [3][plane] (o, H, a)
    R* gamma_d;                  // [N][plane]
    const float* seed;           // [plane] network start points (nullptr: none)
    int32_t* iters;              // [plane] Newton iterations of the last call
    unsigned long long* hist;    // [CHARGE_HIST + 2]: histogram, non-converged cells, total iterations
    unsigned long long* stamps;  // [1]: device clock at the end of a step's charging (the latest block's); null outside a step
    unsigned int* status;        // the step's status word: SHARK_STATUS_NEWTON if a cell did not converge
};

namespace chg {
constexpr double pi = 3.141592653589793238462643383279;
constexpr double e_el = 4.8e-10, m_el = 9.109e-28, clight = 3e10, mH = 1.67e-24;
}

// Compensated FP32 sum (Kahan): s + c carries the sum of the added terms to ~1 ulp.
__device__ __forceinline__ void kahan_add(float& s, float& c, float x) {
    const float y = x - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

// The Newton iteration of ionisation.f90:79-135 with its species sums in psi-independent parts, formed
// once per cell,
//   T1 = sum n_k tau_k,  T3 = sum n_k pi l_k^2,
// and four sums per iteration over r_k = 1/(1 + et alpha_k + et^2), et = eps theta:
//   T2 = sum n_k r_k,  T4 = sum n_k pi l_k^2 r_k / tau_k,
//   S2 = sum n_k (A + B alpha_k) r_k^2,  S5 = sum n_k pi l_k^2 / tau_k (C + theta alpha_k) r_k^2,
//   n_i = -(psi T1 + (1 - et^2) T2)/(1 - eps),   S1 = (1 - psi) T3 + 2 (et^2 + et) T4;
// they are the reference's sums with the factors a cell's species share taken out.  The sums run on
// rho_k unit_d / m_k and take 1/hs afterwards.

// Quotients of the iteration's scalars: FP64 on reciprocals to an ulp, plain FP32 divisions.
__device__ __forceinline__ double recip(double b) { return rcp64_any(b); }
__device__ __forceinline__ float recip(float b) { return 1.0f / b; }

// f(psi) and its derivative from the iteration's sums, 1/hs in all of them, and the update of psi.
// Returns f at the psi it came with.
template <typename C>
__device__ __forceinline__ C charge_update(C T1, C T2, C T3, C T4, C S2, C S5, C eps_psi, C thetai, C rxnH, C sigmav_ie,
                                           C vi, C psi0, C& psi, int& lowT) {
    const C one = C(1), two = C(2);
    const C et = eps_psi * thetai, et2 = et * et, et21 = et2 + et, rom = recip(one - eps_psi);
    const C n_i = -(psi * T1 + (one - et2) * T2) * rom;
    const C S1 = (one - psi) * T3 + two * et21 * T4;
    const C nv = n_i * vi * rxnH, ns = sigmav_ie * n_i * rxnH;
    const C f = ns * eps_psi * n_i + nv * S1 - one;
    const C D = -eps_psi * (two - psi) * recip(one - psi);
    const C dni = -(rom * rom) * D * S2 - (psi * rom * D + one) * T1 * rom;
    const C q = dni * recip(n_i);
    const C df = ns * (n_i * D + two * eps_psi * dni) +
                 two * nv * et21 * ((q + D * (two * et + one) * recip(eps_psi * (one + et))) * T4 + D * S5) +
                 nv * (q * (one - psi) - one) * T3;
    psi = psi - f * recip(df);
    if (psi < psi0) {
        psi = psi0 * C(0.9999999);
        lowT = 1;
    } else if (psi > C(0)) {
        psi = C(-1e-5);
    }
    return f;
}

// FP32 iterations of the mixed path from a cold or network start, until |f| <= tol or psi stops moving.
// The residual is steep (|df/dpsi| ~ 1e2-1e3 at the root), so an FP32 psi pins f only to ~1e-4.
template <typename R>
__device__ __forceinline__ void charge_newton_f(const ChargeParams<R>& p, const float4* tf, const R* uk, float T1, float T3,
                                                float ihs, float nH, float x, float sigmav_ie, float vi, float tol,
                                                float& psi, int& niter, int& lowT) {
    const int N = p.ndust, rows = p.rows;
    const float th = (float)p.thetai, th2 = (float)p.th2, th3 = (float)p.th3, psi0 = (float)p.psi0;
    const float rxnH = 1.0f / (x * nH);
    float conv = 1e4f;
    while (conv > tol && niter < p.nitermax) {
        const float eps = (1.0f - psi) / th * expf(-psi), et = eps * th, et2 = et * et;
        const float A = -(et2 * et2) + 4.f * th2 * (eps * eps) - 4.f * th2 * eps + 1.f, B = -th3 * (eps * eps) + 2.f * th * eps - th;
        const float c5 = 2.f * eps * th2;
        float T2 = 0.f, T4 = 0.f, S2 = 0.f, S5 = 0.f;
        for (int k = 0; k < N; ++k) {
            const float4 a = tf[2 * k * rows];
            const float nf = (float)uk[(long long)k * p.plane] * tf[(2 * k + 1) * rows].x;
            const float r = 1.f / (1.f + et * a.x + et2);
            const float nr = nf * r, w = nr * a.z;
            T2 += nr;
            T4 += w;
            S2 += nr * r * (A + B * a.x);
            S5 += w * r * (c5 + th * a.x);
        }
        const float prev = psi;
        conv = fabsf(charge_update<float>(T1, ihs * T2, T3, ihs * T4, ihs * S2, ihs * S5, eps, th, rxnH, sigmav_ie, vi, psi0, psi, lowT));
        niter = niter + 1;
        if (psi == prev) break;
    }
}

// FP64 iterations to the reference's stopping test |f| < chg_eps.  FP64 path: the four sums in FP64.
// Mixed path: T2 and T4, corrections of a few per cent, in compensated FP32 (f accurate to ~1e-8), and
// the derivative's sums S2 and S5 in FP32 (Newton needs f' to a few digits).
template <typename R>
__device__ __forceinline__ void charge_newton_d(const ChargeParams<R>& p, int row, const R* uk, double T1, double T3, double ihs,
                                                double nH, double x, double sigmav_ie, double vi, double& psi, int& niter,
                                                int& lowT, double& conv) {
    const int N = p.ndust, rows = p.rows;
    const double th = p.thetai, th2 = p.th2, th3 = p.th3, psi0 = p.psi0;
    const double rth = rcp64(th), rxnH = rcp64_any(x * nH);
    while (conv > p.eps && niter < p.nitermax) {
        // eps is the reference's quotient to the bit: where the column shields the ions psi goes to -0 (1e-20 at
        // 4e3 g/cm2), et to 1, and the root lies where 1 - et^2 is exactly zero
        const double eps = div64_const(1.0 - psi, th, rth) * exp(-psi), et = eps * th, et2 = et * et;
        double T2, T4, S2, S5;
        if constexpr (sizeof(R) == 8) {
            const double *al = p.alpha + row, *pt = p.ptau + row;
            const double e2 = eps * eps, et21 = 1.0 + et2;
            const double A = fma(4.0 * th2, e2 - eps, fma(-et2, et2, 1.0)), B = fma(-th3, e2, fma(2.0 * th, eps, -th));
            const double C = 2.0 * eps * th2;
            T2 = T4 = S2 = S5 = 0.0;
            for (int k = 0; k < N; ++k) {
                const double a = al[(size_t)k * rows], nf = uk[(long long)k * p.plane] * p.nfac[k];
                const double r = rcp64(fma(et, a, et21));
                const double nr = nf * r, w = nr * pt[(size_t)k * rows];
                T2 += nr;
                T4 += w;
                S2 = fma(nr * r, fma(B, a, A), S2);
                S5 = fma(w * r, fma(th, a, C), S5);
            }
        } else {
            const float4* tf = p.tf + row;
            const float ef = (float)eps, etf = (float)et, et2f = (float)et2, thf = (float)th, th2f = (float)th2, th3f = (float)th3;
            const float c2a = -(et2f * et2f), c2b = ef * ef, c5 = 2.f * ef * th2f;
            float t2 = 0.f, k2 = 0.f, t4 = 0.f, k4 = 0.f, s2 = 0.f, s5 = 0.f;
            for (int k = 0; k < N; ++k) {
                const float4 a = tf[2 * k * rows];
                const float nf = (float)uk[(long long)k * p.plane] * tf[(2 * k + 1) * rows].x;
                const float r = 1.f / (1.f + etf * a.x + et2f);
                const float nr = nf * r;
                kahan_add(t2, k2, nr);
                kahan_add(t4, k4, nr * a.z);
                const float f2 = (c2a + (4.f * th2f - th3f * a.x) * c2b + (2.f * thf * a.x - 4.f * th2f) * ef + 1.f - thf * a.x) * r;
                s2 = s2 + nr * f2;
                s5 = s5 + nr * a.z * (c5 + thf * a.x) * r;
            }
            T2 = widen(t2); T4 = widen(t4); S2 = widen(s2); S5 = widen(s5);
        }
        const double prev = psi;
        conv = abs64(charge_update<double>(T1, ihs * T2, T3, ihs * T4, ihs * S2, ihs * S5, eps, th, rxnH, sigmav_ie, vi, psi0, psi, lowT));
        niter = niter + 1;
        // an unchanged psi with the residual above the tolerance repeats itself until nitermax
        // (e.g. the psi0 clamp): go there directly, same final state
        if (psi == prev && conv > p.eps) niter = p.nitermax;
    }
}

// Outputs (ionisation.f90:137-206): Z_k, n_i, n_e, psi_old and, with the resistivities, eta_o/H/a and
// gamma_d.  FP64 path: FP64 throughout.  Mixed path: the per-species terms are FP32 (the outputs are
// stored in FP32) with compensated sums; the cell-level electron and ion terms are FP64.
template <typename R>
__device__ __forceinline__ void charge_outputs(const ChargeParams<R>& p, int row, long long c, double ihs, double rho, double nH,
                                               double x, double sigmav_ie, const double* tr, double psi, double eps_psi, int lowT) {
    const int N = p.ndust, rows = p.rows;
    const R* uk = p.u + 5 * p.plane + c;
    const double e = chg::e_el, cl = chg::clight, mel = chg::m_el, mi = p.mu_ions * chg::mH;
    const double B = p.B0 * sqrt(nH / 1e4);
    const double irc = rcp64_any(rho * p.ud * tr[3]);   // t_sd = sqrt(pi gamma/8) rhograin l / (rho_cgs cs_T)
    const double eBc = e * B / cl;
    double zsum, so = 0.0, sp = 0.0, sh = 0.0;          // sums without 1/hs
    if constexpr (sizeof(R) == 8) {
        const double *ta = p.tau + row, *al = p.alpha + row;
        const double e2t = (eps_psi * eps_psi) * p.th2, et1 = eps_psi * p.thetai, ome = 1.0 - e2t, ope = 1.0 + e2t;
        const double wB = eBc * irc;
        zsum = 0.0;
        for (int k = 0; k < N; ++k) {
            const double den = fma(et1, al[(size_t)k * rows], ope);
            const double z = fma(psi, ta[(size_t)k * rows], ome * rcp64(den));
            p.zd[(long long)k * p.plane + c] = z;
            const double nz = uk[(long long)k * p.plane] * p.nfac[k] * z;
            zsum += nz;
            if (!p.res) continue;
            const double W = p.wk[k];
            const double sd = nz * z * W, wt = z * W * wB;
            const double q = abs_less(wt, 1e150) ? rcp64(fma(wt, wt, 1.0)) : 0.0;
            so += sd;
            sp = fma(sd, q, sp);
            sh = fma(sd, wt * q, sh);
            p.gamma_d[(long long)k * p.plane + c] = wt;
        }
        const double e2i = (e * e) * irc;
        so *= e2i; sp *= e2i; sh *= e2i;
    } else {
        const float4* tf = p.tf + row;
        const float psif = (float)psi, e2t = (float)((eps_psi * eps_psi) * p.th2), et1 = (float)(eps_psi * p.thetai);
        const float ircf = (float)irc, eBcf = (float)eBc, ef = (float)e;
        float zs = 0.f, kz = 0.f, fo = 0.f, ko = 0.f, fp = 0.f, kp = 0.f, fh = 0.f, kh = 0.f;
        for (int k = 0; k < N; ++k) {
            const float4 a = tf[2 * k * rows], b = tf[(2 * k + 1) * rows];
            const float z = psif * a.w + (1.f - e2t) / (1.f + et1 * a.x + e2t);
            const float nf = (float)uk[(long long)k * p.plane] * b.x;
            p.zd[(long long)k * p.plane + c] = R(z);
            kahan_add(zs, kz, z * nf);
            if (!p.res) continue;
            const float t_sd = b.w * ircf;
            const float ze = z * ef;
            const float sd = nf * b.z * (ze * ze) * t_sd;
            const float omd = z * eBcf * b.z;
            const float wt = omd * t_sd;
            const float q = 1.f / (1.f + wt * wt);
            const float h = fabsf(wt) > 1e18f ? 1.f / wt : wt * q;   // wt / (1 + wt^2) without overflow
            kahan_add(fo, ko, sd);
            kahan_add(fp, kp, sd * q);
            kahan_add(fh, kh, sd * h);
            p.gamma_d[(long long)k * p.plane + c] = R(wt);
        }
        zsum = zs; so = fo; sp = fp; sh = fh;
    }
    double nsum = -(ihs * zsum) * rcp64_any(1.0 - eps_psi);
    if (lowT > 0 && N > 0) nsum = sqrt(eps_psi * x * nH / sigmav_ie);
    p.ni[c] = R(nsum);
    p.ne[c] = R(eps_psi * nsum);
    p.psi_old[c] = lowT > 0 ? p.psi0 : psi;
    if (!p.res) return;
    const double rnH = rcp64_any(nH);
    const double t_sel = tr[4] * rnH, t_sions = tr[5] * rnH;
    const double sig_el = (eps_psi * nsum) * ((e * e) / mel) * t_sel;
    const double sig_i = (nsum) * ((e * e) / mi) * t_sions;
    const double we = -eBc / mel * t_sel, wi = eBc / mi * t_sions;
    const double qe = recip(1.0 + we * we), qi = recip(1.0 + wi * wi);
    const double sigma_o = ihs * so + sig_i + sig_el;
    const double sigma_p = sig_i * qi + sig_el * qe + ihs * sp;
    const double sigma_h = -sig_i * wi * qi - sig_el * we * qe - ihs * sh;
    const double ro = recip(sigma_o);
    p.eta[c] = R(ro);
    p.eta[p.plane + c] = R(sigma_h * recip(sigma_p * 2.0 + sigma_h * sigma_h));
    p.eta[2 * p.plane + c] = R(sigma_p * recip(sigma_p * sigma_p + sigma_h * sigma_h) - ro);
}

// K5.  A cell starts from psi_old (FP64, the last call's psi), cold from psi0 or the network's seed;
// the mixed path begins a cold or seeded cell with FP32 iterations.  The iteration count is the sum
// of both phases.  Bound by the FP64 pipe: per iteration FP64 spends 17 instructions for a species
// (some 160 as the reference's expressions, whose shared factors and invariants it re-formed) and
// some 75 for the cell, the mixed path those 75 and two a species for T1 and T3.  (With the derivative's
// scalars in FP32 the mixed path took 45, driven box 0.59 and polar disk 0.42 ms, and lost cells whose
// scalars leave FP32's range: shielded columns, test_gpu_charge_shielded.py.)
// Temperature tables are laid out species by species, so that a warp's columns read them together.
// Cold start, 384^2 x 32: FP64 24.4 -> 4.0 ms, mixed 1.54 -> 0.25; warm, driven box 768^2 x 32 mixed 1.00 ->
// 0.71 ms a step, polar disk 512 x 1024 x 16 0.675 -> 0.49, 128 x 256 x 16 FP64 0.68 -> 0.15.
template <typename R>
__global__ void __launch_bounds__(128) k_charge(ChargeParams<R> p) {
    const int N = p.ndust;
    const long long ncell = (long long)p.nx_max * p.ny_max;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    __shared__ unsigned int s_hist[CHARGE_HIST + 1];
    __shared__ unsigned long long s_iter;
    for (int b = threadIdx.x; b <= CHARGE_HIST; b += blockDim.x) s_hist[b] = 0u;
    if (threadIdx.x == 0) s_iter = 0ull;
    __syncthreads();
    if (t < ncell) {
        const int iy = (int)(t / p.nx_max), ix = (int)(t - (long long)iy * p.nx_max);
        const long long c = (long long)iy * p.pitch + ix;
        const int row = p.t_per_col ? ix : 0;
        const double* tr = p.trow + (size_t)row * 8;
        const double hs = p.hs ? p.hs[ix] : 1.0;
        const double u0 = (double)p.u[c];
        const double rho = u0 / hs;
        const double nH = rho * p.unH;
        double x = p.x0;
        if (p.sig_att > 0.0) x = p.x0 * exp(-(u0 * p.ud * p.ul) / p.sig_att);
        const double sigmav_ie = tr[1], vi = tr[2];
        const double psi0 = p.psi0;
        double psi = psi0, conv = 1e4;
        int niter = 0, lowT = 0;
        const double pold = p.psi_old[c];
        bool cold = true;
        if (pold != 0.0) { psi = pold; cold = false; }
        if (p.seed && (p.use_seed == 2 || (p.use_seed == 1 && pold == 0.0))) {
            const float sd = p.seed[c];
            if (sd < 0.0f) { psi = (double)sd; cold = true; }
        }
        const double ihs = 1.0 / hs;
        const R* uk = p.u + 5 * p.plane + c;
        double T1 = 0.0, T3 = 0.0;                 // psi-independent sums
        {
            const double* nt = p.ntau + row;
            for (int k = 0; k < N; ++k) {
                const double u = widen(uk[(long long)k * p.plane]);
                T1 = fma(u, nt[(size_t)k * p.rows], T1);
                T3 = fma(u, p.npl[k], T3);
            }
            T1 *= ihs;
            T3 *= ihs;
        }
        if (sizeof(R) == 4 && cold) {
            float psif = (float)psi;
            charge_newton_f(p, p.tf + row, uk, (float)T1, (float)T3, (float)ihs, (float)nH, (float)x, (float)sigmav_ie, (float)vi,
                            fmaxf((float)p.eps, 1e-3f), psif, niter, lowT);
            psi = (double)psif;
        }
        charge_newton_d(p, row, uk, T1, T3, ihs, nH, x, sigmav_ie, vi, psi, niter, lowT, conv);
        double eps_psi = (1.0 - psi) / p.thetai * exp(-psi);
        if (lowT > 0) eps_psi = 0.99999;
        charge_outputs(p, row, c, ihs, rho, nH, x, sigmav_ie, tr, psi, eps_psi, lowT);
        p.iters[c] = niter;
        atomicAdd(&s_hist[niter < CHARGE_HIST - 1 ? niter : CHARGE_HIST - 1], 1u);
        if (conv > p.eps) atomicAdd(&s_hist[CHARGE_HIST], 1u);
        atomicAdd(&s_iter, (unsigned long long)niter);
    }
    __syncthreads();
    for (int b = threadIdx.x; b <= CHARGE_HIST; b += blockDim.x)
        if (s_hist[b]) atomicAdd(&p.hist[b], (unsigned long long)s_hist[b]);
    if (threadIdx.x == 0 && s_iter) atomicAdd(&p.hist[CHARGE_HIST + 1], s_iter);
    if (threadIdx.x == 0 && s_hist[CHARGE_HIST] && p.status) atomicOr(p.status, (unsigned)SHARK_STATUS_NEWTON);
    if (threadIdx.x == 0 && p.stamps) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        atomicMax(p.stamps + 1, now);
    }
}

// Fujii et al. (2011) analytical charging (ionisation.f90:809-922, functions_NR.f90:15-128,
// newton_raphson.f90:7-97): per cell and species, Newton on the grain charge Z from -1 until
// |f| < 1e-14 or 1e5 iterations, FP64 in both precisions.  f is the small difference of two
// large, nearly equal terms, so its rounding stays above 1e-14 and the reference's loop runs its
// full 1e5 iterations; restated as written.  n_i, n_e are those of the last species (the
// reference overwrites them in its species loop).
__device__ __forceinline__ double fujii_f_d(double y, double zeta, double rho, double m_d, double rho_d, double s_d,
                                            double T, double mu_gas, double mu_ions, double* fp) {
    const double mH = chg::mH, kB = 1.38e-16, e = chg::e_el, pi = chg::pi;
    const double m_i = mu_ions * mH, m_e = chg::m_el;
    const double k_e = pi * (s_d * s_d) * sqrt(8 * kB * T / (pi * m_e)) * exp((e * e) * y / (s_d * kB * T));
    const double k_i = pi * (s_d * s_d) * sqrt(8 * kB * T / (pi * m_i)) * (1 - (e * e) * y / (s_d * kB * T));
    const double a = m_d * rho / (rho_d * mu_gas * mH);
    const double f = mu_gas * mH * zeta / rho * (a * a) * ((1 / k_i) - (1 / k_e)) - y;
    if (fp) {
        const double kp_e = pi * s_d * sqrt(8 * kB * T / pi / m_e) * (e * e) / kB / T * exp((e * e) * (y) / s_d / kB / T);
        const double kp_i = -pi * s_d * sqrt(8 * kB * T / pi / m_i) * (e * e) / kB / T;
        const double b = m_d * rho / rho_d / mu_gas / mH;
        *fp = mu_gas * mH * zeta / rho * (b * b) * (kp_e / (k_e * k_e) - kp_i / (k_i * k_i)) - 1;
    }
    return f;
}

template <typename R>
__global__ void __launch_bounds__(128) k_charge_fujii(ChargeParams<R> p, double smallr, double mu_gas, double ul) {
    const int N = p.ndust;
    const long long ncell = (long long)p.nx_max * p.ny_max;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    __shared__ unsigned int s_hist[CHARGE_HIST + 1];
    __shared__ unsigned long long s_iter;
    for (int b = threadIdx.x; b <= CHARGE_HIST; b += blockDim.x) s_hist[b] = 0u;
    if (threadIdx.x == 0) s_iter = 0ull;
    __syncthreads();
    if (t < ncell) {
        const int iy = (int)(t / p.nx_max), ix = (int)(t - (long long)iy * p.nx_max);
        const long long c = (long long)iy * p.pitch + ix;
        const int row = p.t_per_col ? ix : 0;
        const double T = p.trow[(size_t)row * 8];
        const double hs = p.hs ? p.hs[ix] : 1.0;
        const double u0 = (double)p.u[c];
        double x = p.x0;
        if (p.sig_att > 0.0) x = p.x0 * exp(-(u0 * p.ud * p.ul) / p.sig_att);
        const double rho = (u0 > smallr ? u0 : smallr) / hs * p.ud;
        int total = 0;
        unsigned int nconv = 0;
        double ni = 0.0, ne = 0.0;
        for (int k = 0; k < N; ++k) {
            const double m_d = p.mkum[k];
            const double rho_d = (double)p.u[(long long)(5 + k) * p.plane + c] / hs * p.ud;
            const double s_d = sqrt(p.l2[k]);
            double y = -1.0;
            int it;
            bool conv = false;
            for (it = 1; it <= 100000; ++it) {
                double fp;
                const double fy = fujii_f_d(y, x, rho, m_d, rho_d, s_d, T, mu_gas, p.mu_ions, &fp);
                if (fabs(fy) < 1.e-14) { conv = true; break; }
                y = y - fy / fp;
            }
            if (!conv) conv = fabs(fujii_f_d(y, x, rho, m_d, rho_d, s_d, T, mu_gas, p.mu_ions, nullptr)) <= 1.e-14;
            if (!conv) ++nconv;
            total += it - 1;
            p.zd[(long long)k * p.plane + c] = R(y);
            const double mH = chg::mH, kB = 1.38e-16, e = chg::e_el, pi = chg::pi;
            const double k_e = pi * (s_d * s_d) * sqrt(8 * kB * T / (pi * chg::m_el)) * exp((e * e) * y / (s_d * kB * T));
            const double k_i = pi * (s_d * s_d) * sqrt(8 * kB * T / (pi * (p.mu_ions * mH))) * (1 - (e * e) * y / (s_d * kB * T));
            ni = x * rho * m_d / (k_i * mu_gas * mH * rho_d);
            ne = x * rho * m_d / (k_e * mu_gas * mH * rho_d);
        }
        p.ni[c] = R(ni);
        p.ne[c] = R(ne);
        p.iters[c] = total;
        atomicAdd(&s_hist[total < CHARGE_HIST - 1 ? total : CHARGE_HIST - 1], 1u);
        if (nconv) atomicAdd(&s_hist[CHARGE_HIST], nconv);
        atomicAdd(&s_iter, (unsigned long long)total);
    }
    __syncthreads();
    for (int b = threadIdx.x; b <= CHARGE_HIST; b += blockDim.x)
        if (s_hist[b]) atomicAdd(&p.hist[b], (unsigned long long)s_hist[b]);
    if (threadIdx.x == 0 && s_iter) atomicAdd(&p.hist[CHARGE_HIST + 1], s_iter);
    if (threadIdx.x == 0 && s_hist[CHARGE_HIST] && p.status) atomicOr(p.status, (unsigned)SHARK_STATUS_NEWTON);
    if (threadIdx.x == 0 && p.stamps) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        atomicMax(p.stamps + 1, now);
    }
}

// Network features of the cells (SHARK_MLP_NFEAT floats per cell, plane layout [plane][F]):
// log10 nH, log10 T, log10 zeta, log10 of the grain cross-section, radius and number per H
// (sum_k n_k pi a_k^2 / nH, sum_k n_k a_k / nH, sum_k n_k / nH).  The same state -> input map as
// k_charge.  Pad columns of the plane get zeros.
template <typename R>
__global__ void __launch_bounds__(128) k_charge_features(ChargeParams<R> p, float* __restrict__ feat) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= p.plane) return;
    const int iy = (int)(t / p.pitch), ix = (int)(t - (long long)iy * p.pitch);
    float* f = feat + t * SHARK_MLP_NFEAT;
    if (ix >= p.nx_max) {
        for (int i = 0; i < SHARK_MLP_NFEAT; ++i) f[i] = 0.0f;
        return;
    }
    const int N = p.ndust;
    const int row = p.t_per_col ? ix : 0;
    const double T = p.trow[(size_t)row * 8];
    const double hs = p.hs ? p.hs[ix] : 1.0;
    const double rho = (double)p.u[t] / hs;
    const double nH = rho * p.unH;
    double x = p.x0;
    if (p.sig_att > 0.0) x = p.x0 * exp(-((double)p.u[t] * p.ud * p.ul) / p.sig_att);
    double s2 = 0.0, s1 = 0.0, s0 = 0.0;
    for (int k = 0; k < N; ++k) {
        const double n = ((double)p.u[(long long)(5 + k) * p.plane + t] / hs) * p.ud / p.mkum[k];
        s2 += n * chg::pi * p.l2[k];
        s1 += n * sqrt(p.l2[k]);
        s0 += n;
    }
    f[0] = (float)log10(nH);
    f[1] = (float)log10(T);
    f[2] = (float)log10(x);
    f[3] = (float)log10(s2 / nH);
    f[4] = (float)log10(s1 / nH);
    f[5] = (float)log10(s0 / nH);
}

// Append (features, t = psi/psi0 - 1) of every cell the last charging call converged to the
// network's training set (cap rows of SHARK_MLP_NFEAT + 1 floats; `count` is the fill level).
template <typename R>
__global__ void k_charge_collect(ChargeParams<R> p, const float* __restrict__ feat, float* __restrict__ out,
                                 unsigned long long* count, long long cap) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= p.plane) return;
    const int iy = (int)(t / p.pitch), ix = (int)(t - (long long)iy * p.pitch);
    if (ix >= p.nx_max || iy >= p.ny_max) return;
    if (p.iters[t] >= p.nitermax) return;
    const unsigned long long slot = atomicAdd(count, 1ull);
    if ((long long)slot >= cap) return;
    float* o = out + slot * (SHARK_MLP_NFEAT + 1);
    for (int i = 0; i < SHARK_MLP_NFEAT; ++i) o[i] = feat[t * SHARK_MLP_NFEAT + i];
    o[SHARK_MLP_NFEAT] = (float)(p.psi_old[t] / p.psi0 - 1.0);
}

}  // namespace shark
