// step_kernels.cuh -- the device kernels of one `solve` step (src/solver/solve.f90:10-181).
//
//   k_boundaries   apply_boundaries of the setup (ghost fill), before anything reads the halo
//   k_prepare_step the step's dt and status to the host, the next dt's slot, constant drag coefficients
//   k_flux_*       K1: per species: ctoprim, limited slopes, MUSCL-Hancock predictor, Riemann fluxes
//                  (HLLC/HLL/LLF gas, Huang-Bai/LLF/HLL/HLLC dust), force kick, conservative update
//                  and the local source terms, a warp marching over its columns with the rows in
//                  registers (flux_line.cuh in 1D, flux_strip*.cuh in 2D).  No qm/qp/flux array ever
//                  reaches HBM.
//   k_finalize*    K2: per cell, all species: implicit multi-species drag, dust floor, setup_inloop,
//                  status checks, the CFL dt of the NEXT step (courant on the final state: warp
//                  shuffle -> block -> one atomicMin) and the next step's ghost cells.
//   k_growth_*     dust growth without fragmentation, between K2's drag and the rest of it
//
// Device state layout: variable-major planes, each plane ny_max rows of `pitch` elements
// (pitch >= nx_max, rounded up to 32 elements so every row starts 128-byte aligned), ghost cells
// stored.  Element (v, iy, ix) lives at v*plane + iy*pitch + ix.
#pragma once

#include "physics.cuh"
#include "growth.cuh"
#include "launch.h"
#include "../../include/shark_gpu.h"

namespace shark {

template <typename R>
struct KParams {
    // grid
    int nx, ny, ng, nx_max, ny_max, pitch;
    long long plane;
    int ndust, nvar, ndim, geom, solver, solverdust, slope_type, iso, setup, flags;
    int sod_dir;
    int strip_h;                      // rows a warp of the column-march flux kernel updates
    double gamma, cfl, smallr, smallp, dust_ratio_min, box_l, rhograin;
    double si_q, si_om, si_eta, si_r0;
    double sod_rho_l, sod_rho_r, sod_P_l, sod_P_r;
    // per-column metrics (length nx_max), compute precision
    const R *dx1, *dx2, *surf1, *surf2, *vol, *radc, *xpos, *cs;
    const R *sfx, *sfy, *irp, *rvol;   // division-free tables (mixed path)
    const R* fgrav;                    // polar disk: -Mstar/r^2 (0 for the other setups)
    const R* etav;                     // polar disk: kinematic viscosity alpha H cs
    int visc;                          // viscosity source term on
    // per-column metrics in FP64 (courant, drag)
    const double *dx1d, *dx2d, *radcd, *xposd, *csd;
    // polar disk per-column FP64 tables: gravity, relaxation time (0 = no relaxation),
    // sqrt(2 pi) H, FARGO orbital velocity
    const double *fgravd, *treld, *hsd, *vkd;
    const R* u_init;                   // polar disk relaxation reference state
    GrowthDev gw;                      // dust growth tables and constants
    int ou_nm;                         // dustyTurb forcing modes (0: no forcing)
    const double* ou;                  // [2 nm] this step's coefficients
    const float* ou_f;                 // mixed path, this step: k_x', k_y', k_y'/k, k_x'/k of the modes,
                                       // then the coefficients
    const double* ou_modes;            // [3 nm]
    double box_l_y;
    const R* chg_eta;                  // charging outputs: eta (3 planes), gamma_d (N planes)
    const R* chg_gamma_d;
    // per-species constants
    const double *dK, *dtstop, *dsize, *dstokes;
    const double* dinvts;             // 1/C_k, t_k = C_k / F_cell (dustyTurb, Epstein, polar disk)
    double turb_rho0;
    // time step bookkeeping
    const double* dt;                 // dt of the current step
    unsigned long long* stamps;       // device clock at the step's phases (DeviceView)
    unsigned long long* dt_next;      // bit image of the next dt (positive doubles order as u64)
    unsigned int* status;             // SHARK_STATUS_* bits
    float* coef;                      // [2*SHARK_MAX_DUST] per-step drag coefficients 1/(1+a_k), a_k/(1+a_k)
    const float* dtf;                 // (float) dt of the current step, coef[2*SHARK_MAX_DUST]
    const float* dinvts_f;            // 1/C_k as float (mixed path)
    // FP32 copies of the scalar parameters for the mixed kernels, converted once on the host: a
    // double-to-float conversion issues on the FP64 pipe, which is narrow and variable-latency on
    // this GPU, so per-thread conversions stall the warps that do them
    float f_gamma, f_gm1, f_inv_g1, f_cfl, f_smallr, f_smallp, f_dust_ratio_min, f_box_l, f_half_box_l;
    float f_si_q, f_si_om, f_si_r0, f_si_eta;
    float f_rho_ref;                  // reference gas density of the mixed flux kernel (0: none)
    // Cartesian disk per-cell tables (null for the other setups), plane layout: sound speed,
    // force x, force y and viscosity in the kernel's precision; FP64 sound speed and sqrt(2 pi H);
    // the setup_inloop targets (7 FP64 planes, rho_ana = 0 outside the buffers); the ghost state
    // (2 nvar: the value every ghost takes, then the top ghosts' source of the first fill)
    const R *ccs, *cfx, *cfy, *ceta;
    const double *ccsd, *chsd, *ctgt;
    R* cgs;
    const R* u_cur;                   // state at the start of the step (read only)
    R* u_next;                        // state after the step
};

// The device clock in ns.
__device__ __forceinline__ unsigned long long clock_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// K2's start (its first block) and end (the latest of its blocks): a store, and a reduction a block that
// nothing waits for, in place of two timing events a step (some 2 us each).
__device__ __forceinline__ void stamp_start(unsigned long long* stamps) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) stamps[2] = clock_ns();
}
__device__ __forceinline__ void stamp_end(unsigned long long* stamps) {
    if (threadIdx.x == 0) atomicMax(stamps + 3, clock_ns());
}

// Start of a kernel that may be launched before its predecessor in the stream has ended (launch_chained
// in kernels_impl.cuh): wait for the predecessor, then let the successor's blocks come in as this grid's
// make room.  In that order what a kernel reads ahead of its wait (loads through restricted pointers
// may be moved there) was written by grids that had ended before the predecessor's wait returned: the
// current state, by the step before, and tables.  The state that the predecessor writes, the dt and the
// coefficients go through plain pointers, behind the wait.
__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// A scalar parameter in the kernel's precision: the double itself, or its float copy.
template <typename R>
__device__ __forceinline__ R prm(double d, float f) {
    if constexpr (std::is_same<R, float>::value) return f;
    else return d;
}

// dt of the current step in the kernel's precision (the float copy k_prepare_step wrote).
template <typename R>
__device__ __forceinline__ R step_dt(const KParams<R>& p) {
    if constexpr (std::is_same<R, float>::value) return *p.dtf;
    else return *p.dt;
}

template <typename R>
__device__ __forceinline__ long long uidx(const KParams<R>& p, int v, int iy, int ix) {
    return (long long)v * p.plane + (long long)iy * p.pitch + ix;
}

// Global variable index of component c (0 rho, 1 vx, 2 vy, 3 vz) of species s (0 gas, k+1 dust k)
__device__ __forceinline__ int svar(int s, int c, int N) {
    return s == 0 ? c : 5 + c * N + (s - 1);
}

// Values of `n` variables of one cell at a time, all loads in flight before the first store: a store
// may alias the next load for all the compiler knows, so a loop that copies variable by variable
// waits for memory once a variable.
constexpr int COPY_BATCH = 8;
template <typename R, typename L, typename S>
__device__ __forceinline__ void in_batches(int n, L load, S store) {
    constexpr int B = COPY_BATCH;
    for (int v0 = 0; v0 < n; v0 += B) {
        R val[B];
#pragma unroll
        for (int i = 0; i < B; ++i)
            if (v0 + i < n) val[i] = load(v0 + i);
#pragma unroll
        for (int i = 0; i < B; ++i)
            if (v0 + i < n) store(v0 + i, val[i]);
    }
}

// ---------------------------------------------------------------------------------------------
// Boundaries: one thread per ghost cell.  Periodic and shear-periodic fills are done in a single
// pass with the source at (wrap(ix), wrap(iy)); this equals the reference's two passes (y rows for
// the active columns, then x columns over all rows, src/grid/boundary_types.f90:149-186 and
// src/setups/SI/boundaries.f90:1-81) because the x pass copies values that the y pass produced.
// ---------------------------------------------------------------------------------------------
template <typename R>
__global__ void k_boundaries(KParams<R> p, R* u) {
    const int ng = p.ng, nx = p.nx, ny = p.ny;
    const long long nghost_rows = (p.ndim == 2) ? 2LL * ng * p.nx_max : 0;  // y-ghost rows, full width
    const long long nghost_cols = 2LL * ng * (p.ndim == 2 ? ny : 1);          // x-ghost columns, active rows
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= nghost_rows + nghost_cols) return;
    int ix, iy;
    if (t < nghost_rows) {
        int r = (int)(t / p.nx_max);
        ix = (int)(t % p.nx_max);
        iy = r < ng ? r : ny + r;          // rows 0..ng-1 and ny+ng..ny+2ng-1
    } else {
        long long c = t - nghost_rows;
        int col = (int)(c % (2 * ng));
        iy = (p.ndim == 2) ? (int)(c / (2 * ng)) + ng : 0;
        ix = col < ng ? col : nx + col;
    }
    const bool xg = (ix < ng) || (ix >= ng + nx);
    const bool yg = (p.ndim == 2) && ((iy < ng) || (iy >= ng + ny));
    const int sx = ix < ng ? ix + nx : (ix >= ng + nx ? ix - nx : ix);
    const int sy = (p.ndim == 2) ? (iy < ng ? iy + ny : (iy >= ng + ny ? iy - ny : iy)) : 0;
    const int N = p.ndust;
    if (p.setup == SHARK_SETUP_SOD) {
        // fixed states along the shock direction (SOD/boundaries.f90:49-77), periodic otherwise
        const bool fixed = (p.sod_dir == 0) ? xg : yg;
        if (fixed) {
            const bool left = (p.sod_dir == 0) ? (ix < ng) : (iy < ng);
            const double g1 = p.gamma - 1.0;
            u[uidx(p, 0, iy, ix)] = R(left ? p.sod_rho_l : p.sod_rho_r);
            u[uidx(p, 1, iy, ix)] = R(0);
            u[uidx(p, 2, iy, ix)] = R(0);
            u[uidx(p, 3, iy, ix)] = R(0);
            u[uidx(p, 4, iy, ix)] = R((left ? p.sod_P_l : p.sod_P_r) / g1);
            return;
        }
    }
    if (p.setup == SHARK_SETUP_DISK_POLAR) {
        // disk_polar/boundaries.f90:1-70: periodic in phi; a radial ghost takes the first (last)
        // active cell of its row, phi image included, with the radial velocities clipped so that
        // nothing flows in (the reference's row-less u_prim(first_active) read as the row's cell)
        const int rx = ix < ng ? ng : (ix >= ng + nx ? ng + nx - 1 : ix);
        in_batches<R>(p.nvar, [&](int v) { return u[uidx(p, v, sy, rx)]; }, [&](int v, R val) { u[uidx(p, v, iy, ix)] = val; });
        if (xg) {
            for (int k = -1; k < N; ++k) {
                const long long i = uidx(p, k < 0 ? 1 : 5 + N + k, iy, ix);
                const R val = u[i];
                u[i] = ix < ng ? (val > R(0) ? val : R(0)) : (val < R(0) ? val : R(0));
            }
        }
        return;
    }
    in_batches<R>(p.nvar, [&](int v) { return u[uidx(p, v, sy, sx)]; }, [&](int v, R val) { u[uidx(p, v, iy, ix)] = val; });
    if (p.setup == SHARK_SETUP_SI && xg) {
        // shear: vz momentum -/+ rho * q * Omega * L (SI/boundaries.f90:60-74)
        const R sgn = ix < ng ? R(-1) : R(1);
        const R qsh = R(p.si_q), om = R(p.si_om), L = R(p.box_l);
        auto shear = [&](int k) {   // gas, then the species
            const long long z = uidx(p, k == 0 ? 3 : 4 + 3 * N + k, sy, sx), r = uidx(p, k == 0 ? 0 : 4 + k, sy, sx);
            return u[z] + sgn * (u[r] * qsh * om * L);
        };
        in_batches<R>(N + 1, shear, [&](int k, R val) { u[uidx(p, k == 0 ? 3 : 4 + 3 * N + k, iy, ix)] = val; });
    }
    (void)yg;
}

}  // namespace shark

#include "flux_line.cuh"
#include "flux_strip.cuh"
#include "flux_strip2.cuh"

namespace shark {

// ---------------------------------------------------------------------------------------------
// K2: drag + floor + inloop + status + next-step CFL dt, one thread per active cell.
// NS > 0: compile-time species count (register arrays); NS < 0: run-time count.
// MODE 0: full finalize; MODE 1: dt only (first step after an upload); MODES 2 and 3: the drag with
// its floor and heating, and the rest, as two launches with the growth kernel between them.
// ---------------------------------------------------------------------------------------------

// Producer-side boundary fill: the block with an active cell within nghost of a periodic or
// shear-periodic edge writes that cell's ghost images (with the SI shear of the vz momenta for x
// images) from its final values.  This is apply_boundaries of the next step (SI/boundaries.f90,
// boundary_types.f90:149-186, SOD/boundaries.f90 periodic directions) done by the producer; fixed SOD
// ghosts never change after the upload and are skipped.  Called by every thread of a block after a
// barrier behind the cells' last writes.  The images of a row's ends are shared out among the block's
// threads, a value each: left to the two threads of the edge cells they were nvar waits for memory,
// in two of eight blocks of a 1024-column row (K2 in us, SI 128^2 x 8 14.7 -> 11.4, 1024^2 x 8 79 -> 66, Cartesian disk
// 512^2 x 4 38 -> 29).
template <typename R>
__device__ __forceinline__ void fill_ghost_images(const KParams<R>& p, R* u, int gx, int gy) {
    const int ng = p.ng, nx = p.nx, ny = p.ny, N = p.ndust;
    const int x0 = gx - threadIdx.x, x1 = min(x0 + (int)blockDim.x, ng + nx);   // the block's columns [x0, x1)
    const bool lft = x0 == ng, rgt = x1 == ng + nx;
    const int items = ng * p.nvar;   // of one end of the row: variable v = it / ng, column c = it % ng
    if (p.setup == SHARK_SETUP_DISK_CART) {
        // zero_gradients as written (boundary_types.f90:48-100) from the second call on: every
        // ghost takes the state of cell (first_active, 1), which no step changes (k_cdisk_ghosts
        // does the first call).  The active cells on the edge write the ghosts next to them.
        const bool b = gy == ng, t = gy == ng + ny - 1;
        if (!(lft || rgt || b || t)) return;
        if ((b || t) && gx < x1) {
            in_batches<R>(p.nvar, [&](int v) { return p.cgs[v]; }, [&](int v, R val) {
                for (int g = 0; g < ng; ++g) {
                    if (b) u[uidx(p, v, g, gx)] = val;
                    if (t) u[uidx(p, v, ng + ny + g, gx)] = val;
                }
            });
        }
        if (!(lft || rgt)) return;
        for (int it = threadIdx.x; it < items; it += blockDim.x) {
            const int v = it / ng, c = it - v * ng;
            const R val = p.cgs[v];
            if (lft) u[uidx(p, v, gy, c)] = val;
            if (rgt) u[uidx(p, v, gy, ng + nx + c)] = val;
            for (int g = 0; g < ng; ++g) {   // corners
                if (lft && b) u[uidx(p, v, g, c)] = val;
                if (rgt && b) u[uidx(p, v, g, ng + nx + c)] = val;
                if (lft && t) u[uidx(p, v, ng + ny + g, c)] = val;
                if (rgt && t) u[uidx(p, v, ng + ny + g, ng + nx + c)] = val;
            }
        }
        return;
    }
    const bool polar = p.setup == SHARK_SETUP_DISK_POLAR;
    const bool xper = !polar && !(p.setup == SHARK_SETUP_SOD && p.sod_dir == 0);
    const bool yper = p.ndim == 2 && !(p.setup == SHARK_SETUP_SOD && p.sod_dir == 1);
    int ty = -1;   // this row's image across the periodic seam
    if (yper) {
        if (gy < 2 * ng) ty = gy + ny;
        else if (gy >= ny) ty = gy - ny;
    }
    if (ty >= 0 && gx < x1) {   // y images (no shear)
        const int src = gy * p.pitch + gx, dst = ty * p.pitch + gx, pl = (int)p.plane;
        in_batches<R>(p.nvar, [&](int v) { return u[src + v * pl]; }, [&](int v, R val) { u[dst + v * pl] = val; });
    }
    if (polar) {
        // disk_polar/boundaries.f90:1-70 by the producer: the first (last) active column's cell in its
        // row's radial ghosts (and their phi images) with the radial velocities clipped to outflow
        if (!(lft || rgt)) return;
        for (int it = threadIdx.x; it < items; it += blockDim.x) {
            const int v = it / ng, c = it - v * ng;
            const bool vr = v == 1 || (v >= 5 + N && v < 5 + 2 * N);
            if (lft) {
                R val = u[uidx(p, v, gy, ng)];
                if (vr) val = val > R(0) ? val : R(0);
                u[uidx(p, v, gy, c)] = val;
                if (ty >= 0) u[uidx(p, v, ty, c)] = val;
            }
            if (rgt) {
                R val = u[uidx(p, v, gy, ng + nx - 1)];
                if (vr) val = val < R(0) ? val : R(0);
                u[uidx(p, v, gy, ng + nx + c)] = val;
                if (ty >= 0) u[uidx(p, v, ty, ng + nx + c)] = val;
            }
        }
        return;
    }
    // sources of the right ghosts: columns [ng, 2 ng); of the left ghosts: the others from column nx on
    if (!xper || !(x0 < 2 * ng || x1 > nx)) return;
    const bool shear = p.setup == SHARK_SETUP_SI;
    const R qoL = prm<R>(p.si_q, p.f_si_q), om = prm<R>(p.si_om, p.f_si_om), L = prm<R>(p.box_l, p.f_box_l);
    for (int it = threadIdx.x; it < 2 * items; it += blockDim.x) {
        const bool left = it >= items;   // a left ghost
        const int i = left ? it - items : it, v = i / ng, c = i - v * ng;
        const int sx = left ? nx + c : ng + c, tx = left ? c : ng + nx + c;
        if (sx < x0 || sx >= x1 || (left && sx < 2 * ng)) continue;
        R val = u[uidx(p, v, gy, sx)];
        // vz momenta of the gas and the species: -/+ rho q Omega L (right ghost: +)
        if (shear && (v == 3 || v >= 5 + 3 * N))
            val = val + R(left ? -1 : 1) * (u[uidx(p, v == 3 ? 0 : v - 3 * N, gy, sx)] * qoL * om * L);
        u[uidx(p, v, gy, tx)] = val;                            // x image
        if (ty >= 0) u[uidx(p, v, ty, tx)] = val;               // corner image
    }
}

__device__ __forceinline__ void atomic_min_dt(unsigned long long* a, double v) {
    // positive finite doubles order like their bit patterns
    atomicMin(a, (unsigned long long)__double_as_longlong(v));
}

// Block-wide min of the CFL candidates and OR of the status bits, then one atomic per block.
// Every thread of the block must call it (no early return before it).
__device__ __forceinline__ void block_reduce_dt(double dtc, unsigned int st, unsigned long long* dt_next,
                                                unsigned int* status) {
    for (int o = 16; o > 0; o >>= 1) {   // positive doubles order as their bits
        const double other = __shfl_xor_sync(0xffffffffu, dtc, o);
        dtc = abs_less(other, dtc) ? other : dtc;
        st |= __shfl_xor_sync(0xffffffffu, st, o);
    }
    __shared__ double wmin[32];
    __shared__ unsigned int wst[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) { wmin[wid] = dtc; wst[wid] = st; }
    __syncthreads();
    if (wid == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        dtc = lane < nw ? wmin[lane] : 2e44;
        st = lane < nw ? wst[lane] : 0u;
        for (int o = 16; o > 0; o >>= 1) {
            const double other = __shfl_xor_sync(0xffffffffu, dtc, o);
            dtc = abs_less(other, dtc) ? other : dtc;
            st |= __shfl_xor_sync(0xffffffffu, st, o);
        }
        if (lane == 0) {
            atomic_min_dt(dt_next, dtc);
            if (st) atomicOr(status, st);
        }
    }
}

// FP32 form for the mixed path, whose CFL candidates are FP32: the min runs in FP32 (the FP64
// pipe is narrow) and the block's result is widened once for the atomic.  No candidate: 2e38f.
__device__ __forceinline__ void block_reduce_dt_f(float dtc, unsigned int st, unsigned long long* dt_next,
                                                  unsigned int* status) {
    for (int o = 16; o > 0; o >>= 1) {
        dtc = fminf(dtc, __shfl_xor_sync(0xffffffffu, dtc, o));
        st |= __shfl_xor_sync(0xffffffffu, st, o);
    }
    __shared__ float wminf[32];
    __shared__ unsigned int wstf[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) { wminf[wid] = dtc; wstf[wid] = st; }
    __syncthreads();
    if (wid == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        dtc = lane < nw ? wminf[lane] : 2e38f;
        st = lane < nw ? wstf[lane] : 0u;
        for (int o = 16; o > 0; o >>= 1) {
            dtc = fminf(dtc, __shfl_xor_sync(0xffffffffu, dtc, o));
            st |= __shfl_xor_sync(0xffffffffu, st, o);
        }
        if (lane == 0) {
            atomic_min_dt(dt_next, dtc >= 2e38f ? 2e44 : (double)dtc);
            if (st) atomicOr(status, st);
        }
    }
}

// Where a denominator formed from the state lies: from floats it cannot leave the range of div64_const.
template <typename R> constexpr int STATE_RANGE = std::is_same<R, float>::value ? CONSTANT : ANYWHERE;

// Sound speed of the cell at the start of the step: the isothermal column value, or ctoprim's
// sqrt(gamma P / max(rho, smallr)) of the adiabatic state (solve.f90:205-233).
template <typename R>
__device__ __forceinline__ double cs_start(const KParams<R>& p, int gx, int gy) {
    if (p.iso == 1) return p.ccsd ? p.ccsd[(long long)gy * p.pitch + gx] : p.csd[gx];
    const double rho = widen(p.u_cur[uidx(p, 0, gy, gx)]);
    const Over<double, STATE_RANGE<R>> by_rho(rho);
    const double vx = by_rho(widen(p.u_cur[uidx(p, 1, gy, gx)])), vy = by_rho(widen(p.u_cur[uidx(p, 2, gy, gx)]));
    const double vz = by_rho(widen(p.u_cur[uidx(p, 3, gy, gx)]));
    const double hr = 0.5 * rho;
    const double ekin = hr * (vx * vx) + hr * (vy * vy) + hr * (vz * vz);
    double P = (p.gamma - 1.0) * (widen(p.u_cur[uidx(p, 4, gy, gx)]) - ekin);
    P = max64_pos(P, p.smallp);
    const Over<double, STATE_RANGE<R>> by_q(max64_pos(rho, p.smallr));
    return sqrt(by_q(p.gamma * P));
}

// Stopping times of a cell's species from the state at the start of the step (compute_tstop runs
// before the update, solve.f90:34-35); qrho_old = max(rho_old, smallr).  What the species share (the
// sound speed, the reciprocals) is formed once per cell.
template <typename R, int WHERE = STATE_RANGE<R>>
struct TStop {
    const KParams<R>& p;
    long long cell;
    double c0;
    Over<double, WHERE> by_q, by_d;   // qrho_old; the sound speed (dustyTurb) or Epstein's rho cs
    __device__ __forceinline__ TStop(const KParams<R>& p_, double qrho_old, int gx, int gy)
        : p(p_), cell((long long)gy * p_.pitch + gx), c0(0.0),
          by_q(p_.setup == SHARK_SETUP_DUSTYWAVE || p_.setup == SHARK_SETUP_DUSTYTURB ? qrho_old : 1.0),
          by_d(denominator(p_, qrho_old, gx, gy)) {
        constexpr double pi = 3.141592653589793238462643383279;
        if (p.setup == SHARK_SETUP_DUSTYTURB) c0 = p.turb_rho0;
        else if (p.setup != SHARK_SETUP_SI && p.setup != SHARK_SETUP_DUSTYWAVE) c0 = sqrt(pi * p.gamma / 8.0) * (p.rhograin);
    }
    static __device__ __forceinline__ double denominator(const KParams<R>& p, double qrho_old, int gx, int gy) {
        if (p.setup == SHARK_SETUP_SI || p.setup == SHARK_SETUP_DUSTYWAVE) return 1.0;
        if (p.setup == SHARK_SETUP_DUSTYTURB) return p.csd[gx];
        if (p.setup == SHARK_SETUP_DISK_POLAR)   // Epstein on the midplane density Sigma/(sqrt(2 pi) H)
            return Over<double, CONSTANT>(p.hsd[gx])(qrho_old) * p.csd[gx];
        if (p.setup == SHARK_SETUP_DISK_CART) {  // disk/setup.f90 compute_tstop: Sigma/sqrt(2 pi H)
            const long long e = (long long)gy * p.pitch + gx;
            return Over<double, CONSTANT>(p.chsd[e])(qrho_old) * p.ccsd[e];
        }
        // Epstein (SOD/setup.f90:179-185) with the cell's sound speed
        return qrho_old * cs_start(p, gx, gy);
    }
    __device__ __forceinline__ bool inside() const { return by_q.inside() && by_d.inside(); }
    __device__ __forceinline__ double operator()(int k) const {
        if (p.setup == SHARK_SETUP_SI) return p.dtstop[k];                       // SI/setup.f90:389-397
        if (p.setup == SHARK_SETUP_DUSTYWAVE)                                    // DUSTYWAVE/setup.f90:217
            return by_q(Over<double, CONSTANT>(p.dK[k])((double)p.u_cur[(5 + k) * p.plane + cell] * by_q.b));
        if (p.setup == SHARK_SETUP_DUSTYTURB)                                    // dustyTurb/setup.f90:456
            return by_q(by_d(p.dstokes[k] * p.box_l * c0));
        return by_d(c0 * p.dsize[k]);
    }
};

// Drag heating of an adiabatic gas with back reaction (source_terms.f90:88-97): the energy
// gains sum_k dt v.(v - v_k)/t_k with the velocities and stopping times at the start of the step.
// WHERE = TRIED: `inside` becomes false where a denominator lies outside div64_const's range.
template <typename R, int WHERE>
__device__ __forceinline__ double drag_heating(const KParams<R>& p, const TStop<R, WHERE>& tstop, int gx, int gy, double dt,
                                               bool& inside) {
    const int N = p.ndust;
    const double rho = (double)p.u_cur[uidx(p, 0, gy, gx)];
    const Over<double, WHERE> by_rho(rho);
    inside = tstop.inside() && by_rho.inside();
    const double vx = by_rho((double)p.u_cur[uidx(p, 1, gy, gx)]), vy = by_rho((double)p.u_cur[uidx(p, 2, gy, gx)]);
    const double vz = by_rho((double)p.u_cur[uidx(p, 3, gy, gx)]);
    double S = 0.0;
    for (int k = 0; k < N; ++k) {
        const Over<double, WHERE> by_ts(tstop(k)), by_rd((double)p.u_cur[uidx(p, 5 + k, gy, gx)]);
        inside = inside && by_ts.inside() && by_rd.inside();
        const double vdx = by_rd((double)p.u_cur[uidx(p, 5 + N + k, gy, gx)]);
        const double vdy = by_rd((double)p.u_cur[uidx(p, 5 + 2 * N + k, gy, gx)]);
        const double vdz = by_rd((double)p.u_cur[uidx(p, 5 + 3 * N + k, gy, gx)]);
        S = S + by_ts(dt * (vx * (vx - vdx))) + by_ts(dt * (vy * (vy - vdy))) + by_ts(dt * (vz * (vz - vdz)));
    }
    return S;
}

// setup_inloop of the polar disk (disk_polar/setup.f90:206-284) for one active cell, FP64 or
// FP32 arithmetic: the first active column is reset to its initial state; inside r_relax the
// density and in-plane velocities of gas and dust relax towards the initial state with
// exp(-dt/t_rel).  Returns true when it changed the cell.
template <typename R, typename C>
__device__ __forceinline__ bool disk_inloop_cell(const KParams<R>& p, R* u, int gx, int gy, double dt) {
    const int N = p.ndust;
    if (gx == p.ng) {
        in_batches<R>(p.nvar, [&](int v) { return p.u_init[uidx(p, v, gy, gx)]; }, [&](int v, R val) { u[uidx(p, v, gy, gx)] = val; });
        return true;
    }
    const double trel = p.treld[gx];
    if (!(trel > 0.0)) return false;
    const C e = C(exp(-dt / trel));
    constexpr int CH = 4;   // species whose loads are in flight together
    for (int s0 = 0; s0 <= N; s0 += CH) {
        R q[CH][6];
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            if (s0 + i > N) break;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const long long e = uidx(p, svar(s0 + i, c, N), gy, gx);
                q[i][c] = p.u_init[e];
                q[i][3 + c] = u[e];
            }
        }
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const int s = s0 + i;
            if (s > N) break;
            const C rho_init = C(q[i][0]), rho_old = C(q[i][3]);
            const Over<C> by_init(rho_init), by_old(rho_old);
            const C vx_init = by_init(C(q[i][1])), vy_init = by_init(C(q[i][2]));
            const C vx_old = by_old(C(q[i][4])), vy_old = by_old(C(q[i][5]));
            const C rho_new = (rho_init) * (C(1) - e) + rho_old * e;
            const C vx_new = (vx_init) * (C(1) - e) + vx_old * e;
            const C vy_new = (vy_init) * (C(1) - e) + vy_old * e;
            u[uidx(p, svar(s, 0, N), gy, gx)] = R(rho_new);
            u[uidx(p, svar(s, 1, N), gy, gx)] = R(rho_new * vx_new);
            u[uidx(p, svar(s, 2, N), gy, gx)] = R(rho_new * vy_new);
        }
    }
    return true;
}

// setup_inloop of the Cartesian disk (disk/setup.f90) for one active cell: a buffer cell takes
// the state the host tabulated with the routine's operations (its relaxation rate is 0).
// Returns true when it changed the cell.
template <typename R>
__device__ __forceinline__ bool cdisk_inloop_cell(const KParams<R>& p, R* u, int gx, int gy) {
    const long long e = (long long)gy * p.pitch + gx, pl = p.plane;
    const double rho_ana = p.ctgt[e];
    if (!(rho_ana > 0.0)) return false;
    const int N = p.ndust;
    u[uidx(p, 0, gy, gx)] = R(rho_ana);
    u[uidx(p, 1, gy, gx)] = R(p.ctgt[pl + e]);
    u[uidx(p, 2, gy, gx)] = R(p.ctgt[2 * pl + e]);
    u[uidx(p, 4, gy, gx)] = R(p.ctgt[3 * pl + e]);
    const R rd = R(p.ctgt[4 * pl + e]), mx = R(p.ctgt[5 * pl + e]), my = R(p.ctgt[6 * pl + e]);
    for (int k = 0; k < N; ++k) {
        u[uidx(p, 5 + k, gy, gx)] = rd;
        u[uidx(p, 5 + N + k, gy, gx)] = mx;
        u[uidx(p, 5 + 2 * N + k, gy, gx)] = my;
    }
    return true;
}

// dust_growth of one active cell of K2 (growth.cuh); u holds the post-drag state.  Returns the
// status bits it raises.
template <typename R>
__device__ __noinline__ unsigned grow_in_finalize(const KParams<R>& p, R* u, int gx, int gy, double dt) {
    const int N = p.ndust;
    double rd[GROWTH_MAX_DUST], ts[GROWTH_MAX_DUST], vx[GROWTH_MAX_DUST], vy[GROWTH_MAX_DUST], vz[GROWTH_MAX_DUST];
    double gam[GROWTH_MAX_DUST];
    const double rho_old = (double)p.u_cur[uidx(p, 0, gy, gx)];
    const double qrho_old = rho_old > p.smallr ? rho_old : p.smallr;
    const bool ambi = (p.gw.mode & SHARK_GROWTH_AMBIPOLAR) && p.chg_gamma_d;
    const long long c = (long long)gy * p.pitch + gx;
    const TStop<R> tstop(p, qrho_old, gx, gy);
    for (int k = 0; k < N; ++k) {
        rd[k] = (double)u[uidx(p, 5 + k, gy, gx)];
        ts[k] = tstop(k);
        const double r0 = (double)p.u_cur[uidx(p, 5 + k, gy, gx)];
        vx[k] = (double)p.u_cur[uidx(p, 5 + N + k, gy, gx)] / r0;
        vy[k] = (double)p.u_cur[uidx(p, 5 + 2 * N + k, gy, gx)] / r0;
        vz[k] = (double)p.u_cur[uidx(p, 5 + 3 * N + k, gy, gx)] / r0;
        gam[k] = ambi ? (double)p.chg_gamma_d[(long long)k * p.plane + c] : 0.0;
    }
    const double eta_a = ambi ? (double)p.chg_eta[2 * p.plane + c] : 0.0;
    const double hs = p.setup == SHARK_SETUP_DISK_POLAR ? p.hsd[gx] : 1.0;
    const double rho_gas = (double)u[uidx(p, 0, gy, gx)];
    bool ok;
    if constexpr (sizeof(R) == 4)
        ok = growth_cell_f(p.gw, N, gx, dt, (float)rho_gas, (float)qrho_old, (float)hs, rd, ts, vx, vy, vz,
                           ambi ? gam : nullptr, (float)eta_a);
    else
        ok = growth_cell_d(p.gw, N, gx, dt, rho_gas, qrho_old, hs, rd, ts, vx, vy, vz, ambi ? gam : nullptr, eta_a);
    for (int k = 0; k < N; ++k) u[uidx(p, 5 + k, gy, gx)] = R(rd[k]);
    return ok ? 0u : (unsigned)SHARK_STATUS_GROWTH;
}

// Dust growth of the mixed path without fragmentation (dust_growth.f90:3-256) on the post-drag state
// u_next, one warp per cell, a lane per bin.  Most cells take a single sub-step (on average 1.0-2.3
// on the disk and the driven box), so a cell costs its setup: the relative velocities of its
// N (N + 1)/2 pairs.  A warp takes chunks of 4 cells of a row:
//  1. its lanes read the chunk's densities and momenta, 8 bins x 4 cells at a time, and leave the
//     species' terms of the cells in shared memory (velocities, stopping times, t/t_L);
//  2. two cells at a time (the pair's indices, factors and addresses serve both), the lanes form the
//     rate factors pK dv / hs of pairs q = lane, lane + 32, ... from those terms, only the turbulent
//     case that applies, and the rates of the first sub-step with them; lane b gathers drho_b/dt =
//     sum_t gc[t][b] w[gq[t][b]] from the host-built table of net transfers (in shared memory as
//     four rows' coefficients per 128-bit entry and two rows' pair indices, 16 bits each, per 32-bit
//     word; four partial sums of rows t mod 4, both cells in one packed FMA); the sub-step is the
//     warp minimum of CFL_growth rho_b/|drho_b/dt| (one redux.sync on the candidates' bit patterns),
//     and the part of dt still to integrate is kept as an FP32 fraction (the last sub-step takes all
//     of it).  A cell that needs more sub-steps goes on by itself;
//  3. the cells' densities are written back together.
// Bound by instruction issue (74 % of the slots at 32 species, 76 % at 16).  The loops over pairs are not unrolled: unrolled
// they overflowed the instruction cache (the largest stall).  As a phase of K2 with each cell's
// inputs read by lane = bin and every turbulent case formed for every pair, K2 took 2.09 ms on the
// disk 512 x 1024 x 16 and 5.20 ms on the driven box 768^2 x 32; unrolled per-cell warps 1.06 and
// 3.98 ms, not unrolled 0.99 and 2.72 ms, two cells at a time 0.90 and 2.57 ms; bit for bit the same.
constexpr int GROWTH_PAIR_SLOTS = (GROWTH_MAX_PAIRS + 31) / 32;
// cells of a chunk, warps of a block: two blocks fill an SM's shared memory at 32 species
constexpr int GROWTH_F_CELLS = 4, GROWTH_F_WARPS = 12;
constexpr int GROWTH_SMEM_ROWS = 80;        // gather rows staged in shared memory (64 at 32 species)

// bins a cell's terms are laid out for
__host__ __device__ constexpr int growth_f_bins(int N) { return N <= 16 ? 16 : 32; }

// shared memory of a block in bytes: the tables, then per warp the species' terms of a chunk's cells,
// their constants and two cells' pair rates
struct GrowthSmemF {
    int gc, gi, pair, pk, warp0, per_warp, total;
    __host__ __device__ GrowthSmemF(int N, int P, int L) {
        const int rows = L <= GROWTH_SMEM_ROWS ? (L + 3) & ~3 : 0, slots = (P + 31) / 32 * 32;
        gc = 0;
        gi = gc + rows * 32 * 4;
        pk = gi + rows / 2 * 32 * 4;   // multiples of 256 bytes so far
        pair = pk + slots * 8;
        warp0 = (pair + slots * 4 + 15) & ~15;
        per_warp = ((GROWTH_F_CELLS * growth_f_bins(N) * (16 + 8 + 4) + GROWTH_F_CELLS * 16 * 2 + slots * 8) + 15) & ~15;
        total = warp0 + GROWTH_F_WARPS * per_warp;
    }
};

// SLOTS: the most pairs per lane, 5 up to 16 bins.
template <int SLOTS>
static __global__ void __launch_bounds__(32 * GROWTH_F_WARPS, 2) k_growth_f(KParams<float> p) {
    extern __shared__ __align__(16) unsigned char sgf[];
    const GrowthDev& g = p.gw;
    const int N = p.ndust, P = g.npair, L = g.gL;
    const GrowthSmemF off(N, P, L);
    // gather table: coefficient of row t, lane l at sgc[128 (t >> 2) + 4 l + (t & 3)]; pair
    // indices of rows 4 u + 2 h, 4 u + 2 h + 1 (low, high 16 bits) at sgi[64 u + 2 l + h]
    float* sgc = reinterpret_cast<float*>(sgf + off.gc);
    unsigned* sgi = reinterpret_cast<unsigned*>(sgf + off.gi);
    float2* spk = reinterpret_cast<float2*>(sgf + off.pk);         // rate factor (halved for k == j), Brownian factor
    unsigned* spair = reinterpret_cast<unsigned*>(sgf + off.pair);   // k << 16 | j
    const int slots = (P + 31) / 32;
    const bool staged = L <= GROWTH_SMEM_ROWS;
    if (staged) {   // rows past L are zero (coefficient 0, pair 0)
        const int L4 = (L + 3) & ~3;
        for (int e = threadIdx.x; e < L4 * 32; e += blockDim.x) {
            const int t = e >> 5, l = e & 31;
            sgc[128 * (t >> 2) + 4 * l + (t & 3)] = t < L ? __ldg(g.gc + e) : 0.f;
        }
        for (int e = threadIdx.x; e < L4 / 2 * 32; e += blockDim.x) {
            const int r = e >> 5, l = e & 31, t0 = 2 * r;   // rows t0, t0 + 1 of lane l
            const unsigned i0 = t0 < L ? (unsigned)__ldg(g.gq + t0 * 32 + l) : 0u;
            const unsigned i1 = t0 + 1 < L ? (unsigned)__ldg(g.gq + (t0 + 1) * 32 + l) : 0u;
            sgi[64 * (t0 >> 2) + 2 * l + ((t0 >> 1) & 1)] = i0 | (i1 << 16);
        }
    }
    for (int e = threadIdx.x; e < (P + 31) / 32 * 32; e += blockDim.x) {
        const int pr = e < P ? __ldg(g.pair + e) : 0, k = pr >> 8, j = pr & 255;
        spair[e] = (unsigned)k << 16 | (unsigned)j;
        spk[e] = e < P ? make_float2(__ldg(g.pKf + e) * (k == j ? 0.5f : 1.f), __ldg(g.pBf + e)) : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned char* mine = sgf + off.warp0 + wid * off.per_warp;
    constexpr int NB = SLOTS > 5 ? 32 : 16;
    float4* sv = reinterpret_cast<float4*>(mine);                                   // [cells][NB] vx, vy, vz, |G|
    float4* sc = reinterpret_cast<float4*>(mine + GROWTH_F_CELLS * NB * 16);        // [cells][2] the cells' constants
    float2* sts = reinterpret_cast<float2*>(mine + GROWTH_F_CELLS * (NB + 2) * 16); // [cells][NB] stopping time, t/t_L
    float* srd = reinterpret_cast<float*>(sts + GROWTH_F_CELLS * NB);               // [cells][NB] densities
    float2* w = reinterpret_cast<float2*>(srd + GROWTH_F_CELLS * NB);               // pair rates of two cells
    float* u = p.u_next;
    const float* __restrict__ uc = p.u_cur;
    const int pl = (int)p.plane;
    const unsigned FULL = 0xffffffffu;
    const double dt = *p.dt;
    const bool ambi = (g.mode & SHARK_GROWTH_AMBIPOLAR) && p.chg_gamma_d;
    const bool disk = p.setup == SHARK_SETUP_DISK_POLAR;
    const bool on = lane < N;
    const int b = on ? lane : 0;
    const bool thr_on = g.kernel == 0 && g.eps_thr > 0.0;
    const float dtf = (float)dt, idtf = 1.f / dtf;
    const float fctl = g.dtctl > 0.0 ? (float)(g.dtctl / dt) : 0.f, dtctl = (float)g.dtctl;
    const float stick = (float)g.sticking, cflg = (float)g.cfl;
    const float eps_thr = (float)g.eps_thr, rmin = (float)g.dust_ratio_min, smallr = (float)p.smallr;
    const GrowthRunF rf = growth_run_consts_f(g);
    const float4 row0 = growth_row_f(g, 0);        // the one temperature row (dustyTurb)
    const int nchunk_x = (p.ng + p.nx + GROWTH_F_CELLS - 1) / GROWTH_F_CELLS;   // from column 0: whole sectors
    const int nchunk = nchunk_x * (p.ndim == 2 ? p.ny : 1);
    constexpr int BINS = 32 / GROWTH_F_CELLS;      // bins read at a time
    const int c = lane % GROWTH_F_CELLS, bs = lane / GROWTH_F_CELLS;
    unsigned st = 0;
    // drho_b/dt of this lane's bin: the four partial sums of rows t mod 4, for one cell (rates at
    // we[2 q]) or both
    auto gather = [&](const float* we) -> float {
        float a[4] = {0.f, 0.f, 0.f, 0.f}, d;
        int r = 0;
        if (!staged) {
            d = 0.f;
            for (; r < L; ++r) d += __ldg(g.gc + r * 32 + lane) * we[2 * __ldg(g.gq + r * 32 + lane)];
            return d;
        }
        for (; r + 4 <= L; r += 4) {
            const float4 cg = *reinterpret_cast<const float4*>(sgc + 32 * r + 4 * lane);
            const uint2 ix = *reinterpret_cast<const uint2*>(sgi + 16 * r + 2 * lane);
            a[0] = fmaf(cg.x, we[2 * (ix.x & 0xffffu)], a[0]);
            a[1] = fmaf(cg.y, we[2 * (ix.x >> 16)], a[1]);
            a[2] = fmaf(cg.z, we[2 * (ix.y & 0xffffu)], a[2]);
            a[3] = fmaf(cg.w, we[2 * (ix.y >> 16)], a[3]);
        }
        d = a[0];
        for (; r < L; ++r) {
            const unsigned iw = sgi[64 * (r >> 2) + 2 * lane + ((r >> 1) & 1)];
            d = fmaf(sgc[128 * (r >> 2) + 4 * lane + (r & 3)], we[2 * ((r & 1) ? (iw >> 16) : (iw & 0xffffu))], d);
        }
        return (d + a[1]) + (a[2] + a[3]);
    };
    auto gather2 = [&](float& d0, float& d1) {
        if (!staged) {
            d0 = gather(reinterpret_cast<const float*>(w));
            d1 = gather(reinterpret_cast<const float*>(w) + 1);
            return;
        }
        float2 a[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) a[h] = make_float2(0.f, 0.f);
        int r = 0;
#pragma unroll 2
        for (; r + 4 <= L; r += 4) {
            const float4 cg = *reinterpret_cast<const float4*>(sgc + 32 * r + 4 * lane);
            const uint2 ix = *reinterpret_cast<const uint2*>(sgi + 16 * r + 2 * lane);
            a[0] = __ffma2_rn(make_float2(cg.x, cg.x), w[ix.x & 0xffffu], a[0]);
            a[1] = __ffma2_rn(make_float2(cg.y, cg.y), w[ix.x >> 16], a[1]);
            a[2] = __ffma2_rn(make_float2(cg.z, cg.z), w[ix.y & 0xffffu], a[2]);
            a[3] = __ffma2_rn(make_float2(cg.w, cg.w), w[ix.y >> 16], a[3]);
        }
        float2 d = a[0];
        for (; r < L; ++r) {
            const float cg = sgc[128 * (r >> 2) + 4 * lane + (r & 3)];
            const unsigned iw = sgi[64 * (r >> 2) + 2 * lane + ((r >> 1) & 1)];
            d = __ffma2_rn(make_float2(cg, cg), w[(r & 1) ? (iw >> 16) : (iw & 0xffffu)], d);
        }
        d0 = (d.x + a[1].x) + (a[2].x + a[3].x);
        d1 = (d.y + a[1].y) + (a[2].y + a[3].y);
    };
    // one sub-step of this lane's bin; rem: the part of dt still to integrate
    auto advance = [&](float d, float& rd, float& rem, float fl) {
        // non-negative floats order like their bit patterns read as unsigned integers
        const float cand0 = (on && d != 0.f) ? fmaxf(rd / fabsf(d) * cflg, 0.f) : 1e30f;
        const float cand = __uint_as_float(__reduce_min_sync(FULL, __float_as_uint(cand0)));
        const float dtg0 = fctl > 0.f ? dtctl : cand;
        const float frac = fctl > 0.f ? fctl : cand * idtf;
        float dtg;
        if (frac >= rem) { dtg = rem * dtf; rem = 0.f; }
        else { dtg = dtg0; rem = rem - frac; }
        rd = fmaxf(rd + d * dtg, fl);
    };
    for (int ch = blockIdx.x * GROWTH_F_WARPS + wid; ch < nchunk; ch += gridDim.x * GROWTH_F_WARPS) {
        const int iy = ch / nchunk_x, x0 = (ch - iy * nchunk_x) * GROWTH_F_CELLS;
        const int gy = p.ndim == 2 ? iy + p.ng : 0;
        const int first = max(p.ng - x0, 0), last = min(p.ng + p.nx - x0, GROWTH_F_CELLS);   // cells of the chunk
        {
            const int gx = x0 + min(max(c, first), last - 1), cc = gy * p.pitch + gx;
            const float rho_old = uc[cc];
            const float qrho_old = rho_old > smallr ? rho_old : smallr;
            const float rho_gas = u[cc];
            // stopping times for the pair velocities (FP32): t_k = C_k / F_cell with the tabulated 1/C_k
            // (dustyTurb F = c_s rho, polar disk F = rho/hs c_s: the setups with growth)
            const float F = p.setup == SHARK_SETUP_DUSTYTURB ? p.cs[gx] * qrho_old : qrho_old / (float)p.hsd[gx] * p.cs[gx];
            const float hs = disk ? (float)p.hsd[gx] : 1.f;
            const float eta_a = ambi ? p.chg_eta[2 * p.plane + cc] : 0.f;
            const GrowthCellF cf = growth_cell_consts_f(g, rf, g.t_per_col ? growth_row_f(g, gx) : row0, qrho_old, hs, eta_a);
            if (bs == 0) {
                sc[2 * c] = make_float4(cf.T, cf.cs_v, cf.t_L, cf.t_eta);
                sc[2 * c + 1] = make_float4(cf.rm, cf.vambi, hs, rho_gas);
            }
#pragma unroll 4
            for (int b0 = 0; b0 < N; b0 += BINS) {
                const int k = b0 + bs;
                if (k >= N) continue;
                const float ts = 1.f / (p.dinvts_f[k] * F);
                const float r0 = uc[cc + (5 + k) * pl];
                const float vx = uc[cc + (5 + N + k) * pl] / r0;
                const float vy = uc[cc + (5 + 2 * N + k) * pl] / r0;
                const float vz = uc[cc + (5 + 3 * N + k) * pl] / r0;
                float gm = 0.f;
                if (ambi) {
                    const float ga = p.chg_gamma_d[(long long)k * p.plane + cc];
                    gm = fabsf(ga) * rsqrtf(1.f + ga * ga);
                }
                sv[c * NB + k] = make_float4(vx, vy, vz, gm);
                sts[c * NB + k] = make_float2(ts, ts / cf.t_L);
                srd[c * NB + k] = u[cc + (5 + k) * pl];
            }
        }
        __syncwarp();
        for (int i = first & ~1; i < last; i += 2) {   // two cells at a time (one of them may lie outside)
            const float4 *v0 = sv + i * NB, *v1 = v0 + NB;
            const float2 *t0 = sts + i * NB, *t1 = t0 + NB;
            GrowthCellF cf[2];
            float ihs[2], fl[2], thr[2], rd[2], rdt[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float4 c0 = sc[2 * (i + e)], c1 = sc[2 * (i + e) + 1];
                cf[e] = GrowthCellF{c0.x, c0.y, c0.z, c0.w, c1.x, c1.y};
                ihs[e] = 1.f / c1.z;
                fl[e] = c1.w * rmin;
                thr[e] = thr_on ? eps_thr * c1.w : -1.f;
                rd[e] = srd[(i + e) * NB + b];
                rdt[e] = rd[e] < thr[e] ? 0.f : rd[e];   // a bin below the threshold takes no part
            }
            float kp0[SLOTS], kp1[SLOTS];
#pragma unroll 1
            for (int s = 0; s < slots; ++s) {
                const int q = lane + 32 * s;
                const unsigned pr = spair[q];
                const int k = pr >> 16, j = pr & 0xffffu;
                const float2 pk = spk[q];
                float d0 = 1.f, d1 = 1.f;
                if (g.kernel == 0) {
                    const float2 tk = t0[k], tj = t0[j];
                    const float4 vk = v0[k], vj = v0[j];
                    d0 = growth_dv_f(g, rf, cf[0], tk.x, tj.x, tk.y, tj.y, pk.y, vk.x - vj.x, vk.y - vj.y, vk.z - vj.z, vk.w - vj.w, ambi);
                    const float2 uk = t1[k], uj = t1[j];
                    const float4 wk = v1[k], wj = v1[j];
                    d1 = growth_dv_f(g, rf, cf[1], uk.x, uj.x, uk.y, uj.y, pk.y, wk.x - wj.x, wk.y - wj.y, wk.z - wj.z, wk.w - wj.w, ambi);
                }
                kp0[s] = d0 = pk.x * d0 * ihs[0];
                kp1[s] = d1 = pk.x * d1 * ihs[1];
                w[q] = make_float2(d0 * __shfl_sync(FULL, rdt[0], k) * __shfl_sync(FULL, rdt[0], j) * stick,
                                   d1 * __shfl_sync(FULL, rdt[1], k) * __shfl_sync(FULL, rdt[1], j) * stick);
            }
            __syncwarp();
            // the first sub-step of both
            float d[2];
            gather2(d[0], d[1]);
            float rem[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) { rem[e] = 1.f; advance(d[e], rd[e], rem[e], fl[e]); }
            // the cells that need more, by themselves
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float* kp = e ? kp1 : kp0;
                float* we = reinterpret_cast<float*>(w) + e;
                for (int niter = 1; rem[e] > 0.f && niter < grw::MAX_SUB; ++niter) {
                    rdt[e] = rd[e] < thr[e] ? 0.f : rd[e];
                    __syncwarp();                                   // the rates are read; the next ones may take their place
#pragma unroll 1
                    for (int s = 0; s < slots; ++s) {
                        const int q = lane + 32 * s;
                        const unsigned pr = spair[q];
                        we[2 * q] = kp[s] * __shfl_sync(FULL, rdt[e], pr >> 16) * __shfl_sync(FULL, rdt[e], pr & 0xffffu) * stick;
                    }
                    __syncwarp();
                    advance(gather(we), rd[e], rem[e], fl[e]);
                }
                if (on) srd[(i + e) * NB + b] = rd[e];
                if (rem[e] > 0.f && i + e >= first && i + e < last) st |= (unsigned)SHARK_STATUS_GROWTH;
            }
            __syncwarp();
        }
        if (c >= first && c < last) {
            const int cc = gy * p.pitch + x0 + c;
            for (int k = bs; k < N; k += BINS) u[cc + (5 + k) * pl] = srd[c * NB + k];
        }
        __syncwarp();
    }
    if (st && lane == 0) atomicOr(p.status, st);
}

// Dust growth of the FP64 path without fragmentation (dust_growth.f90:3-256) on the post-drag state
// u_next: G = growth_lanes(N) lanes per cell, blocks of 128 threads.  Bit for bit the oracle's
// sub-cycle: a sub-step's pair rates dn/dt are formed in the oracle's order of operations, the lanes
// taking the pairs in turn, and exchanged through shared memory; then each lane sums its bins' mass
// changes in the oracle's order, one list of (coefficient, pair) per bin.  What the sub-step does
// not change is formed once per cell (the rate's factor A dv) or on the host (the coefficients).
// The kernel is bound by the FP64 pipe: some 11 instructions for a pair's rate (its divisions by the
// two masses share the masses' reciprocals) and two for each entry, against 80 for a pair in a
// thread per cell; several lanes a cell spread the small grids over the chip and leave few cells that
// wait for each other's sub-steps.  K2 with growth, in ms against a thread per cell: polar disk
// 128 x 256 x 16 26.9 -> 3.2, 48 x 64 x 16 38.6 -> 1.4; dusty box 48^2 x 32 97 -> 3.4, 256^2 x 32 39 -> 12.5.
constexpr int GROWTH_D_THREADS = 128;

// doubles of shared memory per cell: densities, then the species' terms, reused by the pair rates;
// a stride of 8 modulo 16 puts the cells of a warp in different banks
__host__ __device__ __forceinline__ int growth_d_stride(int N, int P) {
    const int n = N + (P > 8 * N ? P : 8 * N);
    return n + ((8 - n % 16) + 16) % 16;
}

template <int GL>
static __global__ void __launch_bounds__(GROWTH_D_THREADS) k_growth_d(KParams<double> p) {
    extern __shared__ __align__(16) double sgrow[];
    __shared__ double smk[GROWTH_MAX_DUST], symk[GROWTH_MAX_DUST];
    const GrowthDev& g = p.gw;
    const int N = p.ndust, P = g.npair;
    if (threadIdx.x < N) {
        smk[threadIdx.x] = g.mk[threadIdx.x];
        symk[threadIdx.x] = rcp64(g.mk[threadIdx.x]);
    }
    __syncthreads();
    constexpr int SLOTS = GL == 8 ? 1 : GROWTH_SLOTS;
    const int l = threadIdx.x % GL, grp = threadIdx.x / GL;
    const long long nact = (long long)p.nx * (p.ndim == 2 ? p.ny : 1);
    const long long cell = blockIdx.x * (long long)(GROWTH_D_THREADS / GL) + grp;
    const bool act = cell < nact;
    // a group past the grid's end takes the last cell along and writes nothing
    const long long ac = act ? cell : nact - 1;
    const int gx = (int)(ac % p.nx) + p.ng, gy = p.ndim == 2 ? (int)(ac / p.nx) + p.ng : 0;
    const unsigned mask = (0xffffffffu >> (32 - GL)) << (threadIdx.x & 31 & ~(GL - 1));
    double* rd = sgrow + (size_t)grp * growth_d_stride(N, P);
    double* w = rd + N;                       // pair rates
    double *ts = w, *S = w + N, *W = w + 2 * N, *I = w + 3 * N, *vx = w + 4 * N, *vy = w + 5 * N, *vz = w + 6 * N, *G = w + 7 * N;
    double* u = p.u_next;
    const double dt = *p.dt;
    const bool ambi = (g.mode & SHARK_GROWTH_AMBIPOLAR) && p.chg_gamma_d;
    const long long e = (long long)gy * p.pitch + gx;
    const double rho_old = p.u_cur[e], qrho_old = max64_pos(rho_old, p.smallr);
    const double hs = p.setup == SHARK_SETUP_DISK_POLAR ? p.hsd[gx] : 1.0, yhs = rcp64(hs);
    const double rho_gas = u[e];
    const GrowthCellD c = growth_cell_consts_d(g, gx, qrho_old, hs, ambi ? p.chg_eta[2 * p.plane + e] : 0.0);
    // the species' terms
    const TStop<double> tstop(p, qrho_old, gx, gy);
    const Over<double> by_tL(c.t_L);
    for (int k = l; k < N; k += GL) {
        rd[k] = u[(5 + k) * p.plane + e];
        const double t = tstop(k), St = by_tL(t);
        ts[k] = t;
        S[k] = St;
        W[k] = Over<double>(St + c.rm)(St * St);
        I[k] = Over<double>(1.0 + St)(1.0);
        const double r0 = p.u_cur[(5 + k) * p.plane + e], y = rcp64(r0);
        vx[k] = div64(p.u_cur[(5 + N + k) * p.plane + e], r0, y);
        vy[k] = div64(p.u_cur[(5 + 2 * N + k) * p.plane + e], r0, y);
        vz[k] = div64(p.u_cur[(5 + 3 * N + k) * p.plane + e], r0, y);
        const double gm = ambi ? p.chg_gamma_d[(long long)k * p.plane + e] : 0.0;
        G[k] = abs64(gm) / sqrt(1.0 + gm * gm);
    }
    __syncwarp(mask);
    // A dv of this lane's pairs (the rate's first factor that a sub-step keeps)
    double ka[(GL == 8 ? 36 : GROWTH_MAX_PAIRS) / GL + 1];
    const double cB = 8.0 * grw::kB * c.T / grw::pi, yuv2 = rcp64(g.uv2);
    for (int i = 0, q = l; q < P; ++i, q += GL) {
        const int pr = g.pair[q], k = pr >> 8, j = pr & 255, kj = k * N + j;
        double a = 1.0;
        if (g.kernel == 0) {
            const double pD = g.pD[kj], X = div64_const(div64_const(cB * g.pS[kj], pD, rcp64(pD)), g.uv2, yuv2);
            a = g.pA[kj] * growth_dv_pair_d(g, c, ts[k], ts[j], S[k], S[j], W[k], W[j], I[k], I[j], X, vx[k] - vx[j],
                                            vy[k] - vy[j], vz[k] - vz[j], G[k] - G[j], ambi);
        } else if (g.kernel == 2) {
            a = smk[k] + smk[j];
        }
        ka[i] = a;
    }
    __syncwarp(mask);                         // the terms are read; the rates may take their place
    const double thr = g.eps_thr * rho_gas, fl = rho_gas * g.dust_ratio_min;
    const bool thr_on = g.kernel == 0 && g.eps_thr > 0.0, hs_on = hs != 1.0, stick_on = g.sticking != 1.0;
    int bin[SLOTS];
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) bin[s] = g.sbin[s * GL + l];
    double time = 0.0;
    int niter = 0;
    while (is_less(time, dt) && niter < grw::MAX_SUB) {
        niter = niter + 1;
        for (int i = 0, q = l; q < P; ++i, q += GL) {
            const int pr = g.pair[q], k = pr >> 8, j = pr & 255;
            const double rk = rd[k], rj = rd[j];
            double d = (g.kernel == 1 ? rk : ka[i] * rk) * rj;
            d = div64_const(div64_const(d, smk[k], symk[k]), smk[j], symk[j]);
            if (hs_on) d = div64_const(d, hs, yhs);
            if (k == j) d = 0.5 * d;
            if (thr_on && (is_less(rk, thr) || is_less(rj, thr))) d = 0.0;
            w[q] = d;
        }
        __syncwarp(mask);
        double dr[SLOTS], cand = 1e32;
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
            dr[s] = 0.0;
            if (s * GL >= N) continue;
            double d = 0.0;
            if (!stick_on) {
                for (int t = g.sbase[s]; t < g.sbase[s + 1]; ++t)
                    d = d + __ldg(g.sc + t * GL + l) * w[__ldg(g.sq + t * GL + l)];
            } else {
                for (int t = g.sbase[s]; t < g.sbase[s + 1]; ++t)
                    d = d + __ldg(g.sc + t * GL + l) * w[__ldg(g.sq + t * GL + l)] * g.sticking;
            }
            dr[s] = d;
            const int b = bin[s];
            if (b >= 0 && !is_zero(d)) {
                const double a = abs64(d), x = div64(rd[b], a, rcp64(a)) * g.cfl;
                // positive numbers order as their bits, a result that is none never is the least
                cand = abs_bits(x) < abs_bits(cand) ? x : cand;
            }
        }
#pragma unroll
        for (int o = GL / 2; o > 0; o >>= 1) {
            const double x = __shfl_xor_sync(mask, cand, o);
            cand = abs_bits(x) < abs_bits(cand) ? x : cand;
        }
        const double rest = dt - time;
        double dtg = is_less(cand, rest) ? cand : rest;
        if (g.dtctl > 0.0) dtg = g.dtctl < rest ? g.dtctl : rest;
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
            if (s * GL >= N) continue;
            if (bin[s] >= 0) rd[bin[s]] = max64_pos(rd[bin[s]] + dr[s] * dtg, fl);
        }
        time = time + dtg;
        __syncwarp(mask);
    }
    if (!act) return;
    for (int k = l; k < N; k += GL) u[(5 + k) * p.plane + e] = rd[k];
    if (l == 0 && is_less(time, dt)) atomicOr(p.status, (unsigned)SHARK_STATUS_GROWTH);
}

// Driven-turbulence kick of the dustyTurb box (turb.f90:227-324 in 2D): the gas momentum gains
// rho a dt with the solenoidal Ornstein-Uhlenbeck acceleration of this step at the cell centre.
// C = double follows the oracle's operations; C = float is the mixed-precision form, whose mode
// table k_ou_update leaves in floats (converted by every cell, it was 70 instructions of the FP64
// pipe for 14 modes, three times the sines' time).
template <typename C, typename R>
__device__ __forceinline__ void turb_kick_cell(const KParams<R>& p, R* u, int gx, int gy, double dt) {
    const C x = C(p.xposd[gx]);
    const C y = C(Over<double, CONSTANT>((double)(float)p.ny)(((double)(float)(gy - p.ng) + 0.5) * p.box_l_y));
    C ax = C(0), ay = C(0);
    for (int m = 0; m < p.ou_nm; ++m) {
        if constexpr (sizeof(C) == 8) {
            const C kxp = p.ou_modes[3 * m], kyp = p.ou_modes[3 * m + 1], kk = p.ou_modes[3 * m + 2];
            C sn, cs;
            sincos(kxp * x + kyp * y, &sn, &cs);
            const C w = p.ou[2 * m] * cs + p.ou[2 * m + 1] * sn;
            ax = ax + kyp / kk * w;
            ay = ay - kxp / kk * w;
        } else {
            const float4 k = reinterpret_cast<const float4*>(p.ou_f)[m];
            const float2 c = reinterpret_cast<const float2*>(p.ou_f + 4 * p.ou_nm)[m];
            C sn, cs;
            sincosf(k.x * x + k.y * y, &sn, &cs);
            const C w = c.x * cs + c.y * sn;
            ax = ax + k.z * w;
            ay = ay - k.w * w;
        }
    }
    const C rho = C(u[uidx(p, 0, gy, gx)]);
    u[uidx(p, 1, gy, gx)] = R(C(u[uidx(p, 1, gy, gx)]) + rho * ax * C(dt));
    u[uidx(p, 2, gy, gx)] = R(C(u[uidx(p, 2, gy, gx)]) + rho * ay * C(dt));
}

// dust_drag(1.0) (src/dust/dust_drag.f90:2-75) of a cell, FP64 arithmetic; the stopping times are those of
// the state at the start of the step (compute_tstop runs before the update in solve.f90:34-35).
// CONST_TS: constant stopping times (SI box) take the step's coefficients from k_prepare_step (SI 256^2 x 8:
// K2 0.102 -> 0.088 ms).  WHERE = TRIED: false, and nothing stored, where a denominator lies outside
// div64_const's range.
template <typename R, int NS, bool CONST_TS, int WHERE>
__device__ __forceinline__ bool drag_cell_d(const KParams<R>& p, R* u, const TStop<R, WHERE>& tstop, int gx, int gy, double dt,
                                            double rho, double& px, double& py, double& pz) {
    constexpr int NMAX = NS > 0 ? NS : 1;
    const int N = NS >= 0 ? NS : p.ndust;
    bool inside = tstop.inside();
    const double* cd = reinterpret_cast<const double*>(p.coef + SHARK_COEF_D);
    double alpha[NMAX];
    double rhon = rho, pnx = px, pny = py, pnz = pz;
    for (int k = 0; k < N; ++k) {
        double w;
        if constexpr (CONST_TS) w = cd[k];
        else {
            const Over<double, WHERE> by_ts(tstop(k));
            const double a = by_ts(dt);
            const Over<double, WHERE> by_a(1.0 + a);
            w = by_a(a);
            inside = inside && by_ts.inside() && by_a.inside();
            if (NS > 0) alpha[k < NMAX ? k : 0] = a;
        }
        pnx = pnx + w * (double)u[uidx(p, 5 + N + k, gy, gx)];
        pny = pny + w * (double)u[uidx(p, 5 + 2 * N + k, gy, gx)];
        pnz = pnz + w * (double)u[uidx(p, 5 + 3 * N + k, gy, gx)];
        rhon = rhon + w * (double)u[uidx(p, 5 + k, gy, gx)];
    }
    const Over<double, WHERE> by_rhon(rhon);
    if (WHERE == TRIED) {
        if constexpr (CONST_TS)
            for (int k = 0; k < N; ++k) inside = inside && is_plain(cd[2 * SHARK_MAX_DUST + k]);
        if (!inside || !by_rhon.inside()) return false;
    }
    const double fl = rho * p.dust_ratio_min;   // regularisation floor (dust_drag.f90:63-73)
    constexpr int CH = 4;   // species whose loads are in flight together
#pragma unroll
    for (int k0 = 0; k0 < (NS > 0 ? NS : N); k0 += CH) {
        double d[CH], m[CH][3];
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            if (k0 + i >= N) break;
            d[i] = (double)u[uidx(p, 5 + k0 + i, gy, gx)];
#pragma unroll
            for (int c = 0; c < 3; ++c) m[i][c] = (double)u[uidx(p, 5 + (c + 1) * N + k0 + i, gy, gx)];
        }
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const int k = k0 + i;
            if (k >= N) break;
            double a = 0.0;
            if constexpr (!CONST_TS) {
                if (NS > 0) a = alpha[k < NMAX ? k : 0];
                else a = Over<double, WHERE>(tstop(k))(dt);    // run-time species count
            }
            const Over<double, WHERE> by_a = CONST_TS ? Over<double, WHERE>(cd[SHARK_MAX_DUST + k], cd[2 * SHARK_MAX_DUST + k])
                                                       : Over<double, WHERE>(1.0 + a);
            const double w = CONST_TS ? cd[k] : by_a(a);
            u[uidx(p, 5 + N + k, gy, gx)] = R(by_a(m[i][0]) + by_rhon(w * pnx) * d[i]);
            u[uidx(p, 5 + 2 * N + k, gy, gx)] = R(by_a(m[i][1]) + by_rhon(w * pny) * d[i]);
            u[uidx(p, 5 + 3 * N + k, gy, gx)] = R(by_a(m[i][2]) + by_rhon(w * pnz) * d[i]);
            if (is_less(d[i], fl)) u[uidx(p, 5 + k, gy, gx)] = R(fl);
        }
    }
    if (p.flags & SHARK_FLAG_BACK_REACTION) {
        px = by_rhon(pnx) * rho;
        py = by_rhon(pny) * rho;
        pz = by_rhon(pnz) * rho;
        u[uidx(p, 1, gy, gx)] = R(px);
        u[uidx(p, 2, gy, gx)] = R(py);
        u[uidx(p, 3, gy, gx)] = R(pz);
    }
    return true;
}

// courant on the final state of a cell (src/solver/courant.f90:11-124): the time step it allows and its
// status bits.  WHERE = TRIED: `inside` is false where a denominator lies outside div64_const's range.
struct CourantCell {
    double dt;
    unsigned bits;
    bool inside;
};
template <typename R, int NS, int WHERE>
__device__ __forceinline__ CourantCell courant_cell_d(const KParams<R>& p, const R* u, int gx, int gy, double rho, double px,
                                                      double py, double pz) {
    const int N = NS >= 0 ? NS : p.ndust;
    double dtc;
    unsigned bits = 0;
    const double cfl = p.cfl;
    const Over<double, WHERE> by_rho(rho);
    bool inside = by_rho.inside();
    const double vx = by_rho(px), vy = by_rho(py), vz = by_rho(pz);
    double cs;
    if (p.iso == 1) cs = p.ccsd ? p.ccsd[(long long)gy * p.pitch + gx] : p.csd[gx];
    else {
        const double qrho = max64_pos(rho, p.smallr);
        const double E = (double)u[uidx(p, 4, gy, gx)];
        const double hr = 0.5 * rho;
        const double ekin = hr * (vx * vx) + hr * (vy * vy) + hr * (vz * vz);
        const double P = max64_pos((p.gamma - 1.0) * (E - ekin), p.smallp);
        const Over<double, WHERE> by_q(qrho);
        cs = sqrt(by_q(p.gamma * P));
        inside = inside && by_q.inside();
        if (abs_bits(E) > 0x7ff0000000000000ull) bits |= SHARK_STATUS_NAN;
    }
    double dxx;
    if (p.ndim == 1) dxx = p.dx1d[gx];
    else if (p.geom == 2) dxx = min64(p.dx1d[gx], p.radcd[gx] * p.dx2d[gx]);
    else dxx = min64(p.dx1d[gx], p.dx2d[gx]);
    double vv = abs64(vx) + abs64(vy) + abs64(vz);
    double vmax = cs + vv;
    double fmax_d = 0.0;     // SI: the largest square of a force until its root is taken below
    const bool fk = (p.flags & SHARK_FLAG_FORCE_KICK) != 0;
    const bool fk_si = fk && p.setup == SHARK_SETUP_SI;
    double tide = 0.0, om2 = 0.0;
    if (fk_si) {
        const double xc = p.xposd[gx] - 0.5 * p.box_l, om = p.si_om, qsh = p.si_q;
        tide = 2.0 * qsh * (om * om) * xc;
        om2 = 2.0 * om;
        const double f1 = tide - om2 * vz - 2.0 * p.si_r0 * om * p.si_eta;
        const double f3 = om2 * vx;
        fmax_d = f1 * f1 + f3 * f3;
    } else if (fk && p.setup == SHARK_SETUP_DISK_POLAR) {
        // the same point-mass force acts on gas and every dust species
        const double g = p.fgravd[gx];
        fmax_d = sqrt(g * g);
    } else if (fk && p.setup == SHARK_SETUP_DISK_CART) {   // the star's softened force, gas and dust
        const long long e = (long long)gy * p.pitch + gx;
        const double fx = (double)p.cfx[e], fy = (double)p.cfy[e];
        fmax_d = sqrt(fx * fx + fy * fy);
    }
    for (int k = 0; k < N; ++k) {
        const double rd = (double)u[uidx(p, 5 + k, gy, gx)];
        const Over<double, WHERE> by_rd(rd);
        inside = inside && by_rd.inside();
        const double vdx = by_rd((double)u[uidx(p, 5 + N + k, gy, gx)]);
        const double vdy = by_rd((double)u[uidx(p, 5 + 2 * N + k, gy, gx)]);
        const double vdz = by_rd((double)u[uidx(p, 5 + 3 * N + k, gy, gx)]);
        vv = abs64(vdx) + abs64(vdy) + abs64(vdz);
        vmax = is_less(vv, vmax) ? vmax : vv;
        if (fk_si) {
            const double f1 = tide - om2 * vdz;
            const double f3 = om2 * vdx;
            const double fm = f1 * f1 + f3 * f3;
            fmax_d = is_less(fm, fmax_d) ? fmax_d : fm;
        }
        if (!is_pos(rd)) bits |= SHARK_STATUS_NEG_DENSITY;
        if (!is_finite(vdx) || !is_finite(vdy) || !is_finite(vdz)) bits |= SHARK_STATUS_NAN;
    }
    if (fk_si) fmax_d = sqrt(fmax_d);
    const double cd = cfl * dxx;
    // plain divisions where a wave speed may be zero or its square underflow
    const double c1 = cd / abs64(vmax);
    dtc = is_less(2e44, c1) ? 2e44 : c1;
    if (fk && !is_zero(vv)) {
        double fratio = fmax_d * dxx / (vv * vv);
        fratio = max64_pos(fratio, 1e-3);
        const Over<double, WHERE> by_f(fratio);
        inside = inside && by_f.inside();
        const double c2 = by_f(cd / vv * (sqrt(1.0 + 2.0 * cfl * fratio) - 1.0));
        dtc = is_less(dtc, c2) ? dtc : c2;
    }
    if (!is_pos(rho)) bits |= SHARK_STATUS_NEG_DENSITY;
    if (!is_finite(vx) || !is_finite(vy) || !is_finite(vz) || !is_finite(rho)) bits |= SHARK_STATUS_NAN;
    if (!is_pos(dtc) || !is_finite(dtc)) { bits |= SHARK_STATUS_DT_UNDERFLOW; dtc = 2e44; }
    return CourantCell{dtc, bits, inside};
}

// The same for a cell with a denominator outside the range: out of line, so that the kernels keep to the
// registers and the code of the other form.
template <typename R>
static __device__ __noinline__ void drag_cell_wide(const KParams<R>& p, R* u, int gx, int gy, double dt, double qrho_old, double rho,
                                                   double* m) {
    const TStop<R> tstop(p, qrho_old, gx, gy);
    if (p.setup == SHARK_SETUP_SI) drag_cell_d<R, -1, true, ANYWHERE>(p, u, tstop, gx, gy, dt, rho, m[0], m[1], m[2]);
    else drag_cell_d<R, -1, false, ANYWHERE>(p, u, tstop, gx, gy, dt, rho, m[0], m[1], m[2]);
}
template <typename R>
static __device__ __noinline__ double drag_heating_wide(const KParams<R>& p, double qrho_old, int gx, int gy, double dt) {
    bool inside;
    return drag_heating(p, TStop<R>(p, qrho_old, gx, gy), gx, gy, dt, inside);
}
template <typename R>
static __device__ __noinline__ CourantCell courant_cell_wide(const KParams<R>& p, const R* u, int gx, int gy, double rho, double px,
                                                             double py, double pz) {
    return courant_cell_d<R, -1, ANYWHERE>(p, u, gx, gy, rho, px, py, pz);
}

// Bound by the FP64 pipe (64 clocks of an SM partition for a warp's instruction): quotients share
// reciprocals, compares and finiteness checks run on the bits, one square root takes the largest of
// the force limiter's sums; all exact.  SI boxes of 8 species: 1024^2 2.36 -> 1.38 ms, 256^2 0.183 ->
// 0.088 ms; dusty wave of 2048 x 4 0.075 -> 0.026 ms.  Blocks of 128: the warps of one or two
// thousand cells then each have a partition of their own.
constexpr int K2D_THREADS = 128;

// Blocks an SM: without the bound the compiler takes up to 238 registers to overlap the quotients, and the
// fewer warps cost more (us, SI 256^2: 1 species 46 -> 32, 4 species 75 -> 57, 8 species 109 -> 89).
constexpr int k2d_blocks(int NS) { return NS == 0 ? 6 : NS == 1 || NS == 2 ? 5 : 4; }

template <typename R, int NS, int MODE, bool GROW = false>
__global__ void __launch_bounds__(K2D_THREADS, k2d_blocks(NS)) k_finalize(const __grid_constant__ KParams<R> p) {
    constexpr bool DRAG = MODE == 0 || MODE == 2, REST = MODE == 0 || MODE == 3;
    const int N = NS >= 0 ? NS : p.ndust;
    const int gx = blockIdx.x * blockDim.x + threadIdx.x + p.ng;
    const int gy = (p.ndim == 2) ? blockIdx.y + p.ng : 0;
    double dtc = 2e44;
    unsigned int st = 0;
    chain_begin();
    if (DRAG) stamp_start(p.stamps);
    if (gx < p.ng + p.nx) {
        R* u = p.u_next;
        const double dt = *p.dt;
        double rho = (double)u[uidx(p, 0, gy, gx)];
        double px = (double)u[uidx(p, 1, gy, gx)], py = (double)u[uidx(p, 2, gy, gx)], pz = (double)u[uidx(p, 3, gy, gx)];
        const bool drag = DRAG && N > 0 && (p.flags & SHARK_FLAG_DRAG);
        const bool br = (p.flags & SHARK_FLAG_BACK_REACTION) != 0;
        const bool heat = DRAG && N > 0 && br && p.iso < 1;
        if (drag || heat) {
            // stopping times from the state at the start of the step (compute_tstop runs before the
            // update in solve.f90:34-35)
            const double rho_old = (double)p.u_cur[uidx(p, 0, gy, gx)];
            const double qrho_old = max64_pos(rho_old, p.smallr);
            const TStop<R, TRIED> tstop(p, qrho_old, gx, gy);
            if (drag) {
                bool done;
                if (p.setup == SHARK_SETUP_SI) done = drag_cell_d<R, NS, true, TRIED>(p, u, tstop, gx, gy, dt, rho, px, py, pz);
                else done = drag_cell_d<R, NS, false, TRIED>(p, u, tstop, gx, gy, dt, rho, px, py, pz);
                if (!done) {
                    double m[3] = {px, py, pz};
                    drag_cell_wide(p, u, gx, gy, dt, qrho_old, rho, m);
                    px = m[0]; py = m[1]; pz = m[2];
                }
            }
            if (heat) {   // drag heating, part of S_U (source_terms.f90:88-97)
                const long long ie = uidx(p, 4, gy, gx);
                bool inside = true;
                double gain = drag_heating(p, tstop, gx, gy, dt, inside);
                if (!inside) gain = drag_heating_wide(p, qrho_old, gx, gy, dt);
                u[ie] = R((double)u[ie] + gain);
            }
        }
        if (GROW && MODE == 0) st |= grow_in_finalize(p, u, gx, gy, dt);   // dust_growth (solve.f90:113)
        if (REST && p.ou_nm > 0) {                                         // turbulence kick (solve.f90:129-146)
            turb_kick_cell<double>(p, u, gx, gy, dt);
            px = (double)u[uidx(p, 1, gy, gx)];
            py = (double)u[uidx(p, 2, gy, gx)];
        }
        if (REST && p.setup == SHARK_SETUP_SI && !(p.flags & SHARK_FLAG_FORCE_KICK)) {
            // setup_inloop: Crank-Nicolson rotation (SI/setup.f90:299-332)
            const double om = p.si_om, qsh = p.si_q;
            const double Ohmdt = om * dt;
            const double xc = p.xposd[gx] - 0.5 * p.box_l;
            const Over<double> by_rot(1. + Ohmdt * Ohmdt);
            double AA = 2.0 * qsh * om * xc - 2.0 * p.si_r0 * p.si_eta;
            {
                const Over<double> by_rho(rho);
                const double uz = by_rho(pz), vx = by_rho(px), d = rho;
                pz = by_rot(d * (uz * (1. - Ohmdt * Ohmdt) + 2. * vx * Ohmdt + AA * (Ohmdt * Ohmdt)));
                px = by_rot(d * (vx * (1. - Ohmdt * Ohmdt) - 2. * uz * Ohmdt + AA * Ohmdt));
                u[uidx(p, 3, gy, gx)] = R(pz);
                u[uidx(p, 1, gy, gx)] = R(px);
            }
            AA = 2.0 * qsh * om * xc;
            for (int k = 0; k < N; ++k) {
                const long long iz = uidx(p, 5 + 3 * N + k, gy, gx), ixx = uidx(p, 5 + N + k, gy, gx);
                const double d = (double)u[uidx(p, 5 + k, gy, gx)];
                const Over<double> by_d(d);
                const double uz = by_d((double)u[iz]), vx = by_d((double)u[ixx]);
                u[iz] = R(by_rot(d * (uz * (1. - Ohmdt * Ohmdt) + 2. * vx * Ohmdt + AA * (Ohmdt * Ohmdt))));
                u[ixx] = R(by_rot(d * (vx * (1. - Ohmdt * Ohmdt) - 2. * uz * Ohmdt + AA * Ohmdt)));
            }
        }
        if (REST && ((p.setup == SHARK_SETUP_DISK_POLAR && disk_inloop_cell<R, double>(p, u, gx, gy, dt)) ||
                     (p.setup == SHARK_SETUP_DISK_CART && cdisk_inloop_cell<R>(p, u, gx, gy)))) {
            rho = (double)u[uidx(p, 0, gy, gx)];
            px = (double)u[uidx(p, 1, gy, gx)];
            py = (double)u[uidx(p, 2, gy, gx)];
            pz = (double)u[uidx(p, 3, gy, gx)];
        }
        if (MODE == 2) return;   // k_growth_d and MODE 3 follow
        CourantCell c = courant_cell_d<R, NS, TRIED>(p, u, gx, gy, rho, px, py, pz);
        if (!c.inside) c = courant_cell_wide(p, u, gx, gy, rho, px, py, pz);
        dtc = c.dt;
        st |= c.bits;
    }
    if (MODE == 2) return;
    block_reduce_dt(dtc, st, p.dt_next, p.status);
    if (REST) fill_ghost_images(p, p.u_next, gx, gy);
    if (REST) stamp_end(p.stamps);
}

// ---------------------------------------------------------------------------------------------
// K2, mixed precision (FP32 state).  The stiff part of the implicit drag -- the coefficients
// 1/(1+a_k) and a_k/(1+a_k) with a_k = dt/t_k, which carry the t_stop << dt limit -- is computed in
// FP64 (once per block when t_k is a per-species constant, as in the SI box; per cell otherwise).
// The per-cell barycentric combination (positive weights, no cancellation) and the CFL candidate
// run in FP32 like the rest of the mixed path.  Same algorithm as dust_drag.f90:29-73.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void drag_coeffs(double a, float& r, float& w) {
    const double d = 1.0 + a;
    r = (float)(1.0 / d);
    w = (float)(a / d);
}

// a_k = dt/t_k of the mixed path where the per-cell stopping time factors as t_k = C_k / F_cell
// (dustyTurb C_k = St_0,k L rho_0, F = c_s rho; the disks' Epstein F = rho/hs c_s, Epstein F = rho c_s of an
// isothermal gas): dt F_cell times the tabulated 1/C_k.  The dusty wave's t_k = rho_k/K_k
// divides per species.
__device__ __forceinline__ double drag_cell_factor(const KParams<float>& p, double dt, double qrho_old, int gx, int gy) {
    if (p.setup == SHARK_SETUP_DUSTYTURB) return dt * (p.csd[gx] * qrho_old);
    if (p.setup == SHARK_SETUP_DISK_CART) {
        const long long e = (long long)gy * p.pitch + gx;
        return dt * (qrho_old / p.chsd[e] * p.ccsd[e]);
    }
    if (p.setup == SHARK_SETUP_DISK_POLAR) return dt * (qrho_old / p.hsd[gx] * p.csd[gx]);
    return dt * (qrho_old * p.csd[gx]);
}

// Drag coefficients and drag heating (source_terms.f90:88-97) of one cell in FP64 for the setups
// whose sound speed or stopping times need the state at the start of the step.  Bound by the FP64
// pipe, so the forms take few of its instructions: F_cell = rho cs = sqrt(gamma P rho) once a cell,
// 1/t_k = F_cell / C_k multiplied out, v.(v - v_k) as (p.p/rho - p.p_k/rho_k)/rho with one quotient a
// species, p.p/rho shared with the kinetic energy, conversions to and from floats as integer
// instructions (adiabatic KH box 500 x 301 x 4: K2 0.076 -> 0.050 ms).
struct DragCell {
    const KParams<float>& p;
    int cc;
    double dt, dtF, w, heat, px, py, pz;   // w = p.p/rho, heat: sum of rho dt v.(v - v_k)/t_k
    Over<double, CONSTANT> by_rho;
    bool wave, heats;
    __device__ __forceinline__ DragCell(const KParams<float>& p_, double dt_, double qrho_old, int gx, int gy, bool heats_,
                                        bool used = true)
        : p(p_), cc(gy * p_.pitch + gx), dt(dt_), dtF(0.0), w(0.0), heat(0.0), px(0.0), py(0.0), pz(0.0),
          by_rho(widen(p_.u_cur[gy * p_.pitch + gx])), wave(p_.setup == SHARK_SETUP_DUSTYWAVE), heats(heats_) {
        const bool adi = used && !wave && p.iso != 1;
        if (adi || heats) {
            px = widen(p.u_cur[cc + p.plane]);
            py = widen(p.u_cur[cc + 2 * p.plane]);
            pz = widen(p.u_cur[cc + 3 * p.plane]);
            w = by_rho(px * px + py * py + pz * pz);
        }
        if (adi) {
            const double P = max64_pos((p.gamma - 1.0) * (widen(p.u_cur[cc + 4 * p.plane]) - 0.5 * w), p.smallp);
            dtF = dt * sqrt(p.gamma * P * qrho_old);
        } else if (used && !wave) {
            dtF = drag_cell_factor(p, dt, qrho_old, gx, gy);
        }
    }
    // species k's density and momenta at the start of the step, where they are needed
    __device__ __forceinline__ float4 load(int k) const {
        if (!wave && !heats) return make_float4(1.f, 0.f, 0.f, 0.f);
        const float* __restrict__ u = p.u_cur + cc + (5 + k) * p.plane;
        const long long s = p.ndust * p.plane;
        return make_float4(u[0], u[s], u[2 * s], u[3 * s]);
    }
    // a_k = dt/t_k of species k, its heating added; o = load(k)
    __device__ __forceinline__ double operator()(int k, float4 o) {
        const Over<double, CONSTANT> by_rd(widen(o.x));
        const double a = wave ? by_rd(dt * p.dK[k]) : dtF * p.dinvts[k];
        if (heats) heat += a * (w - by_rd(px * widen(o.y) + py * widen(o.z) + pz * widen(o.w)));
        return a;
    }
    __device__ __forceinline__ double gain() const { return by_rho(heat); }
};

// The same coefficients in FP32 from a = dt F_cell / C_k formed in FP32 (dt F_cell once per cell
// in FP64, then per species one product): r = 1/(1+a) and w = a r are well conditioned for every
// a >= 0 (no cancellation; a = dt/t_k >> 1 gives r ~ 1/a, w ~ 1 to FP32 rounding), so the state's
// FP32 precision bounds them.  a is capped at 1e30 so that 1 + a stays finite.
__device__ __forceinline__ void drag_coeffs_f(float a, float& r, float& w) {
    a = fminf(a, 1e30f);
    r = 1.0f / (1.0f + a);
    w = a * r;
}

__device__ __forceinline__ void drag_coeffs_mix(double a, float& r, float& w) {
    const double d = 1.0 + a;
    if (__double2hiint(d) < 0x46200000) {   // below 6e29, within FP32 range
        const double q = rcp_refined(d);
        r = narrow(q);
        w = narrow(a * q);
    } else {
        drag_coeffs(a, r, w);
    }
}

// Threads per block of the mixed K2 without growth: small blocks, so that the warps of a block
// waiting at the dt reduction's barrier and the last wave hold fewer idle slots.  The variant with
// fragmenting growth within it takes 256: a cell's sub-cycle in one thread outweighs the reduction.
constexpr int K2M_THREADS = 128;

// Blocks per SM: 8 species at 5 blocks of 128 threads (96 registers), measured best of 4-6; a gas
// alone at 10 (48 registers), whose few loads a thread need many warps (1000^2 21.6 -> 19.5 us against 6,
// 20.0 at 8, 19.7 at 12).  1 and 2 species at 8 (64 registers) against 6:
// KH 500 x 301 x 1 28.5 -> 22.5, SI 1024^2 x 2 34.1 -> 31.4; 4 species stay at 6, where 8 gain on the
// adiabatic box (46.8 -> 44.6) and lose on the isothermal one (40.8 -> 45.1).
template <int NS, int MODE, bool GROW = false>
__global__ void __launch_bounds__(GROW ? 256 : K2M_THREADS,
                                  GROW ? 3 : (NS == 0 ? 10 : NS == 1 || NS == 2 ? 8 : NS == 8 ? 5 : ((NS > 8) ? 2 : 3) * (256 / K2M_THREADS)))
k_finalize_mixed(KParams<float> p) {
    constexpr int NMAX = NS > 0 ? NS : 1;
    const int N = NS >= 0 ? NS : p.ndust;
    const bool drag = (MODE == 0 || MODE == 2) && N > 0 && (p.flags & SHARK_FLAG_DRAG);
    // constant stopping times (SI): the FP64 coefficients of this step were computed once by
    // k_prepare_step; other setups compute them per cell below
    const bool const_ts = p.setup == SHARK_SETUP_SI;
    const float* cr = p.coef;
    const float* cw = p.coef + SHARK_MAX_DUST;
    constexpr bool DRAG = MODE == 0 || MODE == 2, REST = MODE == 0 || MODE == 3;
    chain_begin();
    if (DRAG) stamp_start(p.stamps);
    const double dt = *p.dt;
    const int gx = blockIdx.x * blockDim.x + threadIdx.x + p.ng;
    const int gy = (p.ndim == 2) ? blockIdx.y + p.ng : 0;
    float dtc = 2e38f;
    unsigned int st = 0;
    const bool act = gx < p.ng + p.nx;
    float* u = p.u_next;
    // this cell's element of plane 0, variable v v planes further, as 32-bit offsets from the
    // state's (uniform) base pointer (the context guarantees nvar * plane < 2^31): an access is a
    // 32-bit offset on a uniform base, not a 64-bit address formed per thread
    const int cc = gy * p.pitch + gx;
    const float* __restrict__ ucur = p.u_cur;
    const int pl = (int)p.plane;
    float rho = 0.f, px = 0.f, py = 0.f, pz = 0.f;
    // compile-time species count: the cell's dust state is loaded once into registers (all loads
    // in flight together) and the CFL loop reads it there unless a setup hook rewrote it
    float dr[NMAX], dmx[NMAX], dmy[NMAX], dmz[NMAX];
    bool in_regs = false;
    // courant's dust terms taken in the drag update loop, right after each species' final values
    // (the species' registers then die one by one instead of living until the CFL): allowed when
    // no setup hook changes the dust between the drag and the CFL
    const bool fk_si = (p.flags & SHARK_FLAG_FORCE_KICK) != 0 && p.setup == SHARK_SETUP_SI;
    const bool cfl_in_drag = NS > 0 && NS <= 8 && drag && p.ou_nm == 0 && p.setup != SHARK_SETUP_DISK_POLAR &&
                             p.setup != SHARK_SETUP_DISK_CART &&
                             !(p.setup == SHARK_SETUP_SI && !(p.flags & SHARK_FLAG_FORCE_KICK));
    bool cfl_done = false;
    float vmax_d = 0.f, vv_last = 0.f, fmx2_d = 0.f;
    const float xc = act ? p.xpos[gx] - p.f_half_box_l : 0.f;
    // part 1: drag, floor, drag heating; part 2: kick, setup_inloop, CFL.  With growth in between they
    // are two launches (MODES 2 and 3), or with fragmentation have it between them.
    const bool heats = DRAG && N > 0 && (p.flags & SHARK_FLAG_BACK_REACTION) && p.iso < 1;
    const bool direct = !const_ts && p.setup != SHARK_SETUP_DUSTYTURB && p.setup != SHARK_SETUP_DISK_POLAR &&
                        p.setup != SHARK_SETUP_DISK_CART;
    auto part1 = [&]() {
        bool heated = false;
        double gain = 0.0;
        // the loads take their offsets from an opaque copy of the cell offset, so that the
        // compiler forms the stores' offsets anew instead of keeping every load offset live
        int cl = cc;
        asm volatile("" : "+r"(cl));
        rho = u[cl + (0) * pl];
        px = u[cl + (1) * pl]; py = u[cl + (2) * pl]; pz = u[cl + (3) * pl];
        if constexpr (NS > 0) {
            if (drag) {
#pragma unroll
                for (int k = 0; k < NS; ++k) {
                    dr[k] = u[cl + (5 + k) * pl];
                    dmx[k] = u[cl + (5 + N + k) * pl];
                    dmy[k] = u[cl + (5 + 2 * N + k) * pl];
                    dmz[k] = u[cl + (5 + 3 * N + k) * pl];
                }
                float rk[NMAX], wk[NMAX];
                if (const_ts) {          // the step's coefficients (no FP64 work per cell)
#pragma unroll
                    for (int k = 0; k < NS; ++k) { rk[k] = cr[k]; wk[k] = cw[k]; }
                } else {
                    const float rho_old = ucur[cc + (0) * pl];
                    const double qrho_old = widen(fmaxf(rho_old, p.f_smallr));
                    if (direct) {
                        DragCell dc(p, dt, qrho_old, gx, gy, heats);
#pragma unroll
                        for (int k0 = 0; k0 < NS; k0 += 4) {   // four species' loads in flight together
                            float4 o[4];
#pragma unroll
                            for (int i = 0; i < 4 && k0 + i < NS; ++i) o[i] = dc.load(k0 + i);
#pragma unroll
                            for (int i = 0; i < 4 && k0 + i < NS; ++i) drag_coeffs_mix(dc(k0 + i, o[i]), rk[k0 + i], wk[k0 + i]);
                        }
                        gain = dc.gain();
                        heated = heats;
                    } else {
                        const float Fcf = (float)drag_cell_factor(p, dt, qrho_old, gx, gy);
#pragma unroll
                        for (int k = 0; k < NS; ++k) drag_coeffs_f(Fcf * p.dinvts_f[k], rk[k], wk[k]);
                    }
                }
                float rhon = rho, pnx = px, pny = py, pnz = pz;
#pragma unroll
                for (int k = 0; k < NS; ++k) {
                    pnx += wk[k] * dmx[k];
                    pny += wk[k] * dmy[k];
                    pnz += wk[k] * dmz[k];
                    rhon += wk[k] * dr[k];
                }
                const float irhon = 1.0f / rhon;
                const float vbx = pnx * irhon, vby = pny * irhon, vbz = pnz * irhon;
                const float fl = rho * p.f_dust_ratio_min;   // floor (dust_drag.f90:63-73)
                const float om = p.f_si_om, qsh = p.f_si_q;
#pragma unroll
                for (int k = 0; k < NS; ++k) {
                    const float wr = wk[k] * dr[k];
                    dmx[k] = dmx[k] * rk[k] + wr * vbx;
                    dmy[k] = dmy[k] * rk[k] + wr * vby;
                    dmz[k] = dmz[k] * rk[k] + wr * vbz;
                    u[cc + (5 + N + k) * pl] = dmx[k];
                    u[cc + (5 + 2 * N + k) * pl] = dmy[k];
                    u[cc + (5 + 3 * N + k) * pl] = dmz[k];
                    if (fl > dr[k]) { dr[k] = fl; u[cc + (5 + k) * pl] = fl; }
                    if (cfl_in_drag) {   // the dust loop of courant, see part 2
                        const float ird = 1.0f / dr[k];
                        const float vdx = dmx[k] * ird, vdy = dmy[k] * ird, vdz = dmz[k] * ird;
                        const float vv = fabsf(vdx) + fabsf(vdy) + fabsf(vdz);
                        vmax_d = fmaxf(vmax_d, vv);
                        vv_last = vv;
                        if (fk_si) {
                            const float f1 = 2.0f * qsh * (om * om) * xc - 2.0f * om * vdz;
                            const float f3 = 2.0f * om * vdx;
                            fmx2_d = fmaxf(fmx2_d, f1 * f1 + f3 * f3);
                        }
                        if (!(dr[k] > 0.f)) st |= SHARK_STATUS_NEG_DENSITY;
                        if (!isfinite(vv)) st |= SHARK_STATUS_NAN;
                    }
                }
                cfl_done = cfl_in_drag;
                if (p.flags & SHARK_FLAG_BACK_REACTION) {
                    px = vbx * rho; py = vby * rho; pz = vbz * rho;
                    u[cc + (1) * pl] = px;
                    u[cc + (2) * pl] = py;
                    u[cc + (3) * pl] = pz;
                }
                in_regs = true;
            }
        } else if (drag) {
            float rhon = rho, pnx = px, pny = py, pnz = pz;
            const float rho_old = ucur[cc + (0) * pl];
            const double qrho_old = (double)fmaxf(rho_old, p.f_smallr);
            const float Fcf = (const_ts || direct) ? 0.f : (float)drag_cell_factor(p, dt, qrho_old, gx, gy);
            DragCell dc(p, dt, qrho_old, gx, gy, direct && heats, direct);
            // Run-time species count: two passes over the cell's species, CH species' loads in flight
            // together (a species at a time, each waited for its loads behind the one before's
            // stores: 590 k cells of 32 species 0.27 -> 0.13 ms).  Coefficients that cost FP64 work are
            // kept (thread-local memory) for the second pass, the others formed again.
            constexpr int CH = 4;
            float2 rw_local[SHARK_MAX_DUST];
            for (int k0 = 0; k0 < N; k0 += CH) {
                float d[CH], x[CH], y[CH], z[CH];
                float4 o[CH];
#pragma unroll
                for (int i = 0; i < CH; ++i) {
                    const int k = k0 + i;
                    if (k >= N) break;
                    d[i] = u[cc + (5 + k) * pl];
                    x[i] = u[cc + (5 + N + k) * pl];
                    y[i] = u[cc + (5 + 2 * N + k) * pl];
                    z[i] = u[cc + (5 + 3 * N + k) * pl];
                    if (direct) o[i] = dc.load(k);
                }
#pragma unroll
                for (int i = 0; i < CH; ++i) {
                    const int k = k0 + i;
                    if (k >= N) break;
                    float r, w;
                    if (const_ts) { w = cw[k]; }
                    else if (direct) { drag_coeffs_mix(dc(k, o[i]), r, w); rw_local[k] = make_float2(r, w); }
                    else drag_coeffs_f(Fcf * p.dinvts_f[k], r, w);
                    pnx += w * x[i];
                    pny += w * y[i];
                    pnz += w * z[i];
                    rhon += w * d[i];
                }
            }
            gain = dc.gain();
            heated = direct && heats;
            const float irhon = 1.0f / rhon;
            const float vbx = pnx * irhon, vby = pny * irhon, vbz = pnz * irhon;
            const float fl = rho * p.f_dust_ratio_min;   // floor (dust_drag.f90:63-73)
            for (int k0 = 0; k0 < N; k0 += CH) {
                float d[CH], x[CH], y[CH], z[CH];
#pragma unroll
                for (int i = 0; i < CH; ++i) {
                    const int k = k0 + i;
                    if (k >= N) break;
                    d[i] = u[cc + (5 + k) * pl];
                    x[i] = u[cc + (5 + N + k) * pl];
                    y[i] = u[cc + (5 + 2 * N + k) * pl];
                    z[i] = u[cc + (5 + 3 * N + k) * pl];
                }
#pragma unroll
                for (int i = 0; i < CH; ++i) {
                    const int k = k0 + i;
                    if (k >= N) break;
                    float r, w;
                    if (const_ts) { r = cr[k]; w = cw[k]; }
                    else if (direct) { r = rw_local[k].x; w = rw_local[k].y; }
                    else drag_coeffs_f(Fcf * p.dinvts_f[k], r, w);
                    const float wr = w * d[i];
                    u[cc + (5 + N + k) * pl] = fmaf(wr, vbx, __fmul_rn(x[i], r));
                    u[cc + (5 + 2 * N + k) * pl] = fmaf(wr, vby, __fmul_rn(y[i], r));
                    u[cc + (5 + 3 * N + k) * pl] = fmaf(wr, vbz, __fmul_rn(z[i], r));
                    if (fl > d[i]) u[cc + (5 + k) * pl] = fl;
                }
            }
            if (p.flags & SHARK_FLAG_BACK_REACTION) {
                px = vbx * rho; py = vby * rho; pz = vbz * rho;
                u[cc + (1) * pl] = px;
                u[cc + (2) * pl] = py;
                u[cc + (3) * pl] = pz;
            }
        }
        if (heats) {   // drag heating; without the drag, or with a setup's own stopping times, by itself
            const long long ie = uidx(p, 4, gy, gx);
            if (!heated) {
                const double rho_old = (double)ucur[cc];
                bool inside;
                gain = drag_heating(p, TStop<float>(p, max64_pos(rho_old, p.smallr), gx, gy), gx, gy, dt, inside);
            }
            u[ie] = narrow(widen(u[ie]) + gain);
        }
    };
    auto part2 = [&]() {
        if (REST && p.ou_nm > 0) {                                    // turbulence kick (solve.f90:129-146)
            turb_kick_cell<float>(p, u, gx, gy, dt);
            px = u[cc + (1) * pl];
            py = u[cc + (2) * pl];
        }
        if (REST && p.setup == SHARK_SETUP_SI && !(p.flags & SHARK_FLAG_FORCE_KICK)) {
            // setup_inloop: Crank-Nicolson rotation (SI/setup.f90:299-332)
            in_regs = false;
            const float om = p.f_si_om, qsh = p.f_si_q;
            const float Ohmdt = (float)(p.si_om * dt), O2 = Ohmdt * Ohmdt, inv = 1.0f / (1.0f + O2);
            const float xc = p.xpos[gx] - p.f_half_box_l;
            float AA = 2.0f * qsh * om * xc - 2.0f * p.f_si_r0 * p.f_si_eta;
            {
                const float uz = pz / rho, vx = px / rho;
                pz = rho * (uz * (1.f - O2) + 2.f * vx * Ohmdt + AA * O2) * inv;
                px = rho * (vx * (1.f - O2) - 2.f * uz * Ohmdt + AA * Ohmdt) * inv;
                u[cc + (3) * pl] = pz;
                u[cc + (1) * pl] = px;
            }
            AA = 2.0f * qsh * om * xc;
            for (int k = 0; k < N; ++k) {
                const long long iz = uidx(p, 5 + 3 * N + k, gy, gx), ixx = uidx(p, 5 + N + k, gy, gx);
                const float d = u[cc + (5 + k) * pl];
                const float uz = u[iz] / d, vx = u[ixx] / d;
                u[iz] = d * (uz * (1.f - O2) + 2.f * vx * Ohmdt + AA * O2) * inv;
                u[ixx] = d * (vx * (1.f - O2) - 2.f * uz * Ohmdt + AA * Ohmdt) * inv;
            }
        }
        if (REST && ((p.setup == SHARK_SETUP_DISK_POLAR && disk_inloop_cell<float, float>(p, u, gx, gy, dt)) ||
                          (p.setup == SHARK_SETUP_DISK_CART && cdisk_inloop_cell<float>(p, u, gx, gy)))) {
            in_regs = false;
            rho = u[cc + (0) * pl];
            px = u[cc + (1) * pl];
            py = u[cc + (2) * pl];
            pz = u[cc + (3) * pl];
        }
        // ---- courant on the final state (src/solver/courant.f90:11-124), FP32 ----------------------
        const float cfl = p.f_cfl;
        const float irho = 1.0f / rho;
        const float vx = px * irho, vy = py * irho, vz = pz * irho;
        float cs;
        if (p.iso == 1) cs = p.ccs ? p.ccs[cc] : p.cs[gx];
        else {
            const float E = u[cc + (4) * pl];
            const float ekin = 0.5f * rho * (vx * vx) + 0.5f * rho * (vy * vy) + 0.5f * rho * (vz * vz);
            const float P = fmaxf(p.f_gm1 * (E - ekin), p.f_smallp);
            cs = sqrtf(p.f_gamma * P / fmaxf(rho, p.f_smallr));
            if (!(E == E)) st |= SHARK_STATUS_NAN;
        }
        float dxx;
        if (p.ndim == 1) dxx = p.dx1[gx];
        else if (p.geom == 2) dxx = fminf(p.dx1[gx], p.radc[gx] * p.dx2[gx]);
        else dxx = fminf(p.dx1[gx], p.dx2[gx]);
        float vv = fabsf(vx) + fabsf(vy) + fabsf(vz);
        float vmax = cs + vv;
        float fmx = 0.f;
        const bool fk = fk_si || ((p.flags & SHARK_FLAG_FORCE_KICK) != 0 &&
                                  (p.setup == SHARK_SETUP_DISK_POLAR || p.setup == SHARK_SETUP_DISK_CART));
        const float om = p.f_si_om, qsh = p.f_si_q;
        float fmx2 = 0.f;                 // SI: the largest |f|^2, one square root after the loop
        if (fk_si) {
            const float f1 = 2.0f * qsh * (om * om) * xc - 2.0f * om * vz - 2.0f * p.f_si_r0 * om * p.f_si_eta;
            const float f3 = 2.0f * om * vx;
            fmx2 = f1 * f1 + f3 * f3;
        } else if (fk && p.setup == SHARK_SETUP_DISK_CART) {   // the star's softened force, gas and dust
            fmx = sqrtf(p.cfx[cc] * p.cfx[cc] + p.cfy[cc] * p.cfy[cc]);
        } else if (fk) {
            fmx = fabsf(p.fgrav[gx]);   // polar disk: the point-mass force, the same on gas and dust
        }
        if (cfl_done) {   // dust terms taken in the drag loop: the same maxima, the last species' vv
            vmax = fmaxf(vmax, vmax_d);
            fmx2 = fmaxf(fmx2, fmx2_d);
            vv = vv_last;
        } else {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            float rd, mx, my, mz;
            if (NS > 0 && in_regs) {
                rd = dr[k < NMAX ? k : 0]; mx = dmx[k < NMAX ? k : 0]; my = dmy[k < NMAX ? k : 0]; mz = dmz[k < NMAX ? k : 0];
            } else {
                rd = u[cc + (5 + k) * pl];
                mx = u[cc + (5 + N + k) * pl];
                my = u[cc + (5 + 2 * N + k) * pl];
                mz = u[cc + (5 + 3 * N + k) * pl];
            }
            const float ird = 1.0f / rd;
            const float vdx = mx * ird;
            const float vdy = my * ird;
            const float vdz = mz * ird;
            vv = fabsf(vdx) + fabsf(vdy) + fabsf(vdz);
            vmax = fmaxf(vmax, vv);
            if (fk_si) {
                const float f1 = 2.0f * qsh * (om * om) * xc - 2.0f * om * vdz;
                const float f3 = 2.0f * om * vdx;
                fmx2 = fmaxf(fmx2, f1 * f1 + f3 * f3);
            }
            if (!(rd > 0.f)) st |= SHARK_STATUS_NEG_DENSITY;
            if (!isfinite(vv)) st |= SHARK_STATUS_NAN;
        }
        }
        if (fk_si) fmx = sqrtf(fmx2);
        dtc = cfl * dxx / fabsf(vmax);
        if (fk && vv != 0.f) {
            const float fratio = fmaxf(fmx * dxx / (vv * vv), 1e-3f);
            dtc = fminf(dtc, cfl * dxx / vv * (sqrtf(1.0f + 2.0f * cfl * fratio) - 1.0f) / fratio);
        }
        if (!(rho > 0.f)) st |= SHARK_STATUS_NEG_DENSITY;
        if (!isfinite(vx) || !isfinite(vy) || !isfinite(vz)) st |= SHARK_STATUS_NAN;
        if (!(dtc > 0.f) || !isfinite(dtc)) { st |= SHARK_STATUS_DT_UNDERFLOW; dtc = 2e38f; }
    };
    if (act) {
        part1();
        if (GROW && MODE == 0) st |= grow_in_finalize(p, u, gx, gy, dt);   // dust_growth with fragmentation
        if (MODE != 2) part2();
    }
    if (MODE == 2) return;           // k_growth_f and MODE 3 follow
    block_reduce_dt_f(dtc, st, p.dt_next, p.status);
    if (REST) fill_ghost_images(p, p.u_next, gx, gy);
    if (REST) stamp_end(p.stamps);
}

// Per-step preparation, one small block before the flux kernels: reset the next-dt slot and,
// when the stopping times are per-species constants (SI box), compute the stiff drag
// coefficients 1/(1+a_k) and a_k/(1+a_k), a_k = dt/t_k, once in FP64 (dust_drag.f90:29-46): const_ts
// 1 as floats, 2 as K2's FP64 form takes them.
__device__ __forceinline__ double hash_uniform_d(unsigned long long seed, unsigned long long counter) {
    unsigned long long z = seed * 0x9E3779B97F4A7C15ull + counter + 0x632BE59BD9B4E019ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z = z ^ (z >> 31);
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

// Ornstein-Uhlenbeck update of the forcing coefficients for step `step` (one thread each):
// c <- f c + sigma sqrt(1 - f^2) xi with f = exp(-dt/tcorr) and a Box-Muller normal deviate.
// ou_f (mixed path): the modes' table in floats, KParams::ou_f.
static __global__ void k_ou_update(double* ou, const double* modes, float* ou_f, int nm, const double* dt, double sigma,
                                   double tcorr, unsigned long long seed, long long step, unsigned long long* stamps) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= 2 * nm) return;
    const double f = exp(-(*dt) / tcorr);
    const double sg = sigma * sqrt(1.0 - f * f);
    const unsigned long long cnt = (unsigned long long)(step * nm + q / 2) * 2 + (q & 1);
    const double u1 = hash_uniform_d(seed, 2 * cnt), u2 = hash_uniform_d(seed, 2 * cnt + 1);
    const double xi = sqrt(-2.0 * log(1.0 - u1)) * cos(2.0 * 3.141592653589793238462643383279 * u2);
    ou[q] = f * ou[q] + sg * xi;
    if (ou_f) {
        ou_f[4 * nm + q] = (float)ou[q];
        if (q < nm) {
            const float kx = (float)modes[3 * q], ky = (float)modes[3 * q + 1], kk = (float)modes[3 * q + 2];
            reinterpret_cast<float4*>(ou_f)[q] = make_float4(kx, ky, ky / kk, kx / kk);
        }
    }
    if (q == 0) stamps[1] = clock_ns();
}

// It also posts the step's dt, the status word so far and then the step's number to pinned host
// memory, where the host waits for them: no copy and no event per step.
static __global__ void k_prepare_step(unsigned long long* dt_next, const double* dt, const double* dtstop, int ndust,
                                      int const_ts, float* coef, double* dt_log, StepPost* post, const unsigned int* status,
                                      long long step, unsigned long long* stamps) {
    const int k = threadIdx.x;
    chain_begin();
    if (k == 1) {
        stamps[0] = stamps[1] = clock_ns();
        stamps[3] = 0;
    }
    if (k == 0) {
        *dt_next = (unsigned long long)__double_as_longlong(2e44);
        coef[2 * SHARK_MAX_DUST] = (float)*dt;
        if (dt_log) *dt_log = *dt;
    }
    if (post && k == SHARK_MAX_DUST - 1) {
        post->dt = *dt;
        post->status = *status;
        __threadfence_system();
        *(volatile long long*)&post->step = step;
    }
    if (const_ts == 1 && k < ndust) {
        float r, w;
        drag_coeffs(1.0 * (*dt) / dtstop[k], r, w);
        coef[k] = r;
        coef[SHARK_MAX_DUST + k] = w;
    }
    if (const_ts == 2 && k < ndust) {
        const double a = Over<double>(dtstop[k])(*dt);
        const Over<double> by_a(1.0 + a);
        double* cd = reinterpret_cast<double*>(coef + SHARK_COEF_D);
        cd[k] = by_a(a);
        cd[SHARK_MAX_DUST + k] = by_a.b;
        cd[2 * SHARK_MAX_DUST + k] = by_a.y;
    }
}

// ---------------------------------------------------------------------------------------------
// Layout conversion between the caller's Fortran-order FP64 array and the device state.
// ---------------------------------------------------------------------------------------------
template <typename R>
__global__ void k_from_fortran(const double* __restrict__ src, R* __restrict__ dst, int nx_max, int ny_max,
                               int pitch, long long plane, int nvar) {
    const long long ncells = (long long)nx_max * ny_max;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= ncells * nvar) return;
    const int v = (int)(t / ncells);
    const long long i = t - v * ncells;
    const int iy = (int)(i / nx_max), ix = (int)(i - (long long)iy * nx_max);
    dst[v * plane + (long long)iy * pitch + ix] = R(src[t]);
}

template <typename R>
__global__ void k_to_fortran(const R* __restrict__ src, double* __restrict__ dst, int nx_max, int ny_max,
                             int pitch, long long plane, int nvar) {
    const long long ncells = (long long)nx_max * ny_max;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= ncells * nvar) return;
    const int v = (int)(t / ncells);
    const long long i = t - v * ncells;
    const int iy = (int)(i / nx_max), ix = (int)(i - (long long)iy * nx_max);
    dst[t] = (double)src[v * plane + (long long)iy * pitch + ix];
}

// ctoprim of the whole device state into a Fortran-order FP64 q and cs (solve.f90:195-253).
template <typename R>
__global__ void k_ctoprim(KParams<R> p, const R* __restrict__ u, double* __restrict__ q, double* __restrict__ cs) {
    const long long ncells = (long long)p.nx_max * p.ny_max;
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= ncells) return;
    const int iy = (int)(i / p.nx_max), ix = (int)(i - (long long)iy * p.nx_max);
    const int N = p.ndust;
    const double rho = (double)u[uidx(p, 0, iy, ix)];
    const double px = (double)u[uidx(p, 1, iy, ix)], py = (double)u[uidx(p, 2, iy, ix)], pz = (double)u[uidx(p, 3, iy, ix)];
    q[0 * ncells + i] = rho > p.smallr ? rho : p.smallr;
    q[1 * ncells + i] = px / rho;
    q[2 * ncells + i] = py / rho;
    q[3 * ncells + i] = pz / rho;
    const double ekin = 0.5 * rho * ((px / rho) * (px / rho)) + 0.5 * rho * ((py / rho) * (py / rho)) +
                        0.5 * rho * ((pz / rho) * (pz / rho));
    double P = (p.gamma - 1.0) * ((double)u[uidx(p, 4, iy, ix)] - ekin - 0.0);
    P = P > p.smallp ? P : p.smallp;
    double c;
    if (p.iso == 1) { c = p.csd[ix]; P = rho * (c * c); }
    else c = sqrt(p.gamma * P / q[0 * ncells + i]);
    q[4 * ncells + i] = P;
    if (cs) cs[i] = c;
    for (int k = 0; k < N; ++k) {
        const double rd = (double)u[uidx(p, 5 + k, iy, ix)];
        q[(5 + k) * ncells + i] = rd;
        q[(5 + N + k) * ncells + i] = (double)u[uidx(p, 5 + N + k, iy, ix)] / rd;
        q[(5 + 2 * N + k) * ncells + i] = (double)u[uidx(p, 5 + 2 * N + k, iy, ix)] / rd;
        q[(5 + 3 * N + k) * ncells + i] = (double)u[uidx(p, 5 + 3 * N + k, iy, ix)] / rd;
    }
}

// ---------------------------------------------------------------------------------------------
// Kahan-compensated FP64 totals per species (deterministic two-level tree).
// Stage 1: each block Kahan-sums a contiguous range of active cells for all 4*(N+1) sums.
// Stage 2: one block combines the per-block (sum, compensation) pairs in a fixed order.
// ---------------------------------------------------------------------------------------------
template <typename R>
__global__ void k_totals_stage1(KParams<R> p, const R* __restrict__ u, double* __restrict__ part, long long per_block) {
    const int S = p.ndust + 1;
    const long long nact = (long long)p.nx * (p.ndim == 2 ? p.ny : 1);
    const long long b0 = blockIdx.x * per_block;
    const long long b1 = min(nact, b0 + per_block);
    // one quantity per thread group: threads stride over the 4*S quantities
    for (int qi = threadIdx.x; qi < 4 * S; qi += blockDim.x) {
        const int s = qi / 4, c = qi % 4;
        const int v = svar(s, c, p.ndust);
        double sum = 0.0, comp = 0.0;
        for (long long a = b0; a < b1; ++a) {
            const int iy = (p.ndim == 2) ? (int)(a / p.nx) + p.ng : 0;
            const int ix = (int)(a % p.nx) + p.ng;
            const double y = (double)u[uidx(p, v, iy, ix)] - comp;
            const double t = sum + y;
            comp = (t - sum) - y;
            sum = t;
        }
        part[(blockIdx.x * (long long)(4 * S) + qi) * 2 + 0] = sum;
        part[(blockIdx.x * (long long)(4 * S) + qi) * 2 + 1] = comp;
    }
}

static __global__ void k_totals_stage2(const double* __restrict__ part, int nblocks, int nq, double* __restrict__ out) {
    for (int qi = threadIdx.x; qi < nq; qi += blockDim.x) {
        double sum = 0.0, comp = 0.0;
        for (int b = 0; b < nblocks; ++b) {
            // add the block's sum minus its own compensation, compensated
            const double y = (part[((long long)b * nq + qi) * 2 + 0] - part[((long long)b * nq + qi) * 2 + 1]) - comp;
            const double t = sum + y;
            comp = (t - sum) - y;
            sum = t;
        }
        out[qi] = sum;
    }
}

}  // namespace shark
