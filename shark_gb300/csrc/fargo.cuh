// fargo.cuh -- K3: the FARGO orbital remap (src/solver/fargo_scheme.f90:2-81) of the polar disk.
//
// After the conservative update every ring (fixed radius, all phi) is shifted by vk*dt: the shift
// splits into whole cells nshft and a fraction eps of a cell, and each cell's new value is the
// linear remap of its two donor cells plus their limited-slope correction.  The remap is a
// rotation of the ring, so it cannot run in place: the kernel reads the flux kernel's output and
// writes a third state buffer.
//
// The remap moves each value once, so memory bounds it (mixed, 4.2 TB/s); in FP64 the limiter's and the
// remap's operations do (the FP64 pipe 81 % busy).  A thread owns one column of one conserved
// variable and marches down FARGO_ROWS output rows with its window of donor cells in registers:
// an output costs one load, one limited slope (the lower donor's is the next output's upper one) and
// one store; the loads of FARGO_BATCH rows are in flight together.  A warp's 32 lanes are adjacent
// columns: neighbouring columns' shifts differ by few cells, so its loads fall on few rows.
// What a column shares (whole cells, weights) a kernel of one thread per column forms first, in FP64
// in both precisions: the two divisions and the remainder cost more than the remap of a column.
// 512 x 1024, 16 species, mixed: 0.254 -> 0.060 ms; 128 x 256, FP64: 0.081 -> 0.053 ms (before: whole
// rings staged in shared memory by blocks of 64-byte row segments, two limited slopes an output, the
// shifts formed by every block).
//
// Restated with the defects of the reference fixed (the oracle does the same):
//   `one` is 1 and `eps` FP64 (an undeclared uninitialised REAL and an implicit REAL*4 there);
//   slopes exist for every active cell, with the ring's periodic wrap;
//   donor rows wrap modulo ny (the reference wraps once).
#pragma once

#include "step_kernels.cuh"

namespace shark {

constexpr int FARGO_ROWS = 32, FARGO_BATCH = 8, FARGO_WARPS = 8;

template <typename R>
__global__ void k_fargo_shift(KParams<R> p, FargoShift<R>* __restrict__ tab) {
    const int gx = p.ng + blockIdx.x * blockDim.x + threadIdx.x, ny = p.ny;
    if (gx >= p.ng + p.nx) return;
    const double one = 1.0, half = 0.5, forth = 0.25;
    const double vk = p.vkd[gx];
    const double dy_loc = p.dx2d[gx] * p.radcd[gx];
    const double shift = fabs(vk * (*p.dt));
    const double ns = shift / dy_loc;
    const long long nshft = ns < 9.0e18 ? (long long)ns : 0;
    const double eps = fmod(shift, dy_loc) / dy_loc;
    FargoShift<R> t;
    long long off;
    if (vk > 0.0) { off = -(nshft % ny) - 1; t.w0 = R(eps); t.w1 = R(one - eps); }
    else { off = nshft % ny; t.w0 = R(one - eps); t.w1 = R(eps); }
    if (off < 0) off += ny;
    t.off = (int)off;
    t.c1 = R(forth - (half - eps) * (half - eps));
    t.c2 = R((half - eps) * (half - eps) - forth);
    tab[gx] = t;
}

template <typename R, int ST>
__global__ void __launch_bounds__(32 * FARGO_WARPS)
k_fargo(KParams<R> p, const FargoShift<R>* __restrict__ tab, const R* __restrict__ src, R* __restrict__ dst) {
    const int ny = p.ny, pitch = p.pitch;
    const int gx = p.ng + blockIdx.x * 32 + threadIdx.x;
    const int a0 = (blockIdx.y * FARGO_WARPS + threadIdx.y) * FARGO_ROWS;
    if (gx >= p.ng + p.nx || a0 >= ny) return;
    const FargoShift<R> t = tab[gx];
    const long long base = (long long)blockIdx.z * p.plane + (long long)p.ng * pitch + gx;
    const R* __restrict__ q = src + base;
    R* __restrict__ out = dst + base + (long long)a0 * pitch;
    // element offsets within the ring: a state buffer's plane is below 2^31 elements
    const int ring = ny * pitch;
    int o = (a0 + t.off) % ny * pitch;   // the first output's lower donor
    const R half = R(0.5);
    const R um = q[o == 0 ? ring - pitch : o - pitch];
    auto next = [&]() { o += pitch; if (o == ring) o = 0; return q[o]; };
    R u0 = q[o], u1 = next();
    R du0 = slope_limit_t<ST, R>(u0 - um, u1 - u0);
    const int n = min(FARGO_ROWS, ny - a0);
    for (int a = 0; a < n; a += FARGO_BATCH) {
        R u[FARGO_BATCH];
#pragma unroll
        for (int i = 0; i < FARGO_BATCH; ++i) u[i] = next();
#pragma unroll
        for (int i = 0; i < FARGO_BATCH; ++i) {
            const R du1 = slope_limit_t<ST, R>(u1 - u0, u[i] - u1);
            R un = u0 * t.w0 + u1 * t.w1;
            un = un + half * du0 * t.c1 + half * du1 * t.c2;
            if (a + i < n) out[(a + i) * pitch] = un;
            u0 = u1;
            u1 = u[i];
            du0 = du1;
        }
    }
}

}  // namespace shark
