// Calls the FP64 helpers of shark_gb300/csrc/fp64.cuh and the limiters of physics.cuh element by
// element for tests/test_gpu_fp64_forms.py, which compiles this file.
#include "physics.cuh"

using namespace shark;

enum { DIV, RCP, MIN, MAX, LESS, MINMOD, VAN_LEER, MC, NARROW, WIDEN, OPS };

__global__ void k_check(int n, const double* a, const double* b, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = a[i], y = b[i];
    out[(size_t)DIV * n + i] = div64(x, y, rcp64(y));
    out[(size_t)RCP * n + i] = rcp64_any(y);
    out[(size_t)MIN * n + i] = min64(x, y);
    out[(size_t)MAX * n + i] = max64(x, y);
    out[(size_t)LESS * n + i] = is_less(x, y) ? 1.0 : 0.0;
    out[(size_t)MINMOD * n + i] = limit_minmod_d(x, y);
    out[(size_t)VAN_LEER * n + i] = limit_vl_d(x, y);
    out[(size_t)MC * n + i] = limit_mc_d(x, y);
    out[(size_t)NARROW * n + i] = (double)narrow(x);
    out[(size_t)WIDEN * n + i] = widen((float)x);
}

// out: OPS rows of n.  Returns 0, or a CUDA error code.
extern "C" int fp64_check(int n, const double* a, const double* b, double* out) {
    double *da = nullptr, *db = nullptr, *dout = nullptr;
    const size_t bytes = (size_t)n * sizeof(double);
    cudaError_t e = cudaMalloc(&da, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&db, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&dout, OPS * bytes);
    if (e == cudaSuccess) e = cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(db, b, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) k_check<<<(n + 127) / 128, 128>>>(n, da, db, dout);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, OPS * bytes, cudaMemcpyDeviceToHost);
    cudaFree(da);
    cudaFree(db);
    cudaFree(dout);
    return (int)e;
}
