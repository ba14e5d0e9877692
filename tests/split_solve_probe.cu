// The split form's kinematic-wave solve on given values, for tests/test_split_solve_gpu.py (built there
// with the split kernels' flags).
#include <cstdint>

#include <cuda_runtime.h>

#include "wf_kw_ff.cuh"

namespace {
// rows of x: cterm, dt / dx, alpha, previous u; rows of out: u, Q
__global__ void solve_kernel(const double* x, double* out, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    wff::ff u, q;
    wfk::kw_solve_ff(wff::from_d(x[i]), wff::from_d(x[n + i]), (float)x[2 * n + i], (float)x[3 * n + i], u, q);
    out[i] = wff::to_d(u);
    out[n + i] = wff::to_d(q);
}
}  // namespace

extern "C" int solve_device(const double* x, double* out, int64_t n) {
    double *d = nullptr, *o = nullptr;
    cudaMalloc((void**)&d, 32 * n);
    cudaMalloc((void**)&o, 16 * n);
    cudaMemcpy(d, x, 32 * n, cudaMemcpyHostToDevice);
    solve_kernel<<<(unsigned)((n + 127) / 128), 128>>>(d, o, n);
    cudaMemcpy(out, o, 16 * n, cudaMemcpyDeviceToHost);
    const int rc = (int)cudaGetLastError();
    cudaFree(d);
    cudaFree(o);
    return rc;
}
