// The device paths of wf_math.cuh on given values, for tests/test_fp64_math_gpu.py (built there with
// the FP64 kernels' flags). out holds N_OUT arrays of n values.
#include <cstdint>

#include <cuda_runtime.h>

#include "wf_math.cuh"

namespace {
constexpr int N_OUT = 11;

WF_HD void evaluate(double a, double b, double* o) {
    o[0] = wfm::div_(a, b);
    o[1] = wfm::div_by_(a, b, 1.0 / b);
    o[2] = wfm::exp(a);
    o[3] = wfm::log(wfm::fabs_(a));
    o[4] = wfm::pow(wfm::fabs_(a), 0.2);
    o[5] = wfm::jmin(a, b);
    o[6] = wfm::jmax(a, b);
    o[7] = wfm::jclamp(a, -1.0, b);
    o[8] = wfm::cld(a, wfm::fabs_(b));
    o[9] = wfm::cbrt(a);
    o[10] = wfm::lt_(a, b) + 2 * wfm::le_(a, b) + 4 * wfm::gt0_(a) + 8 * wfm::le0_(a) + 16 * wfm::is_zero_(a) +
            32 * wfm::isnan_(a);
}

__global__ void evaluate_kernel(const double* a, const double* b, double* out, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double o[N_OUT];
    evaluate(a[i], b[i], o);
    for (int k = 0; k < N_OUT; ++k) out[k * n + i] = o[k];
}
}  // namespace

extern "C" int probe_host(const double* a, const double* b, double* out, int64_t n) {
    for (int64_t i = 0; i < n; ++i) {
        double o[N_OUT];
        evaluate(a[i], b[i], o);
        for (int k = 0; k < N_OUT; ++k) out[k * n + i] = o[k];
    }
    return N_OUT;
}

extern "C" int probe_device(const double* a, const double* b, double* out, int64_t n) {
    double *da = nullptr, *db = nullptr, *dout = nullptr;
    const size_t bytes = (size_t)n * sizeof(double);
    cudaMalloc((void**)&da, bytes);
    cudaMalloc((void**)&db, bytes);
    cudaMalloc((void**)&dout, bytes * N_OUT);
    cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(db, b, bytes, cudaMemcpyHostToDevice);
    evaluate_kernel<<<(unsigned)((n + 127) / 128), 128>>>(da, db, dout, n);
    cudaMemcpy(out, dout, bytes * N_OUT, cudaMemcpyDeviceToHost);
    const int rc = (int)cudaGetLastError();
    cudaFree(da);
    cudaFree(db);
    cudaFree(dout);
    return rc;
}
