// Device paths of wf_math.cuh, li_scheme.cuh and wf_wave.cuh on given values, for
// tests/test_fp64_bits_gpu.py (built there with the FP64 kernels' flags).
#include <cstdint>

#include <cuda_runtime.h>

#include "li_scheme.cuh"
#include "wf_math.cuh"
#include "wf_wave.cuh"

namespace {
constexpr int N_QUOT = 3;

// quotients: with a kept reciprocal, with the correctly rounded one, and without one
WF_HD void quotients(double a, double b, double* o) {
#ifdef __CUDA_ARCH__
    const double r = wfm::rcp_kept(b);
    o[0] = wfm::is_zero_(r) ? a / b : wfm::div_by_(a, b, r);
    o[1] = wfm::div_by_(a, b, wfm::div_(1.0, b));
    o[2] = wfm::div_(a, b);
#else
    o[0] = o[1] = o[2] = a / b;
#endif
}

__global__ void quotient_kernel(const double* a, const double* b, double* out, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double o[N_QUOT];
    quotients(a[i], b[i], o);
    for (int k = 0; k < N_QUOT; ++k) out[k * n + i] = o[k];
}

// the edge flows of the local-inertial schemes: columns q0, zs0, zs1, hf, width and n^2 (a
// cell length of 100 m, a step of 5 s)
constexpr int N_EDGE = 6;
WF_HD void edge(const double* x, int64_t n, int64_t i, double* out) {
    const double q0 = x[i], zs0 = x[n + i], zs1 = x[2 * n + i], hf = x[3 * n + i], w = x[4 * n + i],
                 nsq = x[5 * n + i];
    const double A = w * hf, R = wfm::div_(A, 2.0 * hf + w);
    out[i] = wfli::flow(q0, zs0, zs1, hf, A, R, 100.0, 1.0 / 100.0, nsq, true, 5.0);
    out[n + i] = wfli::flow_rect(0.9, q0, 0.5 * q0, 0.7 * q0, zs0, zs1, hf, w, 100.0, 1.0 / 100.0, nsq, true, 5.0);
}
__global__ void edge_kernel(const double* x, double* out, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) edge(x, n, i, out);
}

// words published to other warps
__global__ void publish_kernel(const unsigned long long* w, unsigned long long* out, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) wfv::st_relaxed(&out[i], w[i]);
}

template <class Launch>
int on_device(const void* in, size_t in_bytes, void* out, size_t out_bytes, Launch launch) {
    unsigned char *d = nullptr, *o = nullptr;
    cudaMalloc((void**)&d, in_bytes);
    cudaMalloc((void**)&o, out_bytes);
    cudaMemcpy(d, in, in_bytes, cudaMemcpyHostToDevice);
    launch(d, o);
    cudaMemcpy(out, o, out_bytes, cudaMemcpyDeviceToHost);
    const int rc = (int)cudaGetLastError();
    cudaFree(d);
    cudaFree(o);
    return rc;
}
unsigned blocks(int64_t n) { return (unsigned)((n + 127) / 128); }
}  // namespace

extern "C" {
// ab: n values of a, then n of b; out: N_QUOT n values
int quotients_host(const double* ab, double* out, int64_t n) {
    for (int64_t i = 0; i < n; ++i) {
        double o[N_QUOT];
        quotients(ab[i], ab[n + i], o);
        for (int k = 0; k < N_QUOT; ++k) out[k * n + i] = o[k];
    }
    return 0;
}
int quotients_device(const double* ab, double* out, int64_t n) {
    return on_device(ab, 16 * n, out, 8 * N_QUOT * n, [&](unsigned char* d, unsigned char* o) {
        quotient_kernel<<<blocks(n), 128>>>((const double*)d, (const double*)d + n, (double*)o, n);
    });
}
int edges_host(const double* x, double* out, int64_t n) {
    for (int64_t i = 0; i < n; ++i) edge(x, n, i, out);
    return 0;
}
int edges_device(const double* x, double* out, int64_t n) {
    return on_device(x, 8 * N_EDGE * n, out, 16 * n, [&](unsigned char* d, unsigned char* o) {
        edge_kernel<<<blocks(n), 128>>>((const double*)d, (double*)o, n);
    });
}
int publish_device(const uint64_t* w, uint64_t* out, int64_t n) {
    return on_device(w, 8 * n, out, 8 * n, [&](unsigned char* d, unsigned char* o) {
        publish_kernel<<<blocks(n), 128>>>((const unsigned long long*)d, (unsigned long long*)o, n);
    });
}
}
