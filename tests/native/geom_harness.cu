// Test harness: the shortened division and arctangent of geom.cuh on arrays,
// compiled by tests/test_gpu_geom_math.py with the library's flags. Host
// pointers; returns a CUDA error code.
#include <cuda_runtime.h>

#include "geom.cuh"

namespace {

__global__ void k_eval(const double *a, const double *b, double *out, int n, int what) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = what == 0 ? axgb::d_div_by(a[i], b[i], __drcp_rn(b[i])) : axgb::d_twice_atan(a[i], b[i]);
}

}  // namespace

// what 0: d_div_by(a, b), 1: d_twice_atan(a, b)
extern "C" int geom_eval(const double *a, const double *b, double *out, int n, int what) {
    double *d = nullptr;
    cudaError_t e = cudaMalloc(reinterpret_cast<void **>(&d), 3 * sizeof(double) * n);
    if (e != cudaSuccess) return e;
    cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
    k_eval<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * n, n, what);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * n, sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
