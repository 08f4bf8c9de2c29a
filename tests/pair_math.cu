// Errors of the FP64 pair root and reciprocal (equation/ns_pair.cuh), compiled and run by
// tests/test_pair_math_gpu.py.  For every x: the error of each function in units of the last place
// of its result, and the relative error of the hardware approximation it starts from.
#include <cuda_runtime.h>

#include "ns_pair.cuh"

namespace {

__device__ double ulp_of(double r) {
    return __longlong_as_double(__double_as_longlong(r) + 1) - r;
}

// out[0..3] of x: error of the root and of the reciprocal (ulp), of their starts (relative)
__global__ void k_errors(const double* __restrict__ x, int n, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    const double s = sph::pair_sqrt(v), r = sph::pair_rcp(v);
    // sqrt(v) - s = (v - s^2) / (sqrt(v) + s), 1/v - r = (1 - v r) / v: the residuals by fused
    // operations, rounded once, so both errors are good to more than ten digits
    out[4 * i] = __fma_rn(-s, s, v) / (sqrt(v) + s) / ulp_of(s);
    out[4 * i + 1] = __fma_rn(-v, r, 1.0) / v / ulp_of(r);
    double y, z;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(z) : "d"(v));
    // v y^2 - 1 = 2 delta for a start off by delta
    out[4 * i + 2] = 0.5 * __fma_rn(__dmul_rn(v, y), y, -1.0);
    out[4 * i + 3] = __fma_rn(v, z, -1.0);
}

// out[0..3] of x: the two functions, and CUDA's square root and division
__global__ void k_values(const double* __restrict__ x, int n, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[4 * i] = sph::pair_sqrt(x[i]);
    out[4 * i + 1] = sph::pair_rcp(x[i]);
    out[4 * i + 2] = __dsqrt_rn(x[i]);
    out[4 * i + 3] = __ddiv_rn(1.0, x[i]);
}

}  // namespace

// x and out (4 n doubles) in device memory; returns the CUDA status
extern "C" int pair_math(const double* x, int n, double* out, int values) {
    if (n <= 0) return 0;
    if (values)
        k_values<<<(n + 255) / 256, 256>>>(x, n, out);
    else
        k_errors<<<(n + 255) / 256, 256>>>(x, n, out);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
