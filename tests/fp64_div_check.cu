// The division helpers of fp64_div.cuh on arrays, beside plain division.
#include <cuda_runtime.h>

#include "fp64_div.cuh"

namespace {
__global__ void check_kernel(int n, const double* a, const double* b, double* out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double seed;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(seed) : "d"(b[i]));
        const double y = zk::recip(b[i]);
        const size_t N = n;
        out[i] = seed;
        out[N + i] = y;
        out[2 * N + i] = zk::quot(a[i], b[i], y);
        out[3 * N + i] = zk::divide(a[i], b[i]);
        out[4 * N + i] = 1.0 / b[i];
        out[5 * N + i] = a[i] / b[i];
        out[6 * N + i] = __fma_rn(-b[i], seed, 1.0);
        out[7 * N + i] = zk::in_range(b[i]) ? 1.0 : 0.0;
        out[8 * N + i] = zk::num_ok(a[i]) ? 1.0 : 0.0;
    }
}
}  // namespace

// out: 9 rows of n (n > 0), see the kernel.  Returns the CUDA error code.
extern "C" int fp64_div_check(int n, const double* a, const double* b, double* out) {
    double* d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof(double) * 11 * n);
    if (e != cudaSuccess) return e;
    cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
    check_kernel<<<(n + 255) / 256, 256>>>(n, d, d + n, d + 2 * (size_t)n);
    e = cudaMemcpy(out, d + 2 * (size_t)n, sizeof(double) * 9 * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
