// Kernels in parity mode: compiled with -fmad=false, correctly rounded
// division and square root, the reference's bits (gk_physics.cuh).
#define GK_NS gk_parity
#define GK_FASTMATH 0
#include "gk_kernels.cuh"

namespace gk_parity {

// The branch-free quotient, reciprocal and square root of n operand pairs:
// out[0..n) = a/b, out[n..2n) = 1/b, out[2n..3n) = sqrt(a).
__global__ void k_math_eval(int n, const double* __restrict__ a, const double* __restrict__ b,
                            double* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        out[i] = div_rn(a[i], b[i]);
        out[n + i] = rcp_rn(b[i]);
        out[2 * n + i] = sqrt_rn(a[i]);
    }
}

int math_eval(int n, const double* a, const double* b, double* out) {
    const size_t nb = sizeof(double) * (size_t)n;
    double* d = nullptr;
    if (cudaMalloc(&d, 5 * nb) != cudaSuccess) return -1;
    cudaError_t e = cudaMemcpy(d, a, nb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, b, nb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_math_eval<<<148 * 4, 256>>>(n, d, d + n, d + 2 * (size_t)n);
        e = cudaMemcpy(out, d + 2 * (size_t)n, 3 * nb, cudaMemcpyDeviceToHost);
    }
    cudaFree(d);
    return e == cudaSuccess ? 0 : -1;
}

}  // namespace gk_parity
