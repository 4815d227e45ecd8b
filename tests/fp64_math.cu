// The FP64 Newton reciprocal and reciprocal square root of the pair loops, over an array.
#include "../sph-2d_b200/csrc/common.cuh"

__global__ void k_math(int n, const double* x, double* r, double* q) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { r[i] = sph::rcp64(x[i]); q[i] = sph::rsqrt64(x[i]); }
}

extern "C" int fp64_math(int n, const double* x, double* r, double* q) {
    k_math<<<(n + 255) / 256, 256>>>(n, x, r, q);
    return (int)cudaDeviceSynchronize();
}
