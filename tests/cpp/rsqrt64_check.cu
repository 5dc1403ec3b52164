// Runs the functions of rsqrt64.cuh on n values, for the test that holds them against extended precision.
#include "../../grasph2_b200/csrc/rsqrt64.cuh"

__global__ void k_check(const double* x, double* seed, double* half, double* cube, int* in_range, int n) {
    const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= n) return;
    in_range[i] = gsph::series_range64(x[i]);
    seed[i] = gsph::rsqrt_seed64(x[i]);
    half[i] = gsph::inv_sqrt64(x[i]);
    cube[i] = gsph::inv_cube64(x[i]);
}

// x: n inputs; out: 3 n results (seed, x^(-1/2), x^(-3/2)); in_range: n flags; all on the host. Returns a CUDA error code.
extern "C" int rsqrt64_check(const double* x, double* out, int* in_range, int n) {
    double* d = nullptr;
    int* f = nullptr;
    cudaError_t e = cudaMalloc(&d, 4 * sizeof(double) * n);
    if (e == cudaSuccess) e = cudaMalloc(&f, sizeof(int) * n);
    if (e == cudaSuccess) e = cudaMemcpy(d, x, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_check<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * static_cast<size_t>(n), d + 3 * static_cast<size_t>(n), f, n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + n, 3 * sizeof(double) * n, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(in_range, f, sizeof(int) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    cudaFree(f);
    return static_cast<int>(e);
}
