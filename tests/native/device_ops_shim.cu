/*
 * device_ops_shim.cu -- test-only device build of the product's FP64 cell
 * operators (lbm_multigpu_gb300/csrc/d3q19.cuh): their square root and
 * reciprocal exist in device code alone.  Not part of the product library.
 */
#include "../../lbm_multigpu_gb300/csrc/d3q19.cuh"

using namespace lbm;

__global__ void k_map(int what, const double* x, double* y, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    y[i] = what == 0 ? lsqrt<double>(x[i]) : what == 1 ? dsqrt<double>(x[i]) : lrcp<double>(x[i]);
}
__global__ void k_collide(int les, double omega, double cs, double* f, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double g[19];
    for (int q = 0; q < 19; ++q) g[q] = f[19 * i + q];
    collide_mrt_pop<double>(g, omega, les != 0, 1.0 / omega, 18.0 * 1.4142135623730951 * cs);
    for (int q = 0; q < 19; ++q) f[19 * i + q] = g[q];
}

static int run(int what, int les, double omega, double cs, const double* in, double* out, int n, int width) {
    double *a = nullptr, *b = nullptr;
    const size_t bytes = sizeof(double) * size_t(n) * width;
    cudaError_t e = cudaMalloc(&a, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&b, bytes);
    if (e == cudaSuccess) e = cudaMemcpy(a, in, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        if (width == 1) k_map<<<(n + 255) / 256, 256>>>(what, a, b, n);
        else k_collide<<<(n + 127) / 128, 128>>>(les, omega, cs, a, n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, width == 1 ? b : a, bytes, cudaMemcpyDeviceToHost);
    cudaFree(a);
    cudaFree(b);
    return int(e);
}

extern "C" {
/* what: 0 lsqrt, 1 dsqrt, 2 lrcp */
int dev_map(int what, const double* x, double* y, int n) { return run(what, 0, 0, 0, x, y, n, 1); }
int dev_collide(int les, double omega, double cs, const double* in, double* out, int n) {
    return run(0, les, omega, cs, in, out, n, 19);
}
}
