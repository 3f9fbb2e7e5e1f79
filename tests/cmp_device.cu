/* The refined reciprocal, roots and 2/3 power of the device code over arrays,
 * for test_gpu_math.py. */
#include "gf_ghost.cu"

namespace gf {
namespace {

__global__ void eval_kernel(int op, const double* __restrict__ x, double* __restrict__ y, int n)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const double a = x[k];
    y[k] = op == 0 ? gf_rcp(a) : op == 1 ? gf_rsqrt_n(a) : op == 2 ? gf_sqrt_n(a) : pow23<true>(a);
}

} // namespace
} // namespace gf

extern "C" int eval(int op, const double* x, double* y, int n)
{
    double *dx = nullptr, *dy = nullptr;
    cudaError_t e = cudaMalloc(&dx, n * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&dy, n * sizeof(double));
    if (e == cudaSuccess) e = cudaMemcpy(dx, x, n * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        gf::eval_kernel<<<(n + 255) / 256, 256>>>(op, dx, dy, n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(y, dy, n * sizeof(double), cudaMemcpyDeviceToHost);
    if (dx) cudaFree(dx);
    if (dy) cudaFree(dy);
    return (int)e;
}
