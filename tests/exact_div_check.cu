// Shared reciprocals and quotients of csrc/exact_div.cuh beside CUDA's own, for
// tests/test_gpu_exact_div.py.
#include <cstddef>

#include "exact_div.cuh"

namespace {

__global__ void check_kernel(const double* a, const double* b, size_t n, double* quot, double* ref,
                             double* rec, double* rref)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double y = verb::recip(b[i]);
    quot[i] = verb::div_by(a[i], b[i], y);
    ref[i] = a[i] / b[i];
    rec[i] = y;
    rref[i] = __drcp_rn(b[i]);
}

}  // namespace

// device arrays of n
extern "C" int exact_div_check(const double* a, const double* b, size_t n, double* quot, double* ref,
                               double* rec, double* rref)
{
    check_kernel<<<(unsigned)((n + 255) / 256), 256>>>(a, b, n, quot, ref, rec, rref);
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? (int)e : (int)cudaDeviceSynchronize();
}
