// The FP64 matrix instruction of the factorisation and the two filters.
#pragma once
#include <cuda_runtime.h>

namespace verb {
namespace {

// c (8 x 8: row lane / 4, columns 2 (lane % 4), + 1) += a (8 x 4: row lane / 4,
// column lane % 4) times b (4 x 8: row lane % 4, column lane / 4), the four
// products added in ascending order, one fused multiply-add each
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

}  // namespace
}  // namespace verb
