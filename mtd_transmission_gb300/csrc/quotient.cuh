// Divisions as a product with a reciprocal and one correction of the quotient by
// its remainder (P. Markstein, Computation of elementary functions on the IBM
// RISC System/6000 processor, 1990), used by the gather and the Poisson solve.
#pragma once

#include <cuda_runtime.h>

namespace tdm {

// x / n from r the correctly rounded 1 / n, n a whole number of at most 65535:
// correctly rounded where the quotient is a normal number (within one unit of
// 2^-149 below); infinities and NaN as the division gives them.
__device__ __forceinline__ float over(float x, float n, float r) {
    const float q = x * r, rest = fmaf(-q, n, x);
    return rest == rest ? fmaf(rest, r, q) : q;
}

// x / y for y and the quotient well inside the normal range, within one unit in the last
// place of the division's result: from an approximate reciprocal.
__device__ __forceinline__ float quotient(float x, float y) {
    const float r = __fdividef(1.0f, y), q = x * r;
    return fmaf(fmaf(-q, y, x), r, q);
}

}  // namespace tdm
