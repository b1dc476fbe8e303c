// quotient.h -- x / q for many x of one q, without a division each (mlp.cu; checked on the host).
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define PACH_QUOTIENT_FN __host__ __device__ __forceinline__
#else
#define PACH_QUOTIENT_FN inline
#endif

namespace pach {
namespace mlp {

// x / q from rq, the rounded reciprocal of q, and one residual step (Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", 1990).  For 0 <= x <= 1 <= q <= 32: correctly rounded where x is 0 or at
// least 2^-96, as the residual x - q y is then exact; below that it is rounded to a multiple of 2^-149, and the result
// can be the next one to the rounded quotient (a lobe's responsibility of 1e-29 or less).
constexpr float kQuotientExact = 0x1p-96f;
PACH_QUOTIENT_FN float quotient(float x, float q, float rq) {
    const float y = x * rq;
    return fmaf(fmaf(-q, y, x), rq, y);
}

}  // namespace mlp
}  // namespace pach
#undef PACH_QUOTIENT_FN
