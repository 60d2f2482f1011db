// Division of a whole row by its quantisation scale.
#pragma once

#include <cuda_runtime.h>

namespace pk100 {

// x / s for every element of a row, correctly rounded, at three multiply-adds per element instead of
// a full division each: q = x * y with y = RN(1 / s), r = RN(x - q * s), q' = RN(q + r * y)
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990).
// q may be more than one unit off, so the published proof does not cover it; for an fp16 x and a scale m / 448
// or m / 127 of an fp16 m the result is that of IEEE division for all 2^20 pairs of significands, which stand
// for all values because every step scales with powers of two (tests/test_row_division.py).  The sign of x is
// put back because the correction turns -0 into +0 (E4M3 codes keep the sign of zero).
struct RowDivisor {
    float s, y;
    __device__ __forceinline__ explicit RowDivisor(float scale) {
        s = scale;
        y = __frcp_rn(scale);
        if (isinf(scale)) { s = 1.0f; y = 0.0f; }         // finite / inf = 0, inf / inf = NaN
    }
    __device__ __forceinline__ RowDivisor(float divisor, float reciprocal) { s = divisor; y = reciprocal; }
    __device__ __forceinline__ float operator()(float x) const {
        const float q = x * y;
        return copysignf(fmaf(fmaf(-q, s, x), y, q), x);
    }
};

}  // namespace pk100
