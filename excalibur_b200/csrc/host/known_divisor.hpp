// Correctly rounded division by an integer that is known before the dividend, without a division: the two-word reciprocal
// of Brisebarre, Muller and Raina, "Accelerating correctly rounded floating-point division when the divisor is known in
// advance" (IEEE Trans. Computers 53(8), 2004).  With hi = RN(1/d) and lo = RN(1/d - hi), RN(x * hi + RN(x * lo)) is
// x / d but for an error below 2^-46 before its one rounding.  A quotient of a 24-bit x by an integer d <= 25 is either
// exact (d a power of two: lo is 0, the product is) or at least 2^-30 away from the middle of two neighbours, so the
// rounding is that of the quotient.
#pragma once
#include <cfloat>
#include <cmath>

#ifdef __CUDACC__
#define EXB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define EXB_HOST_DEVICE inline
#endif

namespace exb {

struct KnownDivisor {
    float hi, lo;
};
constexpr int kMaxKnownDivisor = 25;

inline KnownDivisor known_divisor(int d) {
    const float hi = (float)(1.0 / d);
    return {hi, (float)(1.0 / d - (double)hi)};
}

// x / d for every x: infinities and NaN are their own quotients.
EXB_HOST_DEVICE float divide_by(float x, const KnownDivisor& d) {
#ifdef __CUDA_ARCH__
    const float q = fmaf(x, d.hi, __fmul_rn(x, d.lo));
#else
    const volatile float low = x * d.lo;
    const float q = std::fma(x, d.hi, (float)low);
#endif
    return fabsf(x) <= FLT_MAX ? q : x;
}

}  // namespace exb
