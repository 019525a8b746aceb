// Correctly rounded division by an integer that is known before the dividend, without a division: the two-word reciprocal
// of Brisebarre, Muller and Raina, "Accelerating correctly rounded floating-point division when the divisor is known in
// advance" (IEEE Trans. Computers 53(8), 2004), RN(x * hi + RN(x * lo)) with hi + lo = 1/d.  That is x / d but for an error
// below 2^-45 before its one rounding, and a quotient of a 24-bit x by an integer d <= 25 is either exact (d a power of
// two: the product with hi is) or at least 2^-30 away from the middle of two neighbours.
// hi is rounded down here and lo is positive, for a power of two the smallest normal number, which is far below half a
// unit of any quotient: so an infinite x gives inf + inf and not inf - inf or inf * 0.
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
    float hi = (float)(1.0 / d);
    if ((double)hi > 1.0 / d) hi = std::nextafter(hi, 0.f);
    const float lo = (float)(1.0 / d - (double)hi);
    return {hi, lo > FLT_MIN ? lo : FLT_MIN};
}

// x / d for |x| of 2^-24 to 2^21, zero, infinities and NaN: sums of up to 25 fp16 values.
EXB_HOST_DEVICE float divide_by(float x, const KnownDivisor& d) {
#ifdef __CUDA_ARCH__
    return fmaf(x, d.hi, __fmul_rn(x, d.lo));
#else
    const volatile float low = x * d.lo;
    return std::fma(x, d.hi, (float)low);
#endif
}

}  // namespace exb
