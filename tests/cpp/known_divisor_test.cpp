// divide_by: bit for bit the division, for every significand and every divisor, and for values that are not finite.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <limits>

#include "known_divisor.hpp"

static uint32_t bits(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
}

int main() {
    using namespace exb;
    long bad = 0;
    for (int d = 1; d <= kMaxKnownDivisor; ++d) {
        const KnownDivisor k = known_divisor(d);
        const volatile float df = (float)d;
        for (uint32_t exponent : {127u - 24, 127u, 127u + 20})
            for (uint32_t m = 0; m < (1u << 23); ++m) {
                const uint32_t u = exponent << 23 | m;
                float x;
                std::memcpy(&x, &u, 4);
                bad += bits(divide_by(x, k)) != bits(x / df);
            }
        // zero, infinities, the range of sums of fp16 values
        const float inf = std::numeric_limits<float>::infinity();
        for (float x : {0.f, -0.f, inf, -inf, 5.9604645e-8f, -5.9604645e-8f, 65504.f * 25, -65504.f * 25}) bad += bits(divide_by(x, k)) != bits(x / df);
        bad += !std::isnan(divide_by(std::numeric_limits<float>::quiet_NaN(), k));
    }
    std::printf(bad ? "%ld differ\n" : "ok\n", bad);
    return bad != 0;
}
