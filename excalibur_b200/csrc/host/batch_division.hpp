// How a forward's batch is divided into sub-batches whose copies and kernels overlap.
#pragma once
#include <algorithm>
#include <cmath>
#include <functional>
#include <vector>

namespace glasssix {
namespace excalibur {

constexpr double kBodyPower = 0.85;

// The division of n images whose modelled time is shortest, or {n} where none promises 3 % and 20 us.  Copies to the
// device, kernels and copies back are three lanes that run side by side; a sub-batch passes through them one after the
// other.  in_us and out_us: the copies of the whole batch; the kernels of a share s of the images take
// fixed_us + body_us * s^kBodyPower (small sub-batches fill the chip less).  Divisions are looked for among all ways to put 16
// units together, n units of one image below 16 images, in at most eight parts.
inline std::vector<int> divide_batch(int n, double in_us, double out_us, double fixed_us, double body_us) {
    constexpr int kUnits = 16, kParts = 8;
    const std::vector<int> undivided{n};
    if (n < 2) return undivided;
    const int units = std::min(n, kUnits);
    double kernels[kUnits + 1];
    for (int u = 0; u <= units; ++u) kernels[u] = fixed_us + body_us * std::pow(u / (double)units, kBodyPower);
    const double whole = in_us + kernels[units] + out_us;
    double best = std::min(0.97 * whole, whole - 20.0);
    std::vector<int> parts, best_parts;
    std::function<void(int, double, double, double)> walk = [&](int left, double in, double run, double out) {
        if (out >= best) return;
        if (left == 0) {
            best = out;
            best_parts = parts;
            return;
        }
        if ((int)parts.size() == kParts) return;
        for (int u = 1; u <= left; ++u) {
            const double in2 = in + in_us * u / units + 6.0, run2 = std::max(run, in2) + kernels[u] + 4.0;
            const double out2 = std::max(out, run2) + out_us * u / units + 6.0;
            parts.push_back(u);
            walk(left - u, in2, run2, out2);
            parts.pop_back();
        }
    };
    walk(units, 0, 0, 0);
    if (best_parts.empty()) return undivided;
    std::vector<int> sizes;
    int done_units = 0, done = 0;
    for (int u : best_parts) {
        done_units += u;
        const int upto = (int)((long long)n * done_units / units);
        sizes.push_back(upto - done);
        done = upto;
    }
    return sizes;
}

}  // namespace excalibur
}  // namespace glasssix
