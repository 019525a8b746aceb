// divide_batch: a whole division for every batch size, divided wherever overlap pays, undivided where it does not.
#include <cstdio>
#include <numeric>

#include "batch_division.hpp"

using glasssix::excalibur::divide_batch;

static int failures = 0;
#define EXPECT(cond, n)                                                       \
    do {                                                                      \
        if (!(cond)) {                                                        \
            std::printf("line %d, %d images: %s\n", __LINE__, (int)(n), #cond); \
            ++failures;                                                       \
        }                                                                     \
    } while (0)

int main() {
    for (int n = 1; n <= 300; n = n < 40 ? n + 1 : n + 37) {
        // large images: copies in, kernels and copies out of one image take a millisecond each
        const double ms = 1000.0 * n;
        const std::vector<int> d = divide_batch(n, ms, ms, 100.0, ms);
        EXPECT(std::accumulate(d.begin(), d.end(), 0) == n, n);
        EXPECT(d.size() <= 8, n);
        for (int k : d) EXPECT(k >= 1, n);
        EXPECT(n == 1 || d.size() > 1, n);
        // two lanes next to nothing: nothing to overlap
        EXPECT(divide_batch(n, 1.0, 1.0, 100.0, ms).size() == 1, n);
    }
    // two images of equal lanes: one each
    EXPECT(divide_batch(2, 2000, 2000, 0, 2000) == (std::vector<int>{1, 1}), 2);
    std::printf(failures ? "%d failures\n" : "ok\n", failures);
    return failures != 0;
}
