// The last column of a range against the same in 64-bit integers, at grid sizes
// up to the largest and coordinates one float apart around each size.
#include "column_range.h"

#include <algorithm>
#include <cstdint>
#include <cstdio>

int main() {
    long bad = 0;
    for (int64_t base : {1ll, 2ll, 1000ll, 1ll << 20, 1ll << 24, 1ll << 25, 1ll << 30, (1ll << 31) - 1})
        for (int64_t n = std::max<int64_t>(base - 40, 1); n <= std::min<int64_t>(base + 40, (1ll << 31) - 1); ++n) {
            float h = (float)n;
            for (int k = 0; k < 50; ++k) h = nextafterf(h, -INFINITY);
            for (int k = 0; k < 100; ++k, h = nextafterf(h, INFINITY)) {
                const int64_t want = std::min<int64_t>((int64_t)std::floor((double)h), n - 1);
                if (lbm::last_column(h, (int)n) != want) {
                    if (bad++ < 5) std::printf("n %lld hi %.9g: %d, %lld\n", (long long)n, h, lbm::last_column(h, (int)n), (long long)want);
                }
            }
            for (float far : {-1e30f, -3.5f, -0.5f, 0.f, 1e30f, INFINITY}) {
                const int64_t want = far < 0 ? (int64_t)std::floor((double)std::max(far, -3.5f)) : (far > 0 ? n - 1 : 0);
                if (far > -1e29f && lbm::last_column(far, (int)n) != want) ++bad;
            }
        }
    std::printf(bad ? "failed\n" : "column range ok\n");
    return bad ? 1 : 0;
}
