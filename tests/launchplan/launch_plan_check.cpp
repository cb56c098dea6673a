// Launch plans against a fake kernel attribute: threads that ask for different
// block sizes of one kernel always find its limit at least as high as their own
// blocks need, each plan is queried once, a failed call leaves no plan behind.
#include "launch_plan.h"

#include <algorithm>
#include <cstdio>
#include <thread>
#include <vector>

using lbm::LaunchPlans;

static std::atomic<long> bad{0};
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); ++bad; } } while (0)

int main() {
    for (int round = 0; round < 200; ++round) {
        LaunchPlans plans;
        std::atomic<size_t> limit[2] = {{LaunchPlans::kDefaultLimit}, {LaunchPlans::kDefaultLimit}};
        std::atomic<int> queries[2][9] = {};
        std::vector<std::thread> th;
        for (int t = 0; t < 8; ++t)
            th.emplace_back([&, t] {
                for (int i = 0; i < 400; ++i) {
                    const int dev = (t + i) & 1, wpb = 1 + (t * 5 + (i / 2) * 3) % 8;
                    const size_t smem = (size_t)wpb * 15712;
                    const int n = plans.blocks(dev, wpb, smem,
                                               [&](size_t b) { limit[dev].store(b); return true; },
                                               [&] { ++queries[dev][wpb]; return 100 * dev + wpb; });
                    CHECK(n == 100 * dev + wpb);
                    CHECK(limit[dev].load() >= smem);       // what a launch of these blocks needs
                }
            });
        for (std::thread& t : th) t.join();
        for (int d = 0; d < 2; ++d) {
            CHECK(limit[d].load() == (size_t)8 * 15712);
            for (int w = 1; w <= 8; ++w) CHECK(queries[d][w] == 1);
        }
    }
    LaunchPlans plans;
    int raised = 0;
    CHECK(plans.blocks(0, 4, 60000, [&](size_t) { return false; }, [] { return 7; }) == 0);     // the raise fails
    CHECK(plans.blocks(0, 4, 60000, [&](size_t) { ++raised; return true; }, [] { return 0; }) == 0);   // the query fails
    CHECK(plans.blocks(0, 4, 60000, [&](size_t) { ++raised; return true; }, [] { return 9; }) == 9);   // tried again
    CHECK(raised == 1);
    CHECK(plans.blocks(0, 1, 15000, [&](size_t) { ++raised; return true; }, [] { return 5; }) == 5);   // below the limit
    CHECK(raised == 1);
    CHECK(plans.blocks(LaunchPlans::kDevices - 1, LaunchPlans::kWarps, 1, [](size_t) { return true; }, [] { return 3; }) == 3);
    std::printf(bad ? "failed\n" : "launch plans ok\n");
    return bad ? 1 : 0;
}
