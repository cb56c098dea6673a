// Launch plans of one kernel: the blocks resident at once, per device and block
// size, and the kernel's dynamic shared memory limit per device.  Handles of
// different block sizes, on different threads, share a kernel, so a plan once
// found stays, the limit is only ever raised, and both happen under a lock; a
// launch after the first of its block size takes one atomic load.
#pragma once
#include <atomic>
#include <cstddef>
#include <mutex>

namespace lbm {

class LaunchPlans {
public:
    static constexpr int kDevices = 64, kWarps = 8;
    static constexpr size_t kDefaultLimit = 48 * 1024;      // without an opt-in

    // Blocks resident at once for blocks of wpb warps (1 .. kWarps) and smem bytes
    // on device dev (0 .. kDevices - 1); 0 if a call failed.  raise(bytes) raises the
    // kernel's limit, query() returns the resident blocks; both return less than 1
    // on failure, and the next call tries again.  smem is a function of wpb.
    template <class Raise, class Query>
    int blocks(int dev, int wpb, size_t smem, Raise raise, Query query) {
        std::atomic<int>& plan = resident_[dev][wpb].blocks;
        const int known = plan.load(std::memory_order_acquire);
        if (known > 0) return known;
        std::lock_guard<std::mutex> lock(mutex_);
        if (const int found = plan.load(std::memory_order_relaxed)) return found;      // by the thread before
        const size_t limit = limit_[dev] ? limit_[dev] : kDefaultLimit;
        if (smem > limit) {
            if (raise(smem) < 1) return 0;
            limit_[dev] = smem;
        }
        const int n = query();
        if (n < 1) return 0;
        plan.store(n, std::memory_order_release);
        return n;
    }

private:
    struct Plan {
        std::atomic<int> blocks{0};
    };
    std::mutex mutex_;
    Plan resident_[kDevices][kWarps + 1];
    size_t limit_[kDevices] = {};
};

}  // namespace lbm
