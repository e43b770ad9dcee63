// Something to be done once on every device of the process.
#pragma once

#include <atomic>
#include <cstdint>
#include <mutex>

namespace dcg {

class OncePerDevice {
public:
    // Runs f() unless it has succeeded (returned 0) on this device before; its status.  Safe with several threads.
    template <typename F>
    int operator()(int device, F f)
    {
        const bool known = device >= 0 && device < 64;
        const uint64_t bit = known ? 1ull << device : 0;
        if (done_.load(std::memory_order_acquire) & bit) return 0;
        std::lock_guard<std::mutex> lock(mutex_);
        if (done_.load(std::memory_order_relaxed) & bit) return 0;
        const int status = (int)f();
        if (status == 0) done_.fetch_or(bit, std::memory_order_release);
        return status;
    }

private:
    std::atomic<uint64_t> done_{0};
    std::mutex mutex_;
};

}  // namespace dcg
