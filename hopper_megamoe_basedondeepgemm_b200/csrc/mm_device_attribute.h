// A kernel attribute of each device that is raised on demand, from any thread: the opt-in shared memory size. Plain host code.
#pragma once
#include <atomic>

namespace mm {

class DeviceAttribute {
 public:
    // Sees to it that the attribute is at least `value` on device `dev`: `set()` sets it and returns 0, or an error, which is handed on. Whoever raises it does so
    // alone: of two threads with two sizes the smaller one could otherwise be set last, under a launch that needs the larger one.
    template <typename Set>
    auto raise(int dev, int value, Set set) -> decltype(set()) {
        if (dev < 0 || dev >= kDevices) return set();
        if (value_[dev].load(std::memory_order_acquire) >= value) return {};
        while (raising_.test_and_set(std::memory_order_acquire)) { }         // (a few calls in a process's life; a mutex could throw through the C entries)
        decltype(set()) error{};
        if (value_[dev].load(std::memory_order_relaxed) < value) {
            error = set();
            if (error == decltype(set()){}) value_[dev].store(value, std::memory_order_release);
        }
        raising_.clear(std::memory_order_release);
        return error;
    }

 private:
    static constexpr int kDevices = 64;
    std::atomic<int> value_[kDevices] = {};
    std::atomic_flag raising_ = ATOMIC_FLAG_INIT;
};

}  // namespace mm
