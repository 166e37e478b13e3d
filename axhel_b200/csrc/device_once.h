// Work that is needed once per device, such as a kernel's function attributes
// (cudaFuncSetAttribute acts on the current device only).
#pragma once

#include <atomic>
#include <cstdint>
#include <mutex>

namespace axhel_impl {

class DeviceOnce {
public:
    // Runs `set`, which returns 0 on success, unless it has succeeded on device
    // `dev`; its result, or 0.  The usual case, done before, takes no lock.
    // (Devices from 64 on, for which there is no bit, run it on every call.)
    template <class Set>
    auto operator()(int dev, std::mutex& mu, const Set& set) -> decltype(set())
    {
        const uint64_t bit = dev >= 0 && dev < 64 ? 1ull << dev : 0;
        if (done_.load(std::memory_order_acquire) & bit) return {};
        std::lock_guard<std::mutex> lk(mu);
        if (done_.load(std::memory_order_relaxed) & bit) return {};
        const auto e = set();
        if (e == decltype(set()){}) done_.fetch_or(bit, std::memory_order_release);
        return e;
    }

private:
    std::atomic<uint64_t> done_{0};
};

}  // namespace axhel_impl
