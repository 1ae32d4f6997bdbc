// croma_once.cuh -- something to be done once on every device: a kernel's
// attributes, which CUDA keeps per device while contexts of one process may sit
// on several.  Nothing of CUDA is needed to compile it.
#pragma once

#include <atomic>

namespace croma {

class OncePerDevice {
public:
    // set() on the first call of each device, its error until it succeeds; 0 is
    // success.  Threads that call at once may both run it.
    template <class F>
    auto operator()(int device, F set) -> decltype(set())
    {
        if (device < 0 || device >= kDevices) return set();
        if (done_[device].load(std::memory_order_acquire)) return decltype(set())(0);
        const auto e = set();
        if (e == decltype(set())(0)) done_[device].store(true, std::memory_order_release);
        return e;
    }

private:
    static constexpr int kDevices = 64;
    std::atomic<bool> done_[kDevices] = {};
};

}  // namespace croma
