// A value made once per device of the process (a kernel's attribute, the number of
// SMs): attributes belong to a kernel on one device, and a process may drive several
// from several threads.
#pragma once
#include <atomic>

namespace xbg {

class PerDevice {
    static constexpr int MAX = 64;
    std::atomic<int> v[MAX] = {};   // 0: not made yet

  public:
    // The device's value, by make() on first use; 0 is a failure, which is not kept.
    // Two threads may both make it (make gives the same to both).
    template <class F>
    int get(int dev, F&& make) {
        if (dev < 0) return 0;
        if (dev >= MAX) return make();
        int r = v[dev].load(std::memory_order_acquire);
        if (!r && (r = make())) v[dev].store(r, std::memory_order_release);
        return r;
    }
};

}  // namespace xbg
