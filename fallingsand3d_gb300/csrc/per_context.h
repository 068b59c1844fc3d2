// A value that holds for one context of one device (a kernel's attributes, what
// they allow): made when first asked for there, and again when another context
// is current on that device.  Safe from any thread.
#pragma once

#include <mutex>

namespace fs3d {

template <class T>
class PerContext {
    static constexpr int kDevices = 64;
    struct Slot {
        unsigned long long ctx = 0;  // the context `v` was made in (0: none)
        T v{};
    };
    Slot slots_[kDevices];
    std::mutex mu_;

public:
    // id(): the calling thread's current context (0: none yet; make() brings it about)
    template <class Id, class Make>
    T get(int dev, Id id, Make make) {
        std::lock_guard<std::mutex> lock(mu_);
        if (dev < 0 || dev >= kDevices) return make();
        Slot& s = slots_[dev];
        const unsigned long long ctx = id();
        if (!ctx || s.ctx != ctx) {
            s.v = make();
            s.ctx = id();
        }
        return s.v;
    }
};

}  // namespace fs3d
