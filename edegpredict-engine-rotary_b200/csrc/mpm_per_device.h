// A positive number worked out once per device of the process: a kernel's
// attributes and what fits on an SM belong to the device that was current when
// they were set or asked for, not to the process.
#pragma once

#include <atomic>

namespace mpmb {

class PerDevice {
  public:
    static constexpr int kMaxDevices = 64;

    // The number of device `dev`; f() works it out (0: not known, asked again
    // the next time).  Threads that ask at once may each run f.
    template <typename F> int get(int dev, F&& f) {
        if (dev < 0 || dev >= kMaxDevices) return f();
        int v = v_[dev].load(std::memory_order_acquire);
        if (v <= 0) {
            v = f();
            if (v > 0) v_[dev].store(v, std::memory_order_release);
        }
        return v;
    }

  private:
    std::atomic<int> v_[kMaxDevices] = {};
};

}  // namespace mpmb
