// Something found or set up once for every device of the process (plain C++).
//
// A kernel's attributes (its limit of dynamic shared memory) and what the occupancy calls
// say belong to the device that was current when they were set or asked; a program may use
// several.
#pragma once

#include <mutex>

namespace eg {

template <typename T>
class PerDevice {
  public:
    // The value of device `dev`: find() the first time, by one thread.
    template <typename F>
    T get(int dev, F find) {
        if (dev < 0 || dev >= kDevices) return find();
        Slot &s = slots_[dev];
        std::call_once(s.once, [&] { s.value = find(); });
        return s.value;
    }

  private:
    static constexpr int kDevices = 64;
    struct Slot {
        std::once_flag once;
        T value{};
    };
    Slot slots_[kDevices];
};

} // namespace eg
