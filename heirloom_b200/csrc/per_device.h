// What has been asked of, or told to, each device once in this process: kernel attributes belong to a device, and so does how many
// CTAs or clusters of a kernel it holds.  One of these is a function's static; any thread may use it.  Threads that come first at
// the same time ask more than once and store the same answer.
#pragma once
#include <atomic>

namespace hl {

class PerDevice {
 public:
  // The device's value: what is stored, or what `ask` returns, which is stored when it is not zero (zero: could not be found out).
  template <typename F>
  int value(int device, F ask) {
    if (device < 0 || device >= kDevices) return ask();
    int v = known_[device].load(std::memory_order_acquire);
    if (v == 0 && (v = ask()) != 0) known_[device].store(v, std::memory_order_release);
    return v;
  }
  // Runs `act` for the device until it has returned zero once; returns what it returned, zero when it was not run.
  template <typename F>
  auto once(int device, F act) -> decltype(act()) {
    decltype(act()) result{};
    value(device, [&] {
      result = act();
      return result == decltype(act()){} ? 1 : 0;
    });
    return result;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<int> known_[kDevices] = {};
};

}  // namespace hl
