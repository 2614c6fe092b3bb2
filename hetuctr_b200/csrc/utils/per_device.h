// Things that a process does once for every device it uses.  Kernel attributes (shared memory beyond 48 KB, cluster sizes)
// and occupancies belong to the device that is current when they are set or asked for, so "once" is once per device; the
// tables of several thread ranks get here at the same time.
#pragma once
#include <atomic>

namespace hetuCTR {

// One value per device: 0 until it is known, then what `make` returned.  Static storage only (zero-initialised).
// `make` may run more than once when several threads ask first; what it does has to bear that.
class PerDevice {
 public:
  template <class F>
  int get(int device, F make) {
    if (device < 0 || device >= kDevices) return make();  // (not remembered)
    int v = known_[device].load(std::memory_order_acquire);
    if (v == 0) {
      v = make();
      if (v != 0) known_[device].store(v, std::memory_order_release);
    }
    return v;
  }
  // `act` returns 0 on success; repeated until it has succeeded on the device, 0 from then on.
  template <class F>
  int once(int device, F act) {
    int status = 0;
    get(device, [&] {
      status = act();
      return status == 0 ? 1 : 0;
    });
    return status;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<int> known_[kDevices];
};

}  // namespace hetuCTR
