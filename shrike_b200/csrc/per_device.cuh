// What a process does once on every device that it uses.  Host code without any CUDA call of its own.
#pragma once
#include <atomic>

// Attributes of a kernel (its limit of dynamic shared memory, above all) belong to a device: one flag for the whole process
// would leave them unset on the second device.  `once` runs `act` (which returns 0 when it has done its work) if it has not
// succeeded on `device` yet, and returns what it returned; threads that come at the same time may both run it.  Devices
// beyond the 64 that are kept track of run it every time.
struct PerDevice {
  std::atomic<unsigned long long> done{0};
  template <typename Act>
  int once(int device, Act&& act) {
    const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0;
    if (done.load(std::memory_order_acquire) & bit) return 0;
    const int status = act();
    if (status == 0) done.fetch_or(bit, std::memory_order_release);
    return status;
  }
};
