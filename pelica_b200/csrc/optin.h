// optin.h - the opt-in of a kernel to more dynamic shared memory than every kernel gets unasked. It belongs to
// (kernel, device): a context on a second GPU of the process needs its own. Raised and never lowered, under a lock: two
// host threads whose layers need different sizes would otherwise leave the smaller one in force. Plain C++, no CUDA.
#pragma once

#include <atomic>
#include <mutex>

struct SmemOptIn {
  static constexpr int DEVICES = 64;
  std::atomic<int> have[DEVICES] = {};  // bytes in force per device
  std::mutex lock;
  // set(bytes): 0 when the device took it, else an error code, which is handed back (and asked for again by the next call).
  // Without the lock once a device has what is asked for.
  template <class Set> int raise(int device, int bytes, Set set) {
    const bool known = device >= 0 && device < DEVICES;
    if (known && have[device].load(std::memory_order_acquire) >= bytes) return 0;
    std::lock_guard<std::mutex> hold(lock);
    if (known && have[device].load(std::memory_order_relaxed) >= bytes) return 0;
    const int e = set(bytes);
    if (e == 0 && known) have[device].store(bytes, std::memory_order_release);
    return e;
  }
};
