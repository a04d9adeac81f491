// once.h -- set-up that runs once per device of the process.
#pragma once

#include <atomic>
#include <mutex>

// Callers that arrive while a device's set-up runs wait for it, and every caller on
// that device gets its status.  (Kernel attributes belong to a device: a process
// that works on several sets them on each.)
struct B200Once {
  static constexpr int DEVICES = 64;
  std::mutex mutex;
  std::atomic<bool> done[DEVICES] = {};
  int status[DEVICES] = {};

  template <class F>
  int run(int device, F setup) {
    if (device < 0 || device >= DEVICES) return setup();
    if (!done[device].load(std::memory_order_acquire)) {
      std::lock_guard<std::mutex> lock(mutex);
      if (!done[device].load(std::memory_order_relaxed)) {
        status[device] = setup();
        done[device].store(true, std::memory_order_release);
      }
    }
    return status[device];
  }
};
