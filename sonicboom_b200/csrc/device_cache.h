// A number that belongs to a kernel on one device (how many of its clusters run at once), asked for once per device.
// Safe with several threads; a query that fails is not kept.
#pragma once

#include <atomic>

struct SbDeviceCache {
  static constexpr int DEVICES = 64;
  std::atomic<int> kept[DEVICES] = {};                 // the answer + 1; 0: not asked yet

  // query() gives the answer (0 or more), or a negative number when it could not be had.
  template <typename Query>
  int get(int device, Query query) {
    const bool keeps = device >= 0 && device < DEVICES;
    if (keeps) {
      const int v = kept[device].load(std::memory_order_relaxed);
      if (v > 0) return v - 1;
    }
    const int answer = query();
    if (keeps && answer >= 0) kept[device].store(answer + 1, std::memory_order_relaxed);
    return answer;
  }
};
