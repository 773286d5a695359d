// What a process sets up once on every device that it launches on: a kernel's limit of shared memory and the like, which
// CUDA keeps per device.
#pragma once
#include <atomic>

#define SNK_MAX_DEVICES 64

// *value: what make(value) left there on this device, a positive number (a device's SMs).  `seen` keeps it: SNK_MAX_DEVICES
// zeros at first.  Returns 0 or make's error, which is not kept: the next call tries again.  Threads that meet on a
// device's first call may both make it.
template <typename Make>
inline int snk_per_device(std::atomic<int>* seen, int device, int* value, Make make) {
  const bool kept = device >= 0 && device < SNK_MAX_DEVICES;
  if (kept && (*value = seen[device].load(std::memory_order_acquire)) > 0) return 0;
  const int rc = make(value);
  if (rc == 0 && kept) seen[device].store(*value, std::memory_order_release);
  return rc;
}
