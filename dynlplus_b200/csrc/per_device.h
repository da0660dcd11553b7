// What is set once per device of a process. Plain C++ (no CUDA header).
#pragma once

#include <stdint.h>

#include <atomic>

namespace dlp {

// set() is called until it succeeds once for device `dev`, and not again for that device; true when it has.
// `done` holds a bit per device (a device past the 64th is set on every call). Two threads may both set.
template <class Set>
inline bool once_per_device(std::atomic<uint64_t> &done, int dev, Set set) {
  const bool known = dev >= 0 && dev < 64;
  if (known && (done.load(std::memory_order_acquire) >> dev & 1u)) return true;
  if (!set()) return false;
  if (known) done.fetch_or(uint64_t(1) << dev, std::memory_order_release);
  return true;
}

}  // namespace dlp
