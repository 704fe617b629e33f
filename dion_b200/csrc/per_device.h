// What has to be done once per device before a kernel's first launch there: the opt-in to more than 48 KB of dynamic shared
// memory belongs to the device that is current, and a backward pass launches from other threads than the forward.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace dion {

// Calls `prepare` unless it has succeeded on the current device before; `done` keeps a bit for each of the first 64 devices, beyond
// them it is called every time.  Two threads may both call it: it must be one that can be repeated.
template <typename Prepare>
cudaError_t once_per_device(std::atomic<unsigned long long>& done, Prepare prepare) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = prepare();
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

}  // namespace dion
