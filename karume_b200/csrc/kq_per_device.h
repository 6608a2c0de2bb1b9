// What a launcher learns about a kernel once for each device.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

namespace kq {

// Attributes set before a kernel's first launch and limits learnt from the device belong to a device, not to the
// process (a host may drive several GPUs from one), and are shared by all contexts, whose threads may make their
// first calls at the same time: nobody sees an entry before it is complete.
template <typename T, int kDevices = 64>
class PerDevice {
 public:
  // The entry of the calling thread's current device; `learn(T&)`, which returns a cudaError_t, fills it the first time.
  template <typename Learn>
  cudaError_t get(Learn learn, const T** out) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kDevices) return cudaErrorInvalidDevice;
    Entry& entry = entries_[device];
    if (!entry.known.load(std::memory_order_acquire)) {
      std::lock_guard<std::mutex> hold(lock_);
      if (!entry.known.load(std::memory_order_relaxed)) {
        T value = {};
        const cudaError_t e = learn(value);
        if (e != cudaSuccess) return e;
        entry.value = value;
        entry.known.store(true, std::memory_order_release);
      }
    }
    *out = &entry.value;
    return cudaSuccess;
  }

 private:
  struct Entry {
    std::atomic<bool> known{false};
    T value = {};
  };
  Entry entries_[kDevices];
  std::mutex lock_;
};

// Attributes only: nothing to remember but that they are set.
class OncePerDevice {
 public:
  template <typename Learn>
  cudaError_t run(Learn learn) {
    const bool* done = nullptr;
    return flags_.get([&](bool& flag) { flag = true; return learn(); }, &done);
  }

 private:
  PerDevice<bool> flags_;
};

}  // namespace kq
