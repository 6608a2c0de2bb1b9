// Host-side check of what launchers learn once for each device (karume_b200/csrc/kq_per_device.h): threads that ask for an
// entry at the same time all see it complete, it is filled once per device, and a failure leaves it to be asked again.
// cudaGetDevice is this program's own: the device of a thread is a variable here.
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>

#include "kq_per_device.h"

static thread_local int t_device = 0;
extern "C" cudaError_t CUDARTAPI cudaGetDevice(int* device) {
  *device = t_device;
  return cudaSuccess;
}

struct Limits { unsigned clusters[16]; };

int main() {
  kq::PerDevice<Limits, 4> limits;
  std::atomic<int> filled[4] = {}, wrong{0}, ready{0};
  constexpr int kThreads = 12;
  auto fill = [&](int device) {
    return [&filled, device](Limits& l) {
      ++filled[device];
      for (unsigned i = 0; i < 16; ++i) {
        l.clusters[i] = 100u * device + i + 1;
        std::this_thread::sleep_for(std::chrono::milliseconds(1));
      }
      return cudaSuccess;
    };
  };
  std::vector<std::thread> threads;
  for (int t = 0; t < kThreads; ++t)
    threads.emplace_back([&, t] {
      const int device = t % 3;
      t_device = device;
      ++ready;
      while (ready.load() < kThreads) std::this_thread::yield();
      std::this_thread::sleep_for(std::chrono::milliseconds(2 * (t / 3)));  // some arrive in the middle of the filling
      const Limits* seen = nullptr;
      if (limits.get(fill(device), &seen) != cudaSuccess || seen == nullptr) ++wrong;
      else
        for (unsigned i = 0; i < 16; ++i) wrong += seen->clusters[i] != 100u * device + i + 1;
    });
  for (std::thread& t : threads) t.join();
  if (wrong.load() != 0) return std::printf("FAIL: %d words not there yet\n", wrong.load()), 1;
  for (int d = 0; d < 3; ++d)
    if (filled[d].load() != 1) return std::printf("FAIL: device %d filled %d times\n", d, filled[d].load()), 1;
  const Limits* seen = nullptr;
  t_device = 3;
  if (limits.get([](Limits&) { return cudaErrorNotSupported; }, &seen) != cudaErrorNotSupported || seen != nullptr)
    return std::printf("FAIL: an error is the caller's\n"), 1;
  if (limits.get(fill(3), &seen) != cudaSuccess || seen->clusters[0] != 301) return std::printf("FAIL: asked again after an error\n"), 1;
  t_device = 4;
  if (limits.get(fill(3), &seen) != cudaErrorInvalidDevice) return std::printf("FAIL: a device past the last\n"), 1;
  std::printf("ok\n");
  return 0;
}
