// device_cfg.h -- launch settings that belong to a device: its SM count, and per kernel the opt-in
// to dynamic shared memory beyond 48 KB with the CTAs that then fit on an SM.  Asked once per
// device: a process may solve on one device after another, and an opt-in made on the first does
// not hold on the next.
#pragma once
#include <cuda_runtime.h>
#include <atomic>

namespace chfem {

constexpr int MAX_DEVICES = 64;  // devices past these are asked every time

// One value per device, 0 while not known yet (static storage; any thread may fill it in).
struct PerDevice {
  std::atomic<int> v[MAX_DEVICES];
};
template <typename Ask>
int per_device(PerDevice& kept, Ask ask) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const bool keep = dev >= 0 && dev < MAX_DEVICES;
  if (keep)
    if (const int n = kept.v[dev].load(std::memory_order_acquire)) return n;
  const int n = ask(dev);
  if (keep && n) kept.v[dev].store(n, std::memory_order_release);
  return n;
}

// SMs of the current device
inline int device_sms() {
  static PerDevice kept;
  const int n = per_device(kept, [](int dev) {
    int sms = 0;
    return cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess ? sms : 0;
  });
  return n > 0 ? n : 148;
}

// CTAs of a kernel that fit on an SM of the current device with smem bytes of dynamic shared
// memory, which the device is asked to grant; 0 where it refuses.  kept: a kernel's own.
template <typename K>
int ctas_per_sm(PerDevice& kept, K kernel, int threads, size_t smem) {
  return per_device(kept, [&](int) {
    int n = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) != cudaSuccess || n < 1) n = 1;
    return n;
  });
}

}  // namespace chfem
