// What a process finds out or sets up once per GPU that it uses: a kernel's opt-in to more than
// 48 KB of shared memory, the SM count and cluster capacities belong to one device.
#pragma once
#include <cuda_runtime.h>

namespace mb200 {

constexpr int kMaxDevices = 64;

template <typename T>
struct PerDevice {
  T v[kMaxDevices] = {};
  // the entry of device `dev`, or null when there is none to keep (nothing is remembered then)
  T* at(int dev) { return dev >= 0 && dev < kMaxDevices ? &v[dev] : nullptr; }
};
static inline int current_device() {
  int dev = -1;
  return cudaGetDevice(&dev) == cudaSuccess ? dev : -1;
}

// Lets `kernel` use `bytes` of dynamic shared memory on the current device, which is `dev`.
// `done` is this kernel's own; setting the attribute twice from two threads does no harm.
template <typename F>
static inline cudaError_t allow_smem(F* kernel, int bytes, PerDevice<int>& done,
                                     int dev = current_device()) {
  int* have = done.at(dev);
  if (have && *have >= bytes) return cudaSuccess;
  const cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && have) *have = bytes;
  return e;
}

}  // namespace mb200
