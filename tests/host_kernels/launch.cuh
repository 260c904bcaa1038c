// Stands in for csrc/kernels/launch.cuh: a launch runs the grid's blocks one after the other
// under the schedule that is set.
#pragma once
#include "ptx.cuh"
#include PER_DEVICE_HEADER

namespace hostsim {
inline unsigned g_seed = 0;
inline int g_starved = -1, g_drop = -1;
inline std::string g_error;
}  // namespace hostsim

namespace mb200 {
static inline void dep_wait() {}
static inline void dep_launch() {}

template <typename... P, typename... A>
static cudaError_t launch_dep(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem_bytes,
                              cudaStream_t, A&&... args) {
  if (smem_bytes == 0) return cudaSuccess;   // no pipeline to check
  if (smem_bytes > 48 * 1024 &&
      (size_t)hostsim::g_allowed[{(const void*)kernel, hostsim::g_device}] < smem_bytes) {
    hostsim::g_error = "the kernel may not use that much shared memory on this device";
    return cudaErrorInvalidValue;
  }
  gridDim.x = grid.x;
  for (unsigned z = 0; z < grid.z; ++z)
    for (unsigned y = 0; y < grid.y; ++y)
      for (unsigned x = 0; x < grid.x; ++x) {
        blockIdx.x = x;
        blockIdx.y = y;
        blockIdx.z = z;
        const std::string e = hostsim::run_block(block.x / 32, hostsim::g_seed, hostsim::g_starved,
                                                 hostsim::g_drop, [&] { kernel(args...); });
        if (!e.empty()) {
          hostsim::g_error = "block " + std::to_string(x) + "," + std::to_string(y) + ": " + e;
          return cudaErrorUnknown;
        }
      }
  return cudaSuccess;
}
}  // namespace mb200
