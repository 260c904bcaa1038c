// Kernel launches that may begin before the kernel ahead of them in the stream has ended.
//
// A kernel launched with launch_dep() may be set up on the SMs as soon as its predecessor's
// blocks have ended; it calls dep_wait() before its first access to global memory (operands,
// results, dynamic row counts -- kernel parameters and tensor maps are no such access), which
// returns once every kernel before it in the stream has completed and its writes are visible.
// Every thread that touches global memory calls it itself, and no thread returns before it.
//
// dep_launch() lets the successor in earlier, while blocks still run.  Only the short kernel
// ahead of the attention backward does that: in the others the waiting blocks took more than
// they gave (RMSNorm forward and backward of 8192x4096 72.5 us with it, 69.0 without; attention
// of 5 row blocks 44.6 and 41.6; linear layer on 1000 tokens 53.6 and 52.8).  A kernel that
// waits for flags which another kernel on this GPU may have to raise must not call it: the
// successor's blocks would hold SM resources that the other kernel needs.
//
// Against plain launches: linear layer 200x256x768, three products, 27.8 -> 25.0 us; 2048 -> 3072
// on 1000 tokens 57.4 -> 52.8; attention of 5 row blocks, four kernels, 49.8 -> 41.6.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "per_device.cuh"

namespace mb200 {

__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_launch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... P, typename... A>
static inline cudaError_t launch_dep(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                                     cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace mb200
