// Launch helpers: programmatic dependent launch, the shared-memory opt-in and
// the SM count the launch rules use.
#pragma once

#include <cuda_runtime.h>

namespace agb {

constexpr int kSMs = 152;

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// launch with programmatic stream serialisation: the kernel may start while
// the previous kernel in the stream finishes and waits in griddepcontrol.wait
template <class... P, class... A>
inline cudaError_t launch_pdl(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

// Opt a kernel in to as much dynamic shared memory as the device grants
// beside the kernel's static use.  The same value on every call: launches of
// one kernel with different sizes from several threads do not disturb each
// other.
template <class... P>
inline cudaError_t allow_max_smem(void (*k)(P...)) {
  int dev = 0, limit = 0;
  cudaFuncAttributes at{};
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, k);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, limit - (int)at.sharedSizeBytes);
  return e;
}

}  // namespace agb
