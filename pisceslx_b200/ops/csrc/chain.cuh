// Launches that overlap the start of a kernel with the end of the one before it in the stream (programmatic dependent
// launch).  A decoding step is a chain of kernels of a few microseconds, of which starting up is a good part: barriers, tensor
// memory, tensor maps, the first bytes of the weights.
//
// A kernel launched by launch_chained calls chain_wait() in every thread before it reads or writes anything that another kernel
// touches; what it does before that may read its own parameters alone (fetching weights into the L2 is harmless: the L2 is where
// all writes meet).  chain_next() lets the next kernel of the stream begin once every block has called it; the next kernel's own
// chain_wait() still waits until this one has finished.  A block that holds tensor memory calls it after its allocation, or the
// next kernel could take what this one needs.  Kernels launched without the attribute wait for the whole kernel, as ever.
#pragma once
#include <cuda_runtime.h>

namespace yv {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
int launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 1;
  if (cluster > 0) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  cfg.attrs = attr;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

}  // namespace yv
