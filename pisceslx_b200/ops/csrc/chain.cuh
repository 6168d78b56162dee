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

// Kernels of small blocks come in two kinds, chained and not, since the two instructions alone cost a block most of a
// microsecond.  Up to one block per SM they are chained: more of them, started while the kernel before runs, are put on
// whichever SMs have room, several to one, and stay there.  Norm of 500 rows of 4096 5.1 us unchained and 7.1 chained, of 8192
// rows of 64 6.7 and 9.3, of 148 rows of 4096 3.2 and 2.9; keys and values of 16384 tokens 10.0 and 17.8.
constexpr int64_t kChainBlocks = 148;

template <bool CHAIN>
__device__ __forceinline__ void chain_start() {
  if (CHAIN) {
    chain_next();
    chain_wait();
  }
}

template <typename... P, typename... A>
int launch_chained_if(bool chain, void (*chained)(P...), void (*plain)(P...), dim3 grid, dim3 block, size_t smem,
                      cudaStream_t stream, A&&... args) {
  if (chain) return launch_chained(chained, grid, block, smem, stream, 0, static_cast<A&&>(args)...);
  plain<<<grid, block, smem, stream>>>(static_cast<P>(args)...);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace yv
