// chain.cuh -- launches of a chain of short dependent kernels on one stream
// (programmatic dependent launch): a kernel's CTAs may start, set up barriers,
// tensor memory and addresses, while the previous kernel still runs, and wait in
// chain_wait for its results.  Every kernel of a chain calls chain_start at its
// beginning and chain_wait in all threads that touch global memory, before they do:
// each then completes after its predecessor, and so after all before it.  Launched
// any other way both calls do nothing.  The network's gradient is 17 kernels of 3 to
// 24 us in a row: 153 us with plain launches, 137 us with these; a 256 x 256 x 256
// product repeated, 5.6 -> 4.9 us.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace espec {

// the next kernel may start once all CTAs of this one have
__device__ __forceinline__ void chain_start() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// the previous kernel is complete and its writes are visible
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                           cudaStream_t st, A&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// Kernels of little work per CTA come in two forms: the two calls take a CTA as long as
// a few hundred of its loads, and beyond kChainMaxCtas CTAs that is more than the overlap
// gains (to_bf16 of 1 M values, 4096 CTAs: 5.0 us chained, 5.8 plain; 2 M 9.2 and 7.3, 16 M
// 68 and 43).  The plain form makes neither call and is launched without the attribute: it
// starts after everything before it, and a chained kernel after it waits for all of it.
constexpr long kChainMaxCtas = 4096;
template <class... P, class... A>
cudaError_t launch_either(void (*chained)(P...), void (*plain)(P...), dim3 grid, dim3 block,
                          cudaStream_t st, A... args) {
  if ((long)grid.x * grid.y * grid.z <= kChainMaxCtas)
    return launch_chained(chained, grid, block, 0, st, args...);
  plain<<<grid, block, 0, st>>>(args...);
  return cudaGetLastError();
}

}  // namespace espec
