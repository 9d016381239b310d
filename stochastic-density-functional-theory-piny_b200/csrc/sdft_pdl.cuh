// sdft_pdl.cuh -- programmatic dependent launch of the kernels of one H
// application.
//
// A kernel launched with launch_pdl may start while the kernel before it in
// the stream still runs (from the moment all of that kernel's CTAs have called
// pdl_trigger or ended): its CTAs set themselves up -- barriers, TMEM, tables
// and operands that no kernel of the chain writes -- and then wait in pdl_wait
// until that kernel is complete and its writes are visible.  So every kernel
// launched this way calls pdl_wait, in every thread, before it touches anything
// an earlier kernel writes, or writes anything an earlier kernel touches; each
// then also stands for all kernels before it.
#pragma once
#include <cuda_runtime.h>

namespace sdft {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// early = false: an ordinary launch, which starts when the kernel before it is
// complete (pdl_wait then returns at once).
template <typename... KA, typename... A>
inline cudaError_t launch_pdl(bool early, void (*k)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                              A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, KA(args)...);
}

}  // namespace sdft
