// rg_launch.cuh -- launches of the kernels a step chains on one stream.
//
// A step is two to eleven kernels of 5 to 200 us, each reading what the one
// before it wrote, and the gap between two of them (the drain of one grid, the
// launch of the next: 2.2 to 2.8 us) was a tenth of a 512^2 FP32-mixed step and
// half of an 8,000-cell one.  chain() launches with programmatic stream
// serialization: the next grid is set up as the one before ends, and every such
// kernel starts with chain_wait(), which returns when the grids before it in the
// stream have completed and their writes are visible.  Nothing else changes: the
// kernels still run one after another.  No kernel triggers the next one's launch
// itself: blocks set up earlier go to whichever SMs have room then, and the
// uneven spread cost more than the last half microsecond saved (FP64 adjoint at
// 256^2 8.28 against 7.56 ms, Sedov 512^2 FP64 3.89 against 3.69 ms).
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

namespace rg {

#ifdef __CUDACC__
// First statement of every kernel that chain() launches (a no-op in a launch
// without the attribute): wait for the grids before this one.
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... P>
inline cudaError_t chain(cudaStream_t s, long long grid, int block, void (*kernel)(P...),
                         std::common_type_t<P>... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(block));
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
#endif

}  // namespace rg
