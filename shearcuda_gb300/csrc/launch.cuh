// Programmatic dependent launches: every kernel of a call's chain starts with
// pdl_sync() and is launched with launch_pdl, so that a launch is set up while
// the kernel before it still runs and only waits for its results.  A chain of
// small kernels otherwise pays the whole of a launch's latency at every step:
// one denoise of 256 x 256 (ten kernels) 101 -> 85 us, one volume of 96^3 (51)
// 373 -> 260 us, inverse_shear at 512 x 512 147 -> 102 us.  The kernels do not
// let their dependents be placed earlier than at their own end: CTAs that wait
// in the SMs' slots cost more (96 and 293 us in the first two).
#pragma once
#include <cuda_runtime.h>

namespace nsst {

// First statement of a kernel: waits until the kernel before it has ended and
// its writes are visible.
// Nothing that another kernel reads or writes may be touched before it.
__device__ __forceinline__ void pdl_sync() {
  cudaGridDependencySynchronize();
}

// kernel<<<grid, block, smem, st>>>(args...) as a dependent launch; the kernel
// must begin with pdl_sync().
template <class... P, class... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace nsst
