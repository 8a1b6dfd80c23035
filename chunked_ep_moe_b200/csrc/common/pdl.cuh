// Programmatic dependent launch: a kernel launched with `launch_behind` may become resident while its predecessor on the stream
// is still running, and waits inside for the predecessor to end. For chains of kernels that are shorter than a launch.
#pragma once

#include <cuda_runtime.h>

namespace cem {

// Behind this line everything the predecessor stored is visible. (Nothing to wait for in an ordinary launch.)
__device__ __forceinline__ void wait_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The successor may become resident from here on.
__device__ __forceinline__ void release_successor() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... Params, typename... Args>
void launch_behind(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(block));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// `launch_behind` if `behind`, else an ordinary launch.
template <typename... Params, typename... Args>
void launch_maybe_behind(bool behind, void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t stream,
                         Args&&... args) {
  if (behind) launch_behind(kernel, grid, block, smem, stream, args...);
  else kernel<<<grid, block, smem, stream>>>(args...);
}

}  // namespace cem
