// Launches that overlap the kernel before them on the stream (internal).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace gpjb {

// Launches `kernel` so that its CTAs may start while the kernel before it on
// `stream` still runs, once all of that kernel's CTAs have executed
// griddepcontrol.launch_dependents or ended: the launch and the prologue cost
// no time of their own (about 2 us a launch).  The kernel executes
// griddepcontrol.wait before it touches anything an earlier kernel writes or
// reads.  After anything but a kernel this is a plain launch.
template <typename... Params, typename... Args>
cudaError_t launch_overlapped(void (*kernel)(Params...), uint32_t grid, uint32_t block,
                              size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(grid);
  config.blockDim = dim3(block);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attr;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, Params(args)...);
}

}  // namespace gpjb
