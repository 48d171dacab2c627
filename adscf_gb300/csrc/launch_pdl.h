// launch_pdl.h -- kernel launch with programmatic stream serialisation.
#pragma once
#include <cuda_runtime.h>

#include <utility>

// Launch with programmatic stream serialisation: the kernel may start while
// the previous kernel on the stream finishes; the TMA passes wait for it
// (griddepcontrol.wait) before they touch its output.
template <typename... KArgs, typename... Args>
inline void launch_pdl(void (*kern)(KArgs...), dim3 grid, int block, size_t smem, cudaStream_t s,
                Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}
