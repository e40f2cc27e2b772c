// Kernel launches with the programmatic-serialization attribute: the kernel's blocks may start, and set themselves up, while the
// kernel before it in the stream still runs. Only for kernels whose every thread executes `pdl_wait()` before it touches anything
// that a predecessor wrote, or ends. `launch_early` sets the attribute while `cosmos::early_on()` (unless the caller wants no
// overlap), for kernels that neither wait for a peer nor read a weight before that point; `launch_pdl` while `cosmos::pdl_on()`.
#pragma once
#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

#include "kernels.h"

namespace cosmos {

template <typename... KArgs, typename... Args>
inline void launch_with(bool early, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                        Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = early ? 1 : 0;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
  if (err != cudaSuccess) throw std::runtime_error(std::string("kernel launch failed: ") + cudaGetErrorString(err));
}
template <typename... KArgs, typename... Args>
inline void launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  launch_with(pdl_on(), kern, grid, block, smem, stream, args...);
}
template <typename... KArgs, typename... Args>
inline void launch_early(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  launch_with(early_on(), kern, grid, block, smem, stream, args...);
}

}  // namespace cosmos
