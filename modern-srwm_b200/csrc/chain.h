// Launch of a kernel that starts with chained() (common.cuh): it is placed while the kernel in front of it on the stream still
// runs, instead of after that one's last block has left and its memory has been flushed.
#pragma once
#include <cuda_runtime.h>

namespace srwm {

template <typename Params>
inline cudaError_t launch_behind(void (*kern)(Params), const Params& p, dim3 grid, int block, size_t smem, cudaStream_t s) {
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &a;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kern, p);
}

}  // namespace srwm
