// Layer normalisation over the last dimension (norm.cu).
#pragma once
#include <cuda_runtime.h>

namespace srwm {

struct NormParams {
  const float *x, *gamma, *beta, *dy;
  float *mean, *rstd;    // out of the forward (mean NULL: not wanted), in of the backward
  float *y;              // y, or dx in the backward
  float *part;           // backward: [norm_blocks(rows)][2][D]
  long long rows;
  int D;                 // a multiple of 4, at most 1024
  float eps;
};
int norm_blocks(long long rows);
cudaError_t norm_forward(const NormParams& p, cudaStream_t s);
cudaError_t norm_backward(const NormParams& p, float* dgamma, float* dbeta, cudaStream_t s);

}  // namespace srwm
