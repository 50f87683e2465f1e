// The part of an agent's block that follows the recurrence, for few rows (block.cu).
#pragma once
#include <cuda_runtime.h>

namespace srwm {

// h = res + att wo^T;  y = relu(norm(h) w1^T + b1) w2^T + b2;  rows dense, weights [out][in]; b1, b2 may be null.
struct BlockParams {
  const float *att, *res, *wo, *gamma, *beta, *w1, *b1, *w2, *b2;
  float* y;
  int rows, K0, D, F, N;   // widths of att, of h, of the hidden row, of y
  float eps;
};
#ifndef SRWM_DEBUG_CHECKS
static_assert(sizeof(BlockParams) % 8 == 0, "arguments of a launch");
#endif

bool block_fits(int K0, int D, int F, int N);              // the kernel can run
bool block_pays(int rows, int K0, int D, int F, int N);    // ... and is faster than its parts
cudaError_t block_launch(const BlockParams& p, cudaStream_t s);

}  // namespace srwm
