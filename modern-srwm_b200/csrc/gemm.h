// fp32 matrix products of the layers' linear maps (gemm.cu).
#pragma once
#include <cuda_runtime.h>

namespace srwm {

// C[m][n] = sum_k a(m, k) b(n, k) (+ add[m][n]);  a(m, k) = A[m lda + k], or A[k lda + m] with trans_a; b likewise.
struct GemmParams {
  const float *A, *B, *add;
  float* C;
  long long lda, ldb, ldc, ldadd;
  int M, N, K;
  int kpart;          // values of k per part; the parts' C lie M * N floats apart
  int units;          // pairs of tiles x parts
  bool relu;          // negative results become zero (few rows only)
  unsigned* gave_up;  // host memory: set by a kernel that has given up waiting (NULL: none)
#ifdef SRWM_DEBUG_CHECKS
  int tries;          // of each wait
#endif
};
#ifndef SRWM_DEBUG_CHECKS
// A launch takes the host 0.3 us less where the arguments are a multiple of 32 bytes (few-row product through torch: 3.5 us
// with 96 bytes, 4.0 with 80 or 104).
static_assert(sizeof(GemmParams) == 96, "arguments of a launch");
#endif

// Parts the sum over k is cut into; with more than one, scratch of [parts][M][N] floats, and C and add dense.
int gemm_parts(int M, int N, int K);
cudaError_t gemm_launch(const GemmParams& p, bool trans_a, bool trans_b, float* scratch, cudaStream_t s);
bool gemm_is_skinny(int M, int N, int K);
cudaError_t gemm_skinny_launch(const GemmParams& p, bool trans_a, bool trans_b, cudaStream_t s);
unsigned gemm_timeouts();
// Whether a kernel has given up since the last time this was asked; waits for nothing.
bool gemm_gave_up();
#ifdef SRWM_DEBUG_CHECKS
extern int gemm_tries;
#endif

}  // namespace srwm
