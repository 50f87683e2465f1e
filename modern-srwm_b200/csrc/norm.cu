// Layer normalisation of the layers (supervised_learning/layer.py:68, :150), fp32, forward and backward.
//
// Bound by HBM: one read of x (and of dy) and one write of y (dx).  A warp takes a row at a time, its lanes four
// columns in turn, the row stays in registers between the statistics and the result.  The gradients of
// weight and bias are kept per lane over all rows of a warp, added over the block and written once per block;
// a second launch adds the blocks, in a fixed order.  16384 x 512 forward + backward: 52 us, 174 with the
// library's kernels, whose weight-gradient pass alone took 127.
#include "norm.h"

#include <type_traits>

#include "chain.h"
#include "common.cuh"
#include "device.h"

namespace srwm {
namespace {

constexpr int WARPS = 8;

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// NV: pieces of four columns per lane (D <= 128 NV)
template <int NV>
__global__ void __launch_bounds__(32 * WARPS) norm_fwd_kernel(const NormParams p) {
  chained();
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const float inv_d = 1.f / (float)p.D;
  for (long long row = (long long)blockIdx.x * WARPS + warp; row < p.rows; row += (long long)gridDim.x * WARPS) {
    float4 v[NV];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (i * 32 + lane) * 4;
      v[i] = c < p.D ? ld4(p.x + row * p.D + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
    }
    const float mean = allreduce_warp(s) * inv_d;
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if ((i * 32 + lane) * 4 >= p.D) continue;
      v[i].x -= mean; v[i].y -= mean; v[i].z -= mean; v[i].w -= mean;
      q += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
    }
    const float rstd = rsqrtf(allreduce_warp(q) * inv_d + p.eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (i * 32 + lane) * 4;
      if (c >= p.D) continue;
      const float4 w = ld4(p.gamma + c), b = ld4(p.beta + c);
      *reinterpret_cast<float4*>(p.y + row * p.D + c) =
          make_float4(fmaf(v[i].x * rstd, w.x, b.x), fmaf(v[i].y * rstd, w.y, b.y), fmaf(v[i].z * rstd, w.z, b.z),
                      fmaf(v[i].w * rstd, w.w, b.w));
    }
    if (lane == 0 && p.mean != nullptr) {
      p.mean[row] = mean;
      p.rstd[row] = rstd;
    }
  }
}

template <int NV>
__global__ void __launch_bounds__(32 * WARPS) norm_bwd_kernel(const NormParams p) {
  __shared__ __align__(16) float4 part[WARPS][32];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const float inv_d = 1.f / (float)p.D;
  float4 gw[NV], gb[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) gw[i] = gb[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (long long row = (long long)blockIdx.x * WARPS + warp; row < p.rows; row += (long long)gridDim.x * WARPS) {
    const float mean = __ldg(p.mean + row), rstd = __ldg(p.rstd + row);
    float4 xh[NV], g[NV];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (i * 32 + lane) * 4;
      xh[i] = g[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c >= p.D) continue;
      const float4 x = ld4(p.x + row * p.D + c), d = ld4(p.dy + row * p.D + c), w = ld4(p.gamma + c);
      xh[i] = make_float4((x.x - mean) * rstd, (x.y - mean) * rstd, (x.z - mean) * rstd, (x.w - mean) * rstd);
      gw[i].x = fmaf(d.x, xh[i].x, gw[i].x); gw[i].y = fmaf(d.y, xh[i].y, gw[i].y);
      gw[i].z = fmaf(d.z, xh[i].z, gw[i].z); gw[i].w = fmaf(d.w, xh[i].w, gw[i].w);
      gb[i].x += d.x; gb[i].y += d.y; gb[i].z += d.z; gb[i].w += d.w;
      g[i] = make_float4(d.x * w.x, d.y * w.y, d.z * w.z, d.w * w.w);
      s1 += (g[i].x + g[i].y) + (g[i].z + g[i].w);
      s2 += (g[i].x * xh[i].x + g[i].y * xh[i].y) + (g[i].z * xh[i].z + g[i].w * xh[i].w);
    }
    const float c1 = allreduce_warp(s1) * inv_d, c2 = allreduce_warp(s2) * inv_d;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (i * 32 + lane) * 4;
      if (c >= p.D) continue;
      *reinterpret_cast<float4*>(p.y + row * p.D + c) =
          make_float4(rstd * (g[i].x - c1 - xh[i].x * c2), rstd * (g[i].y - c1 - xh[i].y * c2),
                      rstd * (g[i].z - c1 - xh[i].z * c2), rstd * (g[i].w - c1 - xh[i].w * c2));
    }
  }
  float* out = p.part + (long long)blockIdx.x * 2 * p.D;
#pragma unroll
  for (int i = 0; i < 2 * NV; ++i) {
    __syncthreads();
    part[warp][lane] = i < NV ? gw[i % NV] : gb[i % NV];
    __syncthreads();
    const int c = ((i % NV) * 32 + lane) * 4;
    if (warp == 0 && c < p.D) {
      float4 t = part[0][lane];
#pragma unroll
      for (int w = 1; w < WARPS; ++w) {
        const float4 o = part[w][lane];
        t.x += o.x; t.y += o.y; t.z += o.z; t.w += o.w;
      }
      *reinterpret_cast<float4*>(out + (i < NV ? 0 : p.D) + c) = t;
    }
  }
}

// The [2][D] sums over the blocks' parts: 32 columns a CTA, eight slices of the blocks
__global__ void __launch_bounds__(256) norm_parts_kernel(const float* part, int blocks, int D, float* dgamma, float* dbeta) {
  __shared__ float s[8][33];
  const int col = threadIdx.x % 32, slice = threadIdx.x / 32, c = blockIdx.x * 32 + col;
  float t = 0.f;
  if (c < 2 * D) {
#pragma unroll 4
    for (int b = slice; b < blocks; b += 8) t += part[(long long)b * 2 * D + c];
  }
  s[slice][col] = t;
  __syncthreads();
  if (slice != 0 || c >= 2 * D) return;
#pragma unroll
  for (int k = 1; k < 8; ++k) t += s[k][col];
  if (c < D) dgamma[c] = t;
  else dbeta[c - D] = t;
}

template <typename F>
cudaError_t by_width(int D, F f) {
  if (D <= 128) return f(std::integral_constant<int, 1>());
  if (D <= 256) return f(std::integral_constant<int, 2>());
  if (D <= 512) return f(std::integral_constant<int, 4>());
  return f(std::integral_constant<int, 8>());
}

}  // namespace

// Backward: four blocks of eight warps per multiprocessor (two at a time at D = 512, whose rows and sums take 95 registers a
// thread), each a part to be added up; fewer rows, fewer blocks
int norm_blocks(long long rows) {
  const long long b = (rows + WARPS - 1) / WARPS, most = 4 * common_sms();
  return (int)(b < most ? b : most);
}
cudaError_t norm_forward(const NormParams& p, cudaStream_t s) {
  const long long blocks = (p.rows + WARPS - 1) / WARPS, most = 16 * common_sms();
  const int grid = (int)(blocks < most ? blocks : most);
  return by_width(p.D, [&](auto nv) {
    return launch_behind(norm_fwd_kernel<decltype(nv)::value>, p, grid, 32 * WARPS, 0, s);
  });
}
cudaError_t norm_backward(const NormParams& p, float* dgamma, float* dbeta, cudaStream_t s) {
  const int grid = norm_blocks(p.rows);
  const cudaError_t e = by_width(p.D, [&](auto nv) {
    norm_bwd_kernel<decltype(nv)::value><<<grid, 32 * WARPS, 0, s>>>(p);
    return cudaGetLastError();
  });
  if (e != cudaSuccess) return e;
  norm_parts_kernel<<<(2 * p.D + 31) / 32, 256, 0, s>>>(p.part, grid, p.D, dgamma, dbeta);
  return cudaGetLastError();
}

}  // namespace srwm
