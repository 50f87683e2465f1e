// Output projection with its residual, layer norm and the two linear maps of the feed-forward part behind it
// (reinforcement_learning/torchbeast/layer.py:340-421 and :30-47, one step of a few dozen actors) as one kernel.
//
// Rows are independent, so a cluster of eight CTAs takes eight rows through all of it: each CTA has an eighth of the columns of a
// product, whose weights it asks for at its start (160 KB with rows of 256 and a hidden row of 512), and writes its results into
// the shared memory of all eight, where the next product finds whole rows.  A warp works on four columns and the eight rows at a
// time, its lanes on four values of k each; the 32 sums are reduced so that each lane ends with one, and the four lanes of a row write
// its four columns to two CTAs each.
//
// Bound: latency.  Of 17 thousand cycles with 48 rows of 256, asking for the weights takes 3.4, the three products 2.1, 4.2 and 3
// (their reads of shared memory, and a thousand each for the last sums), the norm 1, the cluster's barriers 1.4 each.  The four kernels
// that it replaces each wait for all of the one in front.  Tried: weights straight to registers, 9.2 against 9.6 us but 6.1
// against 5.1 with rows of 64; bulk copies 9.4; clusters of 16, 8.4, of which only four run at once; sixteen warps, slower.
#include "block.h"

#include "common.cuh"
#include "device.h"

namespace srwm {
namespace {

constexpr int CL = 8, R = 8, WARPS = 8;   // CTAs of a cluster, its rows, warps of a CTA
constexpr int GROUPS = CL * WARPS;        // groups of four columns the cluster's warps take at a time
constexpr int MAX_SMEM = 220 * 1024;

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Four columns of a row to the same place in all CTAs: v is lane's own one (column lane % 4), place the first one's.
__device__ __forceinline__ void to_all(float* place, float v, int lane) {
  float4 x;
  x.x = __shfl_sync(0xffffffffu, v, lane & ~3);
  x.y = __shfl_sync(0xffffffffu, v, (lane & ~3) + 1);
  x.z = __shfl_sync(0xffffffffu, v, (lane & ~3) + 2);
  x.w = __shfl_sync(0xffffffffu, v, (lane & ~3) + 3);
  const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(place));
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    uint32_t b;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(lane % 4 + 4 * i));
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(b), "f"(x.x), "f"(x.y), "f"(x.z), "f"(x.w) : "memory");
  }
}
// The sums of (row, column) = (lane / 4, lane % 4) over K values: four columns of w, eight rows of x.
__device__ __forceinline__ float sums(const float* w, const float* x, int pitch, int K, int lane) {
  u64 acc[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0ull;
#pragma unroll 1
  for (int k = lane * 4; k < K; k += 128) {
    ulonglong2 v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = *reinterpret_cast<const ulonglong2*>(w + c * K + k);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(x + r * pitch + k);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        acc[r][c] = fma2<true>(a.x, v[c].x, acc[r][c]);
        acc[r][c] = fma2<true>(a.y, v[c].y, acc[r][c]);
      }
    }
  }
  __syncwarp();
  float s[4 * R];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) s[4 * r + c] = hsum2(acc[r][c]);
  reduce_scatter<4 * R, 32, 1>(s, lane);
  return s[0];
}
// Layer norm of a row of D values in shared memory, by a warp.
__device__ __forceinline__ void norm_row(float* x, const float* gamma, const BlockParams& p, int lane) {
  const float inv_d = 1.f / (float)p.D, *beta = gamma + p.D;
  float s = 0.f, q = 0.f;
#pragma unroll 2
  for (int k = lane * 4; k < p.D; k += 128) {
    const float4 v = *reinterpret_cast<const float4*>(x + k);
    s += (v.x + v.y) + (v.z + v.w);
  }
  const float mean = allreduce_warp(s) * inv_d;
#pragma unroll 2
  for (int k = lane * 4; k < p.D; k += 128) {
    const float4 v = *reinterpret_cast<const float4*>(x + k);
    const float d[4] = {v.x - mean, v.y - mean, v.z - mean, v.w - mean};
    q += (d[0] * d[0] + d[1] * d[1]) + (d[2] * d[2] + d[3] * d[3]);
  }
  const float rstd = rsqrtf(allreduce_warp(q) * inv_d + p.eps);
#pragma unroll 2
  for (int k = lane * 4; k < p.D; k += 128) {
    const float4 v = *reinterpret_cast<const float4*>(x + k), a = *reinterpret_cast<const float4*>(gamma + k),
                 o = *reinterpret_cast<const float4*>(beta + k);
    *reinterpret_cast<float4*>(x + k) = make_float4(fmaf((v.x - mean) * rstd, a.x, o.x), fmaf((v.y - mean) * rstd, a.y, o.y),
                                                    fmaf((v.z - mean) * rstd, a.z, o.z), fmaf((v.w - mean) * rstd, a.w, o.w));
  }
}

__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(32 * WARPS, 1) block_kernel(const BlockParams p) {
  extern __shared__ __align__(16) float smem[];
  const int pa = p.K0 + 4, ph = p.D + 4, pf = p.F + 4;
  // rows of att, of h (then normalised), hidden; gamma and beta; weights
  float *sa = smem, *sh = sa + R * pa, *sf = sh + R * ph, *sg = sf + R * pf, *sw = sg + 2 * p.D;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int first = warp * CL + blockIdx.x % CL;   // this warp's groups of columns: first, first + GROUPS, ...
  const int r = lane / 4, c = lane % 4, row = blockIdx.x / CL * R + r;
  chained();
  cluster_arrive();   // (the others' shared memory is there once they have come here)
  // A warp copies its own weights, product after product (a group at its end may not be there), and a row.
  {
    const int q = blockIdx.x / CL * R + warp;
    for (int k = lane * 4; k < p.K0; k += 128) {
      if (q < p.rows) cp_async16(sa + warp * pa + k, p.att + (long long)q * p.K0 + k);
      else *reinterpret_cast<float4*>(sa + warp * pa + k) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int k = (int)threadIdx.x * 4; k < 2 * p.D; k += 128 * WARPS) cp_async16(sg + k, k < p.D ? p.gamma + k : p.beta + (k - p.D));
    float* to = sw;
#pragma unroll 1
    for (int s = 0; s < 3; ++s) {
      const float* W = s == 0 ? p.wo : (s == 1 ? p.w1 : p.w2);
      const int K = s == 0 ? p.K0 : (s == 1 ? p.D : p.F), N = s == 0 ? p.D : (s == 1 ? p.F : p.N);
      for (int g0 = 0; g0 * 4 < N; g0 += GROUPS, to += WARPS * 4 * K)
        if ((g0 + first) * 4 < N)   // the four columns lie behind one another
          for (int k = lane * 4; k < 4 * K; k += 128) cp_async16(to + warp * 4 * K + k, W + (long long)(g0 + first) * 4 * K + k);
      cp_async_commit();
    }
  }
  float b = row < p.rows && first * 4 < p.D ? p.res[(long long)row * p.D + first * 4 + c] : 0.f;
  cp_async_wait<2>();
  __syncthreads();
  // The products one after the other in the same code: a kernel of a few microseconds waits for its instructions too.
  const float *add = p.res + (long long)row * p.D, *x = sa, *w = sw + warp * 4 * p.K0;
  bool on = row < p.rows;   // whether there is something to add
  int K = p.K0, N = p.D;
#pragma unroll 1
  for (int stage = 0; stage < 3; ++stage) {
    cluster_wait();
    if (stage == 1) {
      if (warp < R) norm_row(sh + warp * ph, sg, p, lane);
      __syncthreads();
    }
#pragma unroll 1
    for (int g = first; g - first < (N + 3) / 4; g += GROUPS, w += WARPS * 4 * K) {
      if (g * 4 >= N) continue;
      if (g != first) b = on ? add[g * 4 + c] : 0.f;
      float v = sums(w, x, K + 4, K, lane) + b;
      if (stage == 1 && v < 0.f) v = 0.f;
      if (stage < 2) to_all((stage == 0 ? sh + r * ph : sf + r * pf) + g * 4, v, lane);
      else if (row < p.rows) p.y[(long long)row * p.N + g * 4 + c] = v;
    }
    if (stage == 2) break;
    add = stage == 0 ? p.b1 : p.b2;
    on = add != nullptr;
    w += warp * 4 * (N - K);   // (this warp's place among those of the next product)
    x = stage == 0 ? sh : sf;
    K = N;
    N = stage == 0 ? p.F : p.N;
    b = on && first * 4 < N ? add[first * 4 + c] : 0.f;
    if (stage == 0) cp_async_wait<1>();
    else cp_async_wait<0>();
    __syncwarp();
    cluster_arrive();
  }
}

}  // namespace

static size_t smem_bytes(int K0, int D, int F, int N) {
  auto weights = [](size_t n, size_t k) { return (n + 4 * GROUPS - 1) / (4 * GROUPS) * (4 * WARPS) * k; };   // of a CTA
  return ((size_t)R * (K0 + D + F + 12) + 2 * (size_t)D + weights(D, K0) + weights(F, D) + weights(N, F)) * 4;
}

bool block_fits(int K0, int D, int F, int N) {
  return K0 % 4 == 0 && D % 4 == 0 && F % 4 == 0 && N % 4 == 0 && smem_bytes(K0, D, F, N) <= (size_t)MAX_SMEM;
}
// While the clusters run at once (8 CTAs of a GPC each; 14 of them did, 16 took a second round).  us, four kernels / one, launches
// behind one another, rows x width (hidden row twice as wide):
//   48 x 64: 7.3 / 5.1, 48 x 128: 8.4 / 6.2, 48 x 256: 11.9 / 9.6, 112 x 256: 15.6 / 9.7, 128 x 256: 15.3 / 18.1, 160 x 64: 7.3 / 9.4
// Two layers of 48 actors, hidden size 256, as a captured graph: 39.3 -> 34.1 us.
bool block_pays(int rows, int K0, int D, int F, int N) {
  return rows > 0 && (rows + R - 1) / R <= common_sms() / 10 && block_fits(K0, D, F, N);
}

cudaError_t block_launch(const BlockParams& p, cudaStream_t s) {
  static unsigned long long ready = 0;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(__atomic_load_n(&ready, __ATOMIC_ACQUIRE) & bit)) {
    e = cudaFuncSetAttribute(block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM);
    if (e != cudaSuccess) return e;
    __atomic_fetch_or(&ready, bit, __ATOMIC_RELEASE);
  }
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)((p.rows + R - 1) / R * CL));
  c.blockDim = dim3(32 * WARPS);
  c.dynamicSmemBytes = smem_bytes(p.K0, p.D, p.F, p.N);
  c.stream = s;
  c.attrs = &a;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, block_kernel, p);
}

}  // namespace srwm
