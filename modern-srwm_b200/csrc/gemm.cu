// fp32 matrix products of the layers' linear maps (out_linear, slow_net and their gradients) on the
// 5th-generation tensor cores:  C[M, N] = op(A) op(B)^T (+ add).
//
// Finite fp32 operands are cut into three bf16 pieces, exactly (mma.cuh), and the six products of pieces down to
// 2^-16 of the leading one are summed in fp32, the leading one and the rest in accumulators of their own.
// An infinite one has no such pieces: all outputs it reaches come out as NaN.  The drains look for NaN, and a tile with one
// sums its NaN outputs again on the fp32 pipe (sum_again), where infinities are what arithmetic makes of them.
// 16384 x 512 x 512: 80 us, 123 with an infinity in A, 540 with one in B (a column of every tile), 166 with NaN everywhere.
// The tensor cores' accumulators round towards zero, one unit in 2^24 per 16 values of k, which adds up in one
// direction; so every 256 values of k (512 in sums longer than that) they are emptied into C, whose additions
// round to nearest.  Error of the result, 2-norm, normal inputs: 2.8e-7 at k = 512, 5e-7 beyond, against 4.1e-7
// and 7e-7 of the library's fp32 product.
//
// 128 x 128 tiles, 32 values of k a stage.  Eight warps of a CTA read the fp32 tiles a stage ahead into registers, cut
// them and store the pieces in the no-swizzle K-major layout (8 x 16-byte core matrices), two stages deep; a ninth
// issues twelve tcgen05.mma (128 x 128 x 16) a stage, accumulators in tensor memory (256 columns).  Stages are handed
// over through mbarriers.  Two CTAs share a multiprocessor.
//
// Bound: cutting (some 340 warp instructions a warp and stage, 680 issue cycles for eight warps) beside the tensor cores
// (768).  16384 x 512 x 512: 73 us, the library's fp32 product on the fp32 pipe 174.  On the way here: products issued
// by one of the cutting warps, for which the others waited, 101 us; stages of 16 values, whose loads read half lines, 85;
// drains through registers (loads of C and stores, 7300 cycles each) 78, and from tensor memory straight to rows of C,
// a row a lane, 93.
#include "gemm.h"

#include <atomic>
#include <mutex>

#include "chain.h"
#include "device.h"
#include "mma.cuh"

namespace srwm {
namespace {

constexpr int TM = 128, TN = 128, TK = 32, THREADS = 256, STAGES = 2;   // THREADS: those that cut; one warp more issues the products
constexpr int KDRAIN = 256;                       // values of k between two additions to C, or twice as many
constexpr int CORE = 128;                         // bytes of a core matrix: 8 rows x 8 bf16
constexpr int KSTEP = (TM / 8) * CORE + 64;       // from a core matrix to the next along k; along the rows they are adjacent
constexpr int PIECE = (TK / 8) * KSTEP;           // (+ 64: the lanes of a store, 4 rows x 4 core matrices, miss each other's banks)
constexpr int STAGE = 6 * PIECE;                  // three pieces of A and of B
constexpr int CP = TN + 4;                        // floats of a row of the output stage
constexpr int SMEM = STAGES * STAGE;
constexpr int BAR_READ = 1, BAR_CUT = 2;          // named barriers: the accumulators have been read; the cutting warps
static_assert(TM * CP * 4 <= SMEM, "the output stage reuses the operand stages");
static_assert(KDRAIN % (2 * TK) == 0 && (KDRAIN / TK) % (2 * STAGES) == 0, "parities start over with each drain");

// Waits have a limit (none is expected to reach it).  A CTA in which one has given up leaves NaN in its tile of C, counts
// here and sets the caller's word in host memory, at which the next call fails.
constexpr int TRIES = 4000000;
__device__ unsigned g_timeouts;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// K-major, no swizzle: core matrices KSTEP bytes apart along k, CORE bytes apart along the rows
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(KSTEP >> 4) << 16) | ((uint64_t)(CORE >> 4) << 32) |
         ((uint64_t)1 << 46);
}
__device__ __forceinline__ void mma_issue(uint32_t d, uint32_t a, uint32_t b, bool add) {
  constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((TN / 8) << 17) | ((TM / 16) << 24);   // f32 += bf16 bf16
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(operand_desc(a)), "l"(operand_desc(b)),
      "r"(idesc), "r"(add ? 1u : 0u)
      : "memory");
}
__device__ __forceinline__ bool wait_parity(uint32_t bar, uint32_t parity, int tries) {
  for (int i = 0; i < tries; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// One thread's share of a 128 x 32 tile, sixteen values.  T: k is the outer dimension in memory: sixteen values of k of
// one row, rows in adjacent lanes.  Else: four values of k of four rows, eight lanes reading a whole 128-byte line of
// each (with 16 values of k a stage, half lines: the loads took 560 cycles to issue).  Rows beyond the matrix read its
// first row: they end in rows of C that are not stored.
template <bool T>
struct Loader {
  static constexpr int NR = T ? 1 : 4;
  const float* p;              // first row's value at the next stage to be loaded
  long long ld;
  int left, dst;               // values of k from p to the part's end; place of the first row's values
  int step[NR];                // rows from the first one to the others (they may be clamped to the matrix)
  __device__ __forceinline__ Loader(const float* base, long long ld_, int r0, int rows, int k_lo, int k_hi, int tid) : ld(ld_) {
    const int k_of = T ? (tid >> 7) * 16 : (tid & 7) * 4, row = T ? (tid & 127) : tid >> 3;
    left = k_hi - k_lo - k_of;
    const int r = r0 + row < rows ? r0 + row : 0;
#pragma unroll
    for (int i = 0; i < NR; ++i) step[i] = (r0 + row + i * 32 < rows ? r0 + row + i * 32 : 0) - r;
    p = T ? base + (long long)(k_lo + k_of) * ld + r : base + (long long)r * ld + k_lo + k_of;
    dst = (row / 8) * CORE + (k_of / 8) * KSTEP + (row % 8) * 16 + (k_of % 8) * 2;
  }
  __device__ __forceinline__ void load(float (&v)[16]) {   // nothing is read at or beyond the part's end
    if constexpr (T) {
      const float* q = p;
      if (left >= 16) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          v[j] = __ldg(q);
          q += ld;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          v[j] = j < left ? __ldg(q) : 0.f;
          q += ld;
        }
      }
      p += TK * ld;
    } else {
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (left > 0) x = __ldg(reinterpret_cast<const float4*>(p + step[i] * ld));   // K is a multiple of 4
        v[i * 4] = x.x; v[i * 4 + 1] = x.y; v[i * 4 + 2] = x.z; v[i * 4 + 3] = x.w;
      }
      p += TK;
    }
    left -= TK;
  }
  __device__ __forceinline__ void store(unsigned char* st, const float (&v)[16]) const {
    st += dst;
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
      uint32_t q[3][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) split3(v[4 * i + 2 * j], v[4 * i + 2 * j + 1], q[0][j], q[1][j], q[2][j]);
#pragma unroll
      for (int z = 0; z < 3; ++z) {
        if constexpr (T) {   // eight of the row's sixteen
          *reinterpret_cast<uint4*>(st + (i / 2) * KSTEP + z * PIECE) = make_uint4(q[z][0], q[z][1], q[z][2], q[z][3]);
        } else {             // rows 32 apart
          *reinterpret_cast<uint2*>(st + i * 4 * CORE + z * PIECE) = make_uint2(q[z][0], q[z][1]);
          *reinterpret_cast<uint2*>(st + (i + 1) * 4 * CORE + z * PIECE) = make_uint2(q[z][2], q[z][3]);
        }
      }
    }
  }
};

// Rows of the output stage to global memory, or added to what is there, without going through registers.
__device__ __forceinline__ void bulk_store(float* dst, uint32_t src, int bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_add(float* dst, uint32_t src, int bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes)
               : "memory");
}
// The outputs of a tile that are NaN, as multiply-add chains over k.  (Where the operands hold NaN or infinities only, and
// then all that such a value reaches; finite outputs stay as they are.)
template <bool TA, bool TB>
__device__ __forceinline__ void sum_again(const GemmParams& p, float* C, int m0, int n0, int k_lo, int k_hi, int tid) {
#pragma unroll 1
  for (int i = tid; i < TM * TN; i += THREADS + 32) {
    const int m = m0 + i / TN, n = n0 + i % TN;
    if (m >= p.M || n >= p.N) continue;
    float* c = C + (long long)m * p.ldc + n;
    if (*c == *c) continue;
    const float* a = TA ? p.A + (long long)k_lo * p.lda + m : p.A + (long long)m * p.lda + k_lo;
    const float* b = TB ? p.B + (long long)k_lo * p.ldb + n : p.B + (long long)n * p.ldb + k_lo;
    float s = 0.f;
#pragma unroll 1
    for (int k = k_lo; k < k_hi && s == s; ++k) {
      s = fmaf(*a, *b, s);
      a += TA ? p.lda : 1;
      b += TB ? p.ldb : 1;
    }
    if (p.add != nullptr) s += p.add[(long long)m * p.ldadd + n];
    *c = s;
  }
}

// blockIdx: (tile of N, tile of M, part of K).  With several parts of K each writes its own C (M * N apart).
template <bool TA, bool TB>
__global__ void __launch_bounds__(THREADS + 32, 2) gemm_kernel(const GemmParams p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t s_full[STAGES], s_free[STAGES];
  __shared__ uint32_t s_tmem, s_nan;
  __shared__ volatile uint32_t s_gave_up;
#ifdef SRWM_DEBUG_CHECKS
  const int tries = p.tries;
#else
  constexpr int tries = TRIES;
#endif
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  const int k_lo = blockIdx.z * p.kpart, k_hi = min(p.K, k_lo + p.kpart);
  if (tid == 0) {
    s_nan = s_gave_up = 0;
#pragma unroll
    for (int i = 0; i < STAGES; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&s_full[i])), "r"(THREADS / 32));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_free[i])));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(256));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tm = s_tmem, full0 = smem_u32(&s_full[0]), free0 = smem_u32(&s_free[0]), sb = smem_u32(smem);
  const bool cuts = warp < THREADS / 32;   // else: the warp that issues the products

  Loader<TA> la(p.A, p.lda, m0, p.M, k_lo, cuts ? k_hi : k_lo, tid);
  Loader<TB> lb(p.B, p.ldb, n0, p.N, k_lo, cuts ? k_hi : k_lo, tid);
  float va[16], vb[16];   // the stage to be cut next
  if (cuts) {
    la.load(va);
    lb.load(vb);
  }
  bool alive = true;
  float* so = reinterpret_cast<float*>(smem);
  float* C = p.C + (long long)blockIdx.z * p.M * p.N;
  const int kdrain = p.K > 512 ? 2 * KDRAIN : KDRAIN;
  for (int kd = k_lo; kd < k_hi && alive; kd += kdrain) {
    const int stages = (min(k_hi, kd + kdrain) - kd + TK - 1) / TK;
    if (cuts) {
      for (int s = 0; s < stages && alive; ++s) {
        const int b = s % STAGES;
        unsigned char* st = smem + b * STAGE;
        // the products of stage s - STAGES have read this buffer
        if (s >= STAGES) alive = __all_sync(0xffffffffu, wait_parity(free0 + b * 8, (s / STAGES - 1) & 1, tries));
        if (!alive) break;
        la.store(st, va);
        la.load(va);
        lb.store(st + 3 * PIECE, vb);
        lb.load(vb);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full0 + b * 8) : "memory");
      }
      // all products done: the last stage's commit covers the earlier ones
      if (alive)
        alive = __all_sync(0xffffffffu, wait_parity(free0 + ((stages - 1) % STAGES) * 8, ((stages - 1) / STAGES) & 1, tries));
    } else if (lane == 0) {
      for (int s = 0; s < stages && alive; ++s) {
        const int b = s % STAGES;
        alive = wait_parity(full0 + b * 8, (s / STAGES) & 1, tries);
        if (!alive) {   // the products that have been issued come to their end before the CTA does
          if (s > 0) (void)wait_parity(free0 + ((s - 1) % STAGES) * 8, ((s - 1) / STAGES) & 1, tries);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = sb + b * STAGE, bb = a + 3 * PIECE;
#pragma unroll
        for (int ks = 0; ks < TK / 16; ++ks) {
          const uint32_t o = ks * 2 * KSTEP;
#pragma unroll
          for (int w = 2; w >= 1; --w)
#pragma unroll
            for (int i = 0; i <= w; ++i)
              mma_issue(tm + TN, a + i * PIECE + o, bb + (w - i) * PIECE + o, !(s == 0 && ks == 0 && w == 2 && i == 0));
          mma_issue(tm, a + o, bb + o, s != 0 || ks != 0);
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(free0 + b * 8)
                     : "memory");
      }
    }
    if (!cuts) {   // the next products overwrite the accumulators
      // (the cutting warps come to this barrier whether they have given up or not)
      alive = __shfl_sync(0xffffffffu, alive ? 1 : 0, 0) != 0;
      bar_sync(BAR_READ, THREADS + 32);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (s_gave_up) alive = false;
      continue;
    }
    // every cutting warp has seen the last products, or one has given up: then all leave
    alive = bar_all(BAR_CUT, THREADS, alive);
    if (!alive) {
      s_gave_up = 1;
      bar_arrive(BAR_READ, THREADS + 32);
      break;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // warps 0-3 and 4-7: the four lane quarters of tensor memory, columns 0-63 and 64-127; to the stages, which are free
    const uint32_t tr = tm + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * 64;
    float* d = so + ((warp & 3) * 32 + lane) * CP + (warp >> 2) * 64;
    float nan = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t h[16], l[16];
#define TMEM_LD16(r, addr)                                                                                         \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];" \
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),      \
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])  \
               : "r"(addr))
      TMEM_LD16(h, tr + c * 16);
      TMEM_LD16(l, tr + TN + c * 16);
#undef TMEM_LD16
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        const float4 v =
            make_float4(__uint_as_float(h[j]) + __uint_as_float(l[j]), __uint_as_float(h[j + 1]) + __uint_as_float(l[j + 1]),
                        __uint_as_float(h[j + 2]) + __uint_as_float(l[j + 2]), __uint_as_float(h[j + 3]) + __uint_as_float(l[j + 3]));
        *reinterpret_cast<float4*>(d + c * 16 + j) = v;
        if (c == (warp & 3)) nan += (v.x + v.y) + (v.z + v.w);
      }
    }
    // An infinite operand makes a whole row or column of the tile NaN: each row is looked at in 16 of its columns, each
    // column in the 32 rows of one warp.
    if (nan != nan) s_nan = 1;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    bar_arrive(BAR_READ, THREADS + 32);
    const bool first = kd == k_lo;
    if (first && p.add != nullptr) {   // warp w of eight takes row w, its lanes the columns; four additions in flight
      bar_sync(BAR_CUT, THREADS);
      const int c = lane * 4;
      if (n0 + c < p.N) {              // N is a multiple of 4
#pragma unroll 1
        for (int r0 = warp; r0 < TM; r0 += 32) {
          float4 x[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            x[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (m0 + r0 + 8 * j < p.M)
              x[j] = *reinterpret_cast<const float4*>(p.add + (long long)(m0 + r0 + 8 * j) * p.ldadd + n0 + c);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float4& v = *reinterpret_cast<float4*>(so + (r0 + 8 * j) * CP + c);
            v = make_float4(v.x + x[j].x, v.y + x[j].y, v.z + x[j].z, v.w + x[j].w);
          }
        }
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    bar_sync(BAR_CUT, THREADS);
    if (tid < TM) {   // a row each
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // (the last drain's row has been written)
      if (m0 + tid < p.M) {
        float* row = C + (long long)(m0 + tid) * p.ldc + n0;
        const int bytes = min(TN, p.N - n0) * 4;
        if (first) bulk_store(row, smem_u32(so + tid * CP), bytes);
        else bulk_add(row, smem_u32(so + tid * CP), bytes);
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    bar_sync(BAR_CUT, THREADS);   // the stages are free again
  }
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm), "r"(256));
  if (s_gave_up) {
    if (tid == 0) {
      atomicAdd(&g_timeouts, 1u);
      if (p.gave_up != nullptr) {
        *reinterpret_cast<volatile unsigned*>(p.gave_up) = 1u;
        __threadfence_system();
      }
    }
#pragma unroll 1
    for (int i = tid; i < TM * TN; i += THREADS + 32)
      if (m0 + i / TN < p.M && n0 + i % TN < p.N) C[(long long)(m0 + i / TN) * p.ldc + n0 + i % TN] = __int_as_float(0x7fffffff);
  } else if (s_nan) {
    sum_again<TA, TB>(p, C, m0, n0, k_lo, k_hi, tid);
  }
}

// ---- few outputs: an actor's step ----------------------------------------------------------------
// 16 x 16 outputs a CTA, 128 values of k at a time through shared memory, a quarter of them and 2 x 2 outputs a thread
// (one output a thread over all k read twice as much shared memory per multiply-add).  With 48 rows the
// tensor-core kernel would run on two multiprocessors; the library took 7.5 us for 48 x 256 x 256, this 5.4.
constexpr int SB = 16, SK = 128, SP = SK + 4, SV = SB * SK / 256;   // SV: values of each operand per thread
template <bool T>
__device__ __forceinline__ void skinny_load(const float* base, long long ld, int r0, int rows, int k0, int K, float (&v)[SV],
                                            int tid) {
#pragma unroll
  for (int i = 0; i < SV; ++i) v[i] = 0.f;
  if constexpr (T) {   // adjacent threads along the rows
    const int r = tid % SB, kk = tid / SB;
    if (r0 + r < rows) {
#pragma unroll
      for (int i = 0; i < SV; ++i) {
        const int k = k0 + kk + i * (256 / SB);
        if (k < K) v[i] = base[(long long)k * ld + r0 + r];
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < SV; i += 4) {
      const int piece = tid + (i / 4) * 256, r = piece / (SK / 4), k = k0 + (piece % (SK / 4)) * 4;
      if (r0 + r < rows && k < K) {   // K is a multiple of 4
        const float4 x = *reinterpret_cast<const float4*>(base + (long long)(r0 + r) * ld + k);
        v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
      }
    }
  }
}
template <bool T>
__device__ __forceinline__ void skinny_store(float* s, const float (&v)[SV], int tid) {
  if constexpr (T) {
#pragma unroll
    for (int i = 0; i < SV; ++i) s[(tid % SB) * SP + tid / SB + i * (256 / SB)] = v[i];
  } else {
#pragma unroll
    for (int i = 0; i < SV; i += 4) {
      const int piece = tid + (i / 4) * 256;
      *reinterpret_cast<float4*>(s + (piece / (SK / 4)) * SP + (piece % (SK / 4)) * 4) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    }
  }
}
template <bool TA, bool TB>
__global__ void __launch_bounds__(256) gemm_skinny_kernel(const GemmParams p) {
  __shared__ __align__(16) float sa[SB * SP], sbt[SB * SP];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * SB, n0 = blockIdx.x * SB;
  const int kq = (tid / 64) * (SK / 4), n = tid % 8, m = (tid / 8) % 8;   // a quarter of the k, 2 x 2 outputs 8 apart
  float acc[2][2] = {}, ra[SV], rb[SV];
  chained();
  skinny_load<TA>(p.A, p.lda, m0, p.M, 0, p.K, ra, tid);
  skinny_load<TB>(p.B, p.ldb, n0, p.N, 0, p.K, rb, tid);
  for (int k0 = 0; k0 < p.K; k0 += SK) {
    if (k0 > 0) __syncthreads();
    skinny_store<TA>(sa, ra, tid);
    skinny_store<TB>(sbt, rb, tid);
    __syncthreads();
    skinny_load<TA>(p.A, p.lda, m0, p.M, k0 + SK, p.K, ra, tid);
    skinny_load<TB>(p.B, p.ldb, n0, p.N, k0 + SK, p.K, rb, tid);
#pragma unroll
    for (int k = 0; k < SK / 4; k += 4) {   // (values beyond K are zero)
      float4 a[2], b[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        a[i] = *reinterpret_cast<const float4*>(sa + (m + 8 * i) * SP + kq + k);
        b[i] = *reinterpret_cast<const float4*>(sbt + (n + 8 * i) * SP + kq + k);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
          acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
          acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) sa[(tid / 64) * SB * SB + (m + 8 * i) * SB + n + 8 * j] = acc[i][j];
  __syncthreads();
  const int r = m0 + tid / SB, c = n0 + tid % SB;
  if (r < p.M && c < p.N) {
    float v = (sa[tid] + sa[tid + SB * SB]) + (sa[tid + 2 * SB * SB] + sa[tid + 3 * SB * SB]);
    if (p.add != nullptr) v += p.add[(long long)r * p.ldadd + c];
    p.C[(long long)r * p.ldc + c] = p.relu && v < 0.f ? 0.f : v;
  }
}

// C = (add) + the parts, in their order; dense
__global__ void __launch_bounds__(256) gemm_sum_kernel(const float* part, long long count, int parts, const float* add, float* C) {
  const long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
  if (i >= count) return;
  float4 t = add != nullptr ? *reinterpret_cast<const float4*>(add + i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int k = 0; k < parts; ++k) {
    const float4 v = __ldcs(reinterpret_cast<const float4*>(part + (long long)k * count + i));
    t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
  }
  *reinterpret_cast<float4*>(C + i) = t;
}

template <bool TA, bool TB>
cudaError_t launch(const GemmParams& p, int parts, cudaStream_t s) {
  static unsigned long long ready = 0;   // devices whose shared-memory limit has been raised
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(__atomic_load_n(&ready, __ATOMIC_ACQUIRE) & bit)) {
    e = cudaFuncSetAttribute(gemm_kernel<TA, TB>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return e;
    __atomic_fetch_or(&ready, bit, __ATOMIC_RELEASE);
  }
  const dim3 grid((p.N + TN - 1) / TN, (p.M + TM - 1) / TM, parts);
  gemm_kernel<TA, TB><<<grid, THREADS + 32, SMEM, s>>>(p);
  return cudaGetLastError();
}

}  // namespace

// One part while the tiles fill half the multiprocessors or the sum is short (the parts' sums are a launch of
// their own); else enough parts for two CTAs on each, no part shorter than 64 values.  us on 148 multiprocessors, launches
// back to back, M x N x K:
//   3200 x 512 x 512, 100 tiles     one part 22.7, two 25.8    |  3200 x 256 x 128, 50 tiles   one 10.4, two 12.4
//   800 x 256 x 512, 14 tiles       one 22.7, two 17.5, four 14.5, eight (the rule) 12.4
//   512 x 512 x 3200 (transposed), 16 tiles   one 98.5, four 32.9, eight 20.6, twelve 24.7
// One CTA on each multiprocessor (eight parts in the last line) is as good as two or better up to K of some 3000; from 6000 on
// two are (x 12448: eight 57.4, sixteen 53.6).
int gemm_parts(int M, int N, int K) {
  const int tiles = ((M + TM - 1) / TM) * ((N + TN - 1) / TN), stages = (K + TK - 1) / TK, sms = common_sms();
  if (2 * tiles >= sms || stages < 8) return 1;
  const int want = 2 * sms / tiles, most = stages / 2;   // (one CTA more than fit would run alone)
  return want < most ? want : most;
}

// The word a kernel sets when it gives up: in host memory, so that a call sees it without waiting for the device.  Taken once
// for the process, also while a stream is being captured; null if it cannot be had (the results are NaN all the same).
static unsigned* gave_up_word(bool create) {
  static std::atomic<unsigned*> word{nullptr};
  static std::once_flag once;
  if (create)
    std::call_once(once, [] {
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
      if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return (void)cudaGetLastError();
      void* w = nullptr;
      if (cudaHostAlloc(&w, sizeof(unsigned), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) (void)cudaGetLastError();
      (void)cudaThreadExchangeStreamCaptureMode(&mode);
      if (w) *static_cast<unsigned*>(w) = 0;
      word.store(static_cast<unsigned*>(w), std::memory_order_release);
    });
  return word.load(std::memory_order_acquire);
}
bool gemm_gave_up() {
  unsigned* w = gave_up_word(false);
  return w && __atomic_load_n(w, __ATOMIC_RELAXED) && __atomic_exchange_n(w, 0u, __ATOMIC_RELAXED);
}
#ifdef SRWM_DEBUG_CHECKS
int gemm_tries = TRIES;
#endif

cudaError_t gemm_launch(const GemmParams& q, bool ta, bool tb, float* scratch, cudaStream_t s) {
  GemmParams p = q;
  p.gave_up = gave_up_word(true);
#ifdef SRWM_DEBUG_CHECKS
  p.tries = gemm_tries;
#endif
  int parts = scratch ? gemm_parts(p.M, p.N, p.K) : 1;
  const long long count = (long long)p.M * p.N;
  p.kpart = ((p.K + parts - 1) / parts + TK - 1) / TK * TK;
  parts = (p.K + p.kpart - 1) / p.kpart;
  if (parts > 1) {
    p.C = scratch;
    p.add = nullptr;
    p.ldc = p.N;
  }
  const cudaError_t e = ta ? (tb ? launch<true, true>(p, parts, s) : launch<true, false>(p, parts, s))
                           : (tb ? launch<false, true>(p, parts, s) : launch<false, false>(p, parts, s));
  if (e != cudaSuccess || parts == 1) return e;
  gemm_sum_kernel<<<(unsigned)((count / 4 + 255) / 256), 256, 0, s>>>(scratch, count, parts, q.add, q.C);
  return cudaGetLastError();
}

// Few outputs: up to 16 blocks of 16 x 16 a multiprocessor in sums of 256 values, up to 6 in sums of 512.  Few-row kernel against
// tiles with their best number of parts, us on 148 multiprocessors, launches back to back:
//   K = 64     1600 blocks 8.5 / 8.3, 3200: 15.2 / 8.3      K = 128    1600: 8.7 / 10.4, 3200: 15.6 / 10.4
//   K = 256    800: 8.7 / 12.4, 1600: 14.5 / 12.4           K = 512    208: 6.3 / 12.4, 416: 12.8 / 12.4, 800: 15.2 / 12.4
//   K = 768    208: 8.7 / 12.4, 416: 18.3 / 12.4
// So the lines are the crossing at K of 128 only: at 256 and 512 the last third of the range loses 2 to 3 us, and above 512 up to
// 200 blocks would gain 4.
bool gemm_is_skinny(int M, int N, int K) {
  const long long blocks = (long long)((M + SB - 1) / SB) * ((N + SB - 1) / SB);
  const int sms = common_sms();
  return (K <= 512 && blocks <= 6 * sms) || (K <= 256 && blocks <= 16 * sms);
}
cudaError_t gemm_skinny_launch(const GemmParams& p, bool ta, bool tb, cudaStream_t s) {
  const dim3 grid((p.N + SB - 1) / SB, (p.M + SB - 1) / SB);
  if (ta) return tb ? launch_behind(gemm_skinny_kernel<true, true>, p, grid, 256, 0, s)
                    : launch_behind(gemm_skinny_kernel<true, false>, p, grid, 256, 0, s);
  return tb ? launch_behind(gemm_skinny_kernel<false, true>, p, grid, 256, 0, s)
            : launch_behind(gemm_skinny_kernel<false, false>, p, grid, 256, 0, s);
}

unsigned gemm_timeouts() {
  unsigned v = 0;
  if (cudaMemcpyFromSymbol(&v, g_timeouts, sizeof v) != cudaSuccess) (void)cudaGetLastError();
  return v;
}

}  // namespace srwm
