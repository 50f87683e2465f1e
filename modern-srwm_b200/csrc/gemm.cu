// fp32 matrix products of the layers' linear maps (out_linear, slow_net and their gradients) on the
// 5th-generation tensor cores:  C[M, N] = op(A) op(B)^T (+ add).
//
// Finite fp32 operands are cut into three bf16 pieces, exactly (mma.cuh), and the six products of pieces down to
// 2^-16 of the leading one are summed in fp32, the leading one and the rest in accumulators of their own.
// An infinite one has no such pieces: all outputs it reaches come out as NaN.  The warps that empty the accumulators look for NaN;
// behind its last unit a CTA sums its NaN outputs again on the fp32 pipe (sum_again), where infinities are what arithmetic makes of them.
// 16384 x 512 x 512, one at a time: 73 us, 130 with an infinity in A, 700 with one in B (a column of every tile), 160 with NaN everywhere.
// The tensor cores' accumulators round towards zero, one unit in 2^24 per 16 values of k, which adds up in one
// direction; so every 128 values of k (64 where the sum has 256 or fewer) they are emptied into registers, whose additions
// round to nearest.  Error of the result, 2-norm, normal inputs: 1.2e-7 at k = 256, 1.7e-7 at 512, 1.9e-7 at 16384 (emptied every
// 256: 2.8e-7, every 64: 1.3e-7 at 512 and 6 % more time), against 4.1e-7 and 7e-7 of the library's fp32 product at 512 and 2048.
//
// A pair of CTAs (cluster) works on 256 x 128 outputs, 128 x 128 each, with the pair's tcgen05.mma (256 x 128 x 16): each cuts its own
// 128 rows of A and half of the 128 of B, so that a quarter less is cut and read from shared memory than with a tile of its own.
// One CTA a multiprocessor (the hardware allows no more with pairs), which goes from unit to unit of a fixed list.  Eight
// warps read 32 values of k of the fp32 operands two stages ahead into registers, cut them and store the pieces as core matrices
// (no swizzle; along k or along the rows, whichever is the inner dimension in memory), four stages deep; a warp of the pair's first CTA
// issues twelve products a stage; eight more warps empty the accumulators, of which there are two sets, while the next
// sum is under way, and hold the sums of a unit in registers until it is done.  Stages and accumulators are handed over through
// mbarriers, counted in the first CTA where they concern both.
//
// Bound: 64 stages of a CTA (18944 x 512 x 512) take 48 us with the cutting warps only handing stages over, 52 with constants to cut
// and 58 as it is (launches back to back; 36 at the burst rate of the tensor cores, 42 at their sustained rate).  128 x 128 tiles of
// single CTAs, two a multiprocessor, took 70: their operands alone keep shared memory busy for the time of the products, and stores
// that met in its banks came on top.  16384 x 512 x 512: 71 -> 62 us; 12448 x 1544 x 512: 153 -> 124, its gradients 160 -> 130 and
// 159 -> 145.  Short sums lost: a captured row of launches, 12448 x 256 x 256 (98 units for 74 pairs) 19.3 -> 21, 5000 x 132 x 64 6.9 -> 7.8,
// 256 x 256 x 1024 9.9 -> 11, 3200 x 256 x 256 11.8 -> 12.3 (a pair takes some 0.7 us longer to begin and end; with the first loads in
// front of its set-up these are 1 to 3 % faster, and 12448 x 1544 x 512 119.7 -> 121.3).
// On the way here: loads through temporaries, for which a warp waits where it asks for them, 65 us; waits with cluster
// scope (they empty the L1 cache) 110; six stages, which leave the loads no L1 cache to arrive in, 63; A's pieces in tensor memory and
// one set of accumulators 58, and 115 where k is not the inner dimension; all sixteen warps cutting and emptying 80, in two groups
// of alternate stages 65.
#include "gemm.h"

#include <atomic>
#include <mutex>

#include "chain.h"
#include "device.h"
#include "mma.cuh"

namespace srwm {
namespace {

constexpr int TM = 128, TN = 128, TK = 32, STAGES = 4;   // a CTA's outputs and values of k a stage
constexpr int CUT = 256, DRAIN = 256, THREADS = CUT + DRAIN + 32;   // those that cut, those that empty the accumulators, a warp that issues
constexpr int AHEAD = 2;                          // stages of fp32 values on their way into a thread's registers
constexpr int CORE = 128;                         // bytes of a core matrix: 8 rows x 8 bf16
// Pieces of a tile of ROWS x 32 lie as core matrices.  Rows that are contiguous along k (K-major): those of adjacent rows
// adjacent, KSTEP bytes to the next along k.  Rows that are the inner dimension in memory (T, MN-major: a core matrix is 8 values of
// k x 8 rows): those of adjacent k adjacent, MSTEP bytes to the next along the rows.  (+ 32, + 16: the lanes of a half warp that
// store side by side miss each other's banks)
template <int ROWS>
constexpr int KSTEP = (ROWS / 8) * CORE + 32;
constexpr int MSTEP = (TK / 8) * CORE + 16;
template <bool T, int ROWS>
constexpr int PIECE = T ? ROWS / 8 * MSTEP : (TK / 8) * KSTEP<ROWS>;
constexpr int HN = TN / 2;                        // a CTA's rows of B: the other half of the pair's tile comes from the other CTA
template <bool TA, bool TB>
constexpr int STAGE = 3 * (PIECE<TA, TM> + PIECE<TB, HN>);   // three pieces of A and of B
constexpr int BAR_DRAIN = 1;                      // named barrier: the draining warps

// Waits have a limit (none is expected to reach it).  A CTA in which one has given up leaves NaN in its tile of C, counts
// here and sets the caller's word in host memory, at which the next call fails.
constexpr int TRIES = 4000000;
__device__ unsigned g_timeouts;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// No swizzle.  Strides from core matrix to core matrix: along k, along the rows.
template <bool T, int ROWS>
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
  constexpr int along_k = T ? CORE : KSTEP<ROWS>, along_rows = T ? MSTEP : CORE;
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(along_k >> 4) << 16) | ((uint64_t)(along_rows >> 4) << 32) |
         ((uint64_t)1 << 46);
}
// 256 x 128 x 16 of a pair of CTAs: rows 128 r.. of A and of the result are CTA r's, as are rows 64 r.. of B
template <bool TA, bool TB>
__device__ __forceinline__ void mma_issue(uint32_t d, uint32_t a, uint32_t b, bool add) {
  constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((TA ? 1u : 0u) << 15) | ((TB ? 1u : 0u) << 16) |
                             ((TN / 8) << 17) | ((2 * TM / 16) << 24);   // f32 += bf16 bf16
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(operand_desc<TA, TM>(a)),
      "l"(operand_desc<TB, HN>(b)), "r"(idesc), "r"(add ? 1u : 0u)
      : "memory");
}
// The pair's first CTA's word at this one's address
__device__ __forceinline__ uint32_t of_first(uint32_t addr) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void arrive_at(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void commit_both(uint32_t bar) {   // when the products so far are done: arrives at both CTAs' word
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"((uint16_t)3)
               : "memory");
}
// 16 lanes x 16 columns: rows g and g + 8 of the lanes, columns 2t, 2t + 1 of each eight (lane = 4 g + t)
__device__ __forceinline__ void tm_ld_16x16(uint32_t (&r)[8], uint32_t addr) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(addr));
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
  u64 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
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

// The four values at a place in global memory, or zeros.  (Written out so that they land in v itself: through temporaries the
// thread waits for them where it asks for them.)
__device__ __forceinline__ void ldg4_if(float* v, const float* p, bool on) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
      "@q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
      : "l"(p), "r"(on ? 1 : 0));
}
// One thread's share of a tile of ROWS x 32: NL times four values.
//   K-major: four values of k of rows 32 apart; eight lanes read a whole 128-byte line of each.
//   T: four rows at values of k KS apart; a half or a whole warp reads the rows of one.
// Rows beyond the matrix read its first rows: they end in rows of C that are not stored.  Nothing is read at or beyond the
// part's end, nor beside the rows where their number is no multiple of four.
template <bool T, int ROWS>
struct Loader {
  static constexpr int NL = ROWS / 32, LR = ROWS / 4, KS = T ? 32 / LR : 0;   // LR: lanes side by side along the rows
  const float* p;              // the first four at the next stage to be loaded
  long long ld;
  long long off[T ? 1 : NL];   // K-major: from the first row to the others (they may be clamped to the matrix)
  int left;                    // values of k from p to the part's end
  int edge;                    // T: the rows there are of the four, where there are fewer
  int row, k_of;               // this thread's place in a tile
  __device__ __forceinline__ Loader(long long ld_, int tid)
      : p(nullptr), ld(ld_), left(0), edge(4), row(T ? tid % LR * 4 : tid / 8),
        k_of(T ? tid / 32 * 4 + tid % 32 / LR : tid % 8 * 4) {
    static_assert(!T || NL * KS == 4, "a warp has four values of k");
  }
  __device__ __forceinline__ void start(const float* base, int r0, int rows, int k_lo, int k_hi) {
    left = k_hi - k_lo - k_of;
    const int r = r0 + row < rows ? r0 + row : 0;
    if constexpr (T) {
      edge = min(4, rows - r);
      p = base + (long long)(k_lo + k_of) * ld + r;
    } else {
#pragma unroll
      for (int i = 0; i < NL; ++i) off[i] = ((r0 + row + i * 32 < rows ? r0 + row + i * 32 : 0) - r) * ld;
      p = base + (long long)r * ld + k_lo + k_of;
    }
  }
  __device__ __forceinline__ void load(float (&v)[4 * NL]) {
    if constexpr (T) {
      const float* q = p;
#pragma unroll
      for (int i = 0; i < NL; ++i) {
        ldg4_if(&v[4 * i], q, i * KS < left && edge == 4);
        q += KS * ld;
      }
      if (edge < 4) {
#pragma unroll
        for (int i = 0; i < NL; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j)
            if (i * KS < left && j < edge) v[4 * i + j] = __ldg(p + i * KS * ld + j);
      }
      p += TK * ld;
    } else {
#pragma unroll
      for (int i = 0; i < NL; ++i) ldg4_if(&v[4 * i], p + off[i], left > 0);   // K is a multiple of 4
      p += TK;
    }
    left -= TK;
  }
  __device__ __forceinline__ void store(unsigned char* st, const float (&v)[4 * NL]) const {
    st += T ? row / 8 * MSTEP + k_of / 8 * CORE + k_of % 8 * 16 + row % 8 * 2
            : row / 8 * CORE + k_of / 8 * KSTEP<ROWS> + row % 8 * 16 + k_of % 8 * 2;
#pragma unroll
    for (int i = 0; i < NL; ++i) {
      uint32_t q[3][2];
#pragma unroll
      for (int j = 0; j < 2; ++j) split3(v[4 * i + 2 * j], v[4 * i + 2 * j + 1], q[0][j], q[1][j], q[2][j]);
#pragma unroll
      for (int z = 0; z < 3; ++z)
        *reinterpret_cast<uint2*>(st + i * (T ? KS * 16 : 4 * CORE) + z * PIECE<T, ROWS>) = make_uint2(q[z][0], q[z][1]);
    }
  }
};

// The outputs of a tile that are NaN, as multiply-add chains over k.  (Where the operands hold NaN or infinities only, and
// then all that such a value reaches; finite outputs stay as they are.)  It can take longer than the waits of the other roles and of
// the other CTA last (a whole tile is 30 outputs a thread, one after the other), so it comes behind them, and all threads take part.
template <bool TA, bool TB>
__device__ __forceinline__ void sum_again(const GemmParams& p, float* C, int m0, int n0, int k_lo, int k_hi, int tid) {
#pragma unroll 1
  for (int i = tid; i < TM * TN; i += THREADS) {
    // (each row begins one column further on, so that the outputs of a column, which an infinity in B reaches, fall to a thread each)
    const int m = m0 + i / TN, n = n0 + (i + i / TN) % TN;
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

// A unit of work: a pair of tiles (256 x 128) and a part of K.  With several parts each writes its own C (M * N apart).
struct Unit {
  int m0, n0, k_lo, k_hi, part;   // m0: the pair's first row
  int drain;                      // stages an accumulator takes: 64 values of k in short sums, 128 else
  __device__ __forceinline__ Unit(const GemmParams& p, int u) {
    const int nt = (p.N + TN - 1) / TN, tiles = nt * ((p.M + 2 * TM - 1) / (2 * TM)), tile = u % tiles;
    part = u / tiles;
    m0 = tile / nt * 2 * TM;      // (tiles of N side by side: a pair's rows of A are still in L2)
    n0 = tile % nt * TN;
    k_lo = part * p.kpart;
    k_hi = min(p.K, k_lo + p.kpart);
    drain = p.kpart <= 256 ? 2 : 4;
  }
  __device__ __forceinline__ int stages() const { return (k_hi - k_lo + TK - 1) / TK; }
  __device__ __forceinline__ int drains() const { return (stages() + drain - 1) / drain; }
};
// A place in a ring, and how often it has been gone round.
template <int N>
struct Ring {
  int i = 0;
  uint32_t round = 0;
  __device__ __forceinline__ void next() {
    if (++i == N) {
      i = 0;
      ++round;
    }
  }
};

// Of a CTA's units those marked in again: bit u / step % 32 for unit u.  (Of units that share a bit, one without NaN is only read.)
template <bool TA, bool TB>
__device__ __noinline__ void sum_again_units(const GemmParams& p, uint32_t again, int rank, int step, int tid) {
#pragma unroll 1
  for (int u = blockIdx.x / 2; u < p.units; u += step) {
    if ((again >> (u / step % 32) & 1) == 0) continue;
    const Unit w(p, u);
    sum_again<TA, TB>(p, p.C + (long long)w.part * p.M * p.N, w.m0 + rank * TM, w.n0, w.k_lo, w.k_hi, tid);
  }
}

// Units blockIdx.x / 2, + gridDim.x / 2, ... of the pair (cluster) of CTAs.
template <bool TA, bool TB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1) gemm_kernel(const __grid_constant__ GemmParams p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  // stages cut (both CTAs, counted in the first) and read; accumulators summed and read (counted in the first)
  __shared__ __align__(8) uint64_t s_full[STAGES], s_free[STAGES], s_sum[2], s_read[2];
  __shared__ uint32_t s_tmem, s_again;
#ifdef SRWM_DEBUG_CHECKS
  const int tries = p.tries;
#else
  constexpr int tries = TRIES;
#endif
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, rank = blockIdx.x & 1, step = gridDim.x / 2;
  if (tid == 0) {
    s_again = 0;   // units with NaN among their outputs, see sum_again_units
#pragma unroll
    for (int i = 0; i < STAGES; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&s_full[i])), "r"(2 * CUT / 32));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_free[i])));
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_sum[i])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&s_read[i])), "r"(2 * DRAIN / 32));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tm = s_tmem, full0 = smem_u32(s_full), free0 = smem_u32(s_free), sum0 = smem_u32(s_sum), read0 = smem_u32(s_read);
  bool alive = true;

  if (warp < CUT / 32) {
    // ================= cut =================
    const uint32_t full_first = of_first(full0);
    int u = blockIdx.x / 2, left = 0, todo = 0;   // the unit being loaded, its stages to be loaded; stages loaded and not yet stored
    Loader<TA, TM> la(p.lda, tid);
    Loader<TB, HN> lb(p.ldb, tid);
    float va[AHEAD][TM / 8], vb[AHEAD][HN / 8];
    auto load = [&](int i) {
      if (left == 0 && u < p.units) {
        const Unit w(p, u);
        la.start(p.A, w.m0 + rank * TM, p.M, w.k_lo, w.k_hi);
        lb.start(p.B, w.n0 + rank * HN, p.N, w.k_lo, w.k_hi);
        left = w.stages();
        u += step;
      }
      la.load(va[i]);   // (zeros behind the last unit)
      lb.load(vb[i]);
      if (left > 0) {
        --left;
        ++todo;
      }
    };
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) load(i);
    Ring<STAGES> r;
    while (todo > 0 && alive) {
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        if (todo == 0) break;
        --todo;
        unsigned char* st = smem + r.i * STAGE<TA, TB>;
        // the products of the round before have read this place
        if (r.round > 0) alive = __all_sync(0xffffffffu, wait_parity(free0 + r.i * 8, (r.round - 1) & 1, tries));
        if (!alive) break;
        la.store(st, va[i]);
        lb.store(st + 3 * PIECE<TA, TM>, vb[i]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) arrive_at(full_first + r.i * 8);
        load(i);   // (behind the fence, which waits for loads in front of it)
        r.next();
      }
    }
  } else if (warp < (CUT + DRAIN) / 32) {
    // ================= empty the accumulators =================
    const uint32_t read_first = of_first(read0);
    const int q = warp & 3, half = (warp - CUT / 32) >> 2;                       // rows 32 q.., columns 64 half..
    const uint32_t tr = tm + ((uint32_t)(q * 32) << 16) + half * 64;
    Ring<2> r;
    int u = blockIdx.x / 2;
    for (; u < p.units; u += step) {
      const Unit w(p, u);
      const int m0 = w.m0 + rank * TM, row0 = m0 + q * 32 + lane / 4, c0 = w.n0 + half * 64 + 2 * (lane % 4);
      u64 acc[2][8][2];   // rows (+ 16) x tiles of 8 columns x (row g, row g + 8): two columns
      // What is added comes first: its loads have until the first sum.  (Behind the sums they took longer than the next sums.)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const bool on = p.add != nullptr && row0 + i * 16 + h * 8 < p.M;
          const float* add = p.add + (long long)(row0 + i * 16 + h * 8) * p.ldadd + c0;
#pragma unroll
          for (int j = 0; j < 8; ++j)   // N is a multiple of 4
            acc[i][j][h] = on && c0 + 8 * j < p.N ? *reinterpret_cast<const u64*>(add + 8 * j) : 0ull;
        }
      for (int d = w.drains(); d > 0 && alive; --d) {
        alive = __all_sync(0xffffffffu, wait_parity(sum0 + r.i * 8, r.round & 1, tries));
        if (!alive) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 8; j += 2) {
            const uint32_t a = tr + r.i * 2 * TN + ((uint32_t)(i * 16) << 16) + j * 8;
            uint32_t h[8], l[8];
            tm_ld_16x16(h, a);
            tm_ld_16x16(l, a + TN);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              asm volatile("" : "+r"(h[2 * c]), "+r"(h[2 * c + 1]), "+r"(l[2 * c]), "+r"(l[2 * c + 1]));   // (read after the wait)
              u64& v = acc[i][j + c / 2][c % 2];
              v = add2(v, add2(pack2(__uint_as_float(h[2 * c]), __uint_as_float(h[2 * c + 1])),
                               pack2(__uint_as_float(l[2 * c]), __uint_as_float(l[2 * c + 1]))));
            }
          }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) arrive_at(read_first + r.i * 8);
        r.next();
      }
      float nan = 0.f;
      float* C = p.C + (long long)w.part * p.M * p.N;
      if (alive) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int row = row0 + i * 16 + h * 8;
            if (row < p.M) {
              float* c = C + (long long)row * p.ldc + c0;
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                if (c0 + 8 * j < p.N) {
                  float2 v;
                  unpack2(acc[i][j][h], v.x, v.y);
                  nan += v.x + v.y;
                  *reinterpret_cast<float2*>(c + 8 * j) = v;
                }
              }
            }
          }
      }
      alive = bar_all(BAR_DRAIN, DRAIN, alive);
      if (!alive) break;
      if (!bar_all(BAR_DRAIN, DRAIN, nan == nan) && tid == CUT) s_again |= 1u << (u / step % 32);
    }
    if (!alive) {   // what this CTA has not finished is NaN
      if (tid == CUT) {
        atomicAdd(&g_timeouts, 1u);
        if (p.gave_up != nullptr) {
          *reinterpret_cast<volatile unsigned*>(p.gave_up) = 1u;
          __threadfence_system();
        }
      }
#pragma unroll 1
      for (; u < p.units; u += step) {
        const Unit w(p, u);
        float* C = p.C + (long long)w.part * p.M * p.N;
#pragma unroll 1
        for (int i = tid - CUT; i < TM * TN; i += DRAIN) {
          const int m = w.m0 + rank * TM + i / TN, n = w.n0 + i % TN;
          if (m < p.M && n < p.N) C[(long long)m * p.ldc + n] = __int_as_float(0x7fffffff);
        }
      }
    }
  } else if (rank == 0 && lane == 0) {
    // ================= issue the products =================
    Ring<STAGES> r;
    Ring<2> acc;
    uint32_t last = 0, last_parity = 0;   // the place whose products were issued last
    bool any = false;
    for (int u = blockIdx.x / 2; u < p.units && alive; u += step) {
      const Unit w(p, u);
      for (int left = w.stages(); left > 0 && alive; left -= w.drain, acc.next()) {
        // the sums of the round before have been read by both CTAs
        if (acc.round > 0) alive = wait_parity(read0 + acc.i * 8, (acc.round - 1) & 1, tries);
        const uint32_t d = tm + acc.i * 2 * TN;
        const int n = min(left, w.drain);
        for (int s = 0; s < n && alive; ++s) {
          alive = wait_parity(full0 + r.i * 8, r.round & 1, tries);
          if (!alive) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a = smem_u32(smem) + r.i * STAGE<TA, TB>, b = a + 3 * PIECE<TA, TM>;
#pragma unroll
          for (int ks = 0; ks < TK / 16; ++ks) {
            const uint32_t oa = a + ks * 2 * (TA ? CORE : KSTEP<TM>), ob = b + ks * 2 * (TB ? CORE : KSTEP<HN>);
#pragma unroll
            for (int x = 2; x >= 1; --x)
#pragma unroll
              for (int i = 0; i <= x; ++i)
                mma_issue<TA, TB>(d + TN, oa + i * PIECE<TA, TM>, ob + (x - i) * PIECE<TB, HN>, !(s == 0 && ks == 0 && x == 2 && i == 0));
            mma_issue<TA, TB>(d, oa, ob, s != 0 || ks != 0);
          }
          commit_both(free0 + r.i * 8);
          if (s == n - 1) commit_both(sum0 + acc.i * 8);
          last = free0 + r.i * 8;
          last_parity = r.round & 1;
          any = true;
          r.next();
        }
      }
    }
    // the products that have been issued come to their end before the CTAs do
    if (any) (void)wait_parity(last, last_parity, tries);
  }
  __syncwarp();
  __syncthreads();
  const uint32_t again = s_again;
  cluster_sync();   // neither CTA leaves while the other, or a product, may still come to its memory
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tm), "r"(512));
  if (again != 0) sum_again_units<TA, TB>(p, again, rank, step, tid);
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
cudaError_t launch(const GemmParams& p, cudaStream_t s) {
  static unsigned long long ready = 0;   // devices whose shared-memory limit has been raised
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(__atomic_load_n(&ready, __ATOMIC_ACQUIRE) & bit)) {
    e = cudaFuncSetAttribute(gemm_kernel<TA, TB>, cudaFuncAttributeMaxDynamicSharedMemorySize, STAGES * STAGE<TA, TB>);
    if (e != cudaSuccess) return e;
    __atomic_fetch_or(&ready, bit, __ATOMIC_RELEASE);
  }
  const int pairs = common_sms() / 2 > 0 ? common_sms() / 2 : 1;
  gemm_kernel<TA, TB><<<2 * (p.units < pairs ? p.units : pairs), THREADS, STAGES * STAGE<TA, TB>, s>>>(p);
  return cudaGetLastError();
}

}  // namespace

// One part while the units fill half the pairs of multiprocessors or the sum is short (the parts' sums are a launch of their
// own); else the number that takes the least time, in stages: rounds of units, each with some four more to begin and end with, and the
// launch.  us on 148 multiprocessors, a captured row of launches, M x N x K:
//   512 x 512 x 3200 (transposed), 8 tiles   one part 80, two 45, four 26.6, eight 18.8, nine (the rule) 18.5, ten 25.1
//   1544 x 512 x 12448 (transposed), 28 tiles   one 305, two 159, three 211, five (the rule) 132, six 161
//   800 x 256 x 512, 8 tiles   one 17.2, four 10.5, six 10.5   |  3200 x 256 x 256, 26 tiles   one (the rule) 12.0, four 12.1
//   2000 x 1024 x 1024, 64 tiles   one (the rule) 30.9, two 35.1
static int gemm_tiles(int M, int N) { return ((M + 2 * TM - 1) / (2 * TM)) * ((N + TN - 1) / TN); }   // pairs of tiles
int gemm_parts(int M, int N, int K) {
  const int tiles = gemm_tiles(M, N), stages = (K + TK - 1) / TK, pairs = common_sms() / 2 > 0 ? common_sms() / 2 : 1;
  if (2 * tiles >= pairs || stages < 8) return 1;
  int best = 1, cost = 1 << 30;
  for (int parts = 1; parts <= stages / 2 && tiles * (parts - 1) < 2 * pairs; ++parts) {
    const int c = (tiles * parts + pairs - 1) / pairs * ((stages + parts - 1) / parts + 4) + (parts > 1 ? 4 + parts / 4 : 0);
    if (c < cost) {
      cost = c;
      best = parts;
    }
  }
  return best;
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
  p.units = gemm_tiles(p.M, p.N) * parts;
  if (parts > 1) {
    p.C = scratch;
    p.add = nullptr;
    p.ldc = p.N;
  }
  const cudaError_t e = ta ? (tb ? launch<true, true>(p, s) : launch<true, false>(p, s))
                           : (tb ? launch<false, true>(p, s) : launch<false, false>(p, s));
  if (e != cudaSuccess || parts == 1) return e;
  gemm_sum_kernel<<<(unsigned)((count / 4 + 255) / 256), 256, 0, s>>>(scratch, count, parts, q.add, q.C);
  return cudaGetLastError();
}

// Few outputs: up to 16 blocks of 16 x 16 a multiprocessor in sums of 256 values, up to 6 in sums of 512.  Few-row kernel against
// tiles by the rule for parts, us on 148 multiprocessors, a captured row of launches, k the inner dimension of both operands (of
// neither: the few-row kernel takes up to 45 % longer, the tiles the same):
//   K = 64     800 blocks 5.2 / 7.1, 1600: 8.3 / 7.1, 2048: 10.4 / 7.1, 3200: 15.1 / 7.2
//   K = 128    1024: 6.1 / 8.7, 1600: 8.6 / 8.7, 2048: 10.5 / 8.7, 3200: 15.5 / 8.9
//   K = 256    800: 8.6 / 10.3, 1024: 9.8 / 10.2, 1600: 14.4 / 10.5, 2048: 17.9 / 10.6
//   K = 384    208: 5.0 / 9.6, 416: 10.0 / 9.9, 800: 12.1 / 10.1
//   K = 512    208: 6.2 / 10.5, 416: 12.7 / 10.8, 800: 15.2 / 10.8   K = 768    208: 8.5 / 11.2, 416: 18.2 / 11.2
//   K = 1024   48: 7.1 / 10.3, 208: 10.9 / 11.5, 416: 23.5 / 11.5
// So the lines are the crossing at K of 128 only.  The tiles would be the faster ones by up to 3 us at K = 64, 7 at 256 and 4 at 512 (8, 14
// and 9 with k inner in neither) towards the ends of the ranges, and few rows by up to 4 above 512.  The lines stay because what the few-row kernel alone takes hangs on them: ReLU
// in the product, which a call asks for by this rule, and a bias, which tiles in parts do not add.
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
