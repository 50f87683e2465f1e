// Warp-level matrix products for the chunked delta-rule kernels: mma.sync m16n8k16 on bf16
// operands with fp32 accumulators, and fp32 operands as exact sums of three bf16 pieces.
//
// Why this instruction: the products of a chunk are 16 x 64 x 64 on operands that sit in registers
// (the state is the accumulator of one product and the A operand of the next); a 5th-generation
// MMA would move each of them through shared or tensor memory, and its smallest tile has eight times
// the rows of a chunk.  Measured on B200: 1020 multiply-adds per clock and multiprocessor, 21 cycles
// from issue to a dependent issue, against 128 per clock of the fp32 pipe.
//
// Fragment layouts (lane = 4 g + t):
//   A (16 x 16)  a0: (g, 2t..2t+1)  a1: (g+8, 2t..)  a2: (g, 2t+8..)  a3: (g+8, 2t+8..)
//   B (16 x 8)   b0: (k = 2t..2t+1, n = g)  b1: (k = 2t+8.., n = g)
//   C (16 x 8)   c0,c1: (g, 2t..2t+1)  c2,c3: (g+8, 2t..)
// so the accumulators of two neighbouring 16 x 8 tiles, packed in pairs, are an A operand.
#pragma once
#include "common.cuh"

namespace srwm {

__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void* row) {
  const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(row));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], const void* row) {
  const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(row));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}

__device__ __forceinline__ void stsm4(void* row, const uint32_t (&r)[4]) {
  const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(row));
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}

// Two finite fp32 values as three packed bf16 pairs, exactly: x = p0 + p1 + p2 (24 significant bits cut into
// 8 + 8 + 8; cutting instead of rounding makes every residual exact and each piece one byte permute).
// Of an infinite value the second piece is NaN, and with it everything a product of pieces puts it into, a zero of the
// other operand included: what uses these products looks for NaN in its results and computes those again without them.
__device__ __forceinline__ u64 sub2(u64 a, u64 b) {
  u64 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ void split3(float x0, float x1, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  const uint32_t u0 = __float_as_uint(x0), u1 = __float_as_uint(x1);
  p0 = __byte_perm(u0, u1, 0x7632);
  float r0, r1, s0, s1;
  unpack2(sub2(pack2(x0, x1), pack2(__uint_as_float(u0 & 0xffff0000u), __uint_as_float(u1 & 0xffff0000u))), r0, r1);
  const uint32_t v0 = __float_as_uint(r0), v1 = __float_as_uint(r1);
  p1 = __byte_perm(v0, v1, 0x7632);
  unpack2(sub2(pack2(r0, r1), pack2(__uint_as_float(v0 & 0xffff0000u), __uint_as_float(v1 & 0xffff0000u))), s0, s1);
  p2 = __byte_perm(__float_as_uint(s0), __float_as_uint(s1), 0x7632);
}

// Two neighbouring accumulator tiles as the three pieces of an A operand.
__device__ __forceinline__ void split_frag(const float (&c0)[4], const float (&c1)[4], uint32_t (&a)[3][4]) {
  split3(c0[0], c0[1], a[0][0], a[1][0], a[2][0]);
  split3(c0[2], c0[3], a[0][1], a[1][1], a[2][1]);
  split3(c1[0], c1[1], a[0][2], a[1][2], a[2][2]);
  split3(c1[2], c1[3], a[0][3], a[1][3], a[2][3]);
}

// d[n] += A B[n] for NT neighbouring tiles, A in NA and B in NB pieces (1: the operand is bf16 exactly;
// 3: fp32).  Products below 2^-24 of the leading one are left out (piece indices above 2 in sum).  The
// small products are summed first -- into `lo`, which may be `d` itself where the sum is one
// instruction deep -- and the leading one last, so that the accumulator's rounding acts on full-size
// values once per 16 terms.  The tiles are the inner loop: an accumulator is used again only after the
// other tiles' instructions.  b[piece][tile]: the two registers of a tile's B operand.
template <int NA, int NB, int NT>
__device__ __forceinline__ void mma_tiles(float (&d)[NT][4], float (&lo)[NT][4], const uint32_t (&a)[NA][4],
                                          const uint32_t (&b)[NB][NT][2]) {
#pragma unroll
  for (int s = 2; s >= 1; --s)
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      const int j = s - i;
      if (j >= 0 && j < NB) {
#pragma unroll
        for (int n = 0; n < NT; ++n) mma16816(lo[n], a[i], b[j][n][0], b[j][n][1]);
      }
    }
#pragma unroll
  for (int n = 0; n < NT; ++n) mma16816(d[n], a[0], b[0][n][0], b[0][n][1]);
}
// B operands of two tiles from one ldmatrix.x4
__device__ __forceinline__ void ldsm_b(uint32_t (&b)[2][2], const void* row) {
  uint32_t r[4];
  ldsm4(r, row);
  b[0][0] = r[0]; b[0][1] = r[1]; b[1][0] = r[2]; b[1][1] = r[3];
}
__device__ __forceinline__ void ldsm_bt(uint32_t (&b)[2][2], const void* row) {
  uint32_t r[4];
  ldsm4_t(r, row);
  b[0][0] = r[0]; b[0][1] = r[1]; b[1][0] = r[2]; b[1][1] = r[3];
}

// 8 x 8 blocks transposed across the warp: (row g, cols 2t..) becomes (row = old col g, old rows 2t..)
__device__ __forceinline__ uint32_t movm(uint32_t a) {
  uint32_t d;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}
// From the A operand of X^T (16 x 16): the A operand of X
__device__ __forceinline__ void transpose_a(const uint32_t (&xt)[4], uint32_t (&x)[4]) {
  x[0] = movm(xt[0]); x[1] = movm(xt[2]); x[2] = movm(xt[1]); x[3] = movm(xt[3]);
}

__device__ __forceinline__ void bar_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int count) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}
// Barrier of `count` threads; true where all came with true.
__device__ __forceinline__ bool bar_all(int id, int count, bool ok) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %3, 0;\n\tbarrier.cta.red.and.pred q, %1, %2, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(id), "r"(count), "r"(ok ? 1 : 0)
      : "memory");
  return r != 0;
}

}  // namespace srwm
