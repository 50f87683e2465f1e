// Delta rule in chunks of 16 steps on the tensor cores (head sizes 16, 32, 64).
//
// With W0 the state before a chunk, k_i, q_i, v_i, b_i its rows and u_i = v_i - v_old_i:
//   (I + L) U = V - K W0           L[i][j] = (k_i.k_j) b_j, j < i      (unit lower triangular)
//   ins_i = b_i u_i                v_old = V - U
//   OUT = Q W0 + tril(Q K^T) INS   W = W0 + K^T INS
// (the WY form of supervised_learning/fast_weight/__init__.py:186-191).  L depends on the inputs
// only, so its inverse is off the chain from chunk to chunk, which is three products long.
//
// Roles.  The E/16 main warps of a CTA hold the state, 16 columns m each, transposed as the
// accumulator fragments of (m x e) tiles: columns never meet, so a main warp never waits for
// another.  Accumulators packed in pairs are the next product's A operand, so the state, U, INS go
// from product to product in registers.  The prep warps run ahead through a ring of slots: rows
// from global memory (cp.async), cut into bf16 pieces, the two 16 x 16 products of the rows and the
// inverse, by forward substitution with one column per lane.  Named barriers hand slots over.
//
// Precision is that of fp32 arithmetic: fp32 operands are three bf16 pieces (mma.cuh), bf16 streams
// one, sums are fp32.
//
// Infinities and NaN.  The pieces of an infinite value, and the zeros of the triangular matrices times what is
// not finite, spread NaN over a chunk, its earlier steps included.  The warps look for what is not finite among their results;
// where there is some, the sequence is run again step by step on the fp32 pipe (delta_*_again), with what arithmetic makes of it.
// 1024 sequences x 1024 steps, E = 64, bf16: forward 0.44 ms, 1.3 with one infinity among them, 5.2 with NaN everywhere;
// backward 1.35, 2.2 and 14.9.
//
// Code size.  All roles of a kernel run at once, and a multiprocessor's instruction cache holds about 2000
// instructions (measured: 1.0 cycle per instruction and scheduler up to 32 KB of straight code, 2.7 beyond
// 40 KB); the loops whose operands come from shared memory are therefore left rolled.
//
// What bounds it at E = 64: the tensor pipe, 112 instructions of a main warp per chunk with bf16 rows
// (57 cycles a step), 192 with fp32 rows.
#pragma once
#include "delta.cuh"
#include "mma.cuh"

namespace srwm {

constexpr int DC = 16;   // steps of a chunk: the side of one MMA tile

template <typename TIO, int E, bool PACKED>
struct DeltaChunk {
  static constexpr int NW = E / 16;                                // main warps (16 columns of the state each)
  static constexpr int NP = (sizeof(TIO) == 4 || PACKED) ? 3 : 1;  // bf16 pieces of a q, k row
  static constexpr int PITCH = E * 2 + 16;                         // bytes of a piece row (ldmatrix without conflicts)
  static constexpr int PIECE = DC * PITCH;
  static constexpr int RSB = (3 * E + 1) * (int)sizeof(TIO);
  static constexpr int PK_PITCH = ((RSB + 30) / 16) * 16;
  static constexpr int FRAG = 3 * 32 * 16;                         // a 16 x 16 operand: 3 pieces x 32 lanes x 4 registers
  static constexpr int VP = E + 4;                                 // floats of a v row (packed form)
  static constexpr int TP = 20;                                    // floats of a row of the triangular scratch
};

// Stage the rows of a chunk (16-byte pieces, 2^lg of them a row) with a pointer that advances with the rows:
// row addresses from 64-bit strides took longer than the copies.  Missing rows become zero.
__device__ __forceinline__ void stage_chunk_rows(unsigned char* dst, int pitch, const char* row0, long long sl, int lg,
                                                 int nt, int lane) {
  const int r0 = lane >> lg, b = (lane & ((1 << lg) - 1)) * 16, rpp = 32 >> lg;
  const char* src = row0 + r0 * sl + b;
  unsigned char* d = dst + r0 * pitch + b;
#pragma unroll 2
  for (int r = r0; r < DC; r += rpp) {
    if (r < nt) cp_async16(d, src);
    else *reinterpret_cast<uint4*>(d) = make_uint4(0u, 0u, 0u, 0u);
    src += rpp * sl;
    d += rpp * pitch;
  }
}

// fp32 rows of a chunk as bf16 pieces in a slot.
template <int E>
__device__ __forceinline__ void rows_to_pieces(const unsigned char* raw, unsigned char* slot, int lane) {
  using D = DeltaChunk<float, E, false>;
#pragma unroll 2
  for (int idx = lane; idx < DC * E / 8; idx += 32) {   // (not unrolled further: see the note on code size)
    const int r = idx / (E / 8), g = idx % (E / 8);
    unsigned char* d = slot + r * D::PITCH + g * 16;
    float x[8];
    ld_vec<8>(reinterpret_cast<const float*>(raw) + r * E + g * 8, x);
    uint32_t p[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) split3(x[2 * j], x[2 * j + 1], p[0][j], p[1][j], p[2][j]);
#pragma unroll
    for (int q = 0; q < 3; ++q)
      *reinterpret_cast<uint4*>(d + q * D::PIECE) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
  }
}

// ... rows and pieces in the same place.
template <int E>
__device__ __forceinline__ void rows_to_pieces_in_place(unsigned char* rows, int lane) {
  using D = DeltaChunk<float, E, false>;
  constexpr int N = DC * E / 8 / 32;
  static_assert(DC * E * 4 <= 3 * D::PIECE && DC * E / 8 % 32 == 0, "rows fit where their pieces go");
  float x[N][8];
#pragma unroll
  for (int i = 0; i < N; ++i) ld_vec<8>(reinterpret_cast<const float*>(rows) + (lane + 32 * i) * 8, x[i]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int idx = lane + 32 * i;
    unsigned char* d = rows + idx / (E / 8) * D::PITCH + idx % (E / 8) * 16;
    uint32_t p[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) split3(x[i][2 * j], x[i][2 * j + 1], p[0][j], p[1][j], p[2][j]);
#pragma unroll
    for (int q = 0; q < 3; ++q)
      *reinterpret_cast<uint4*>(d + q * D::PIECE) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
  }
}

// The layers' preparation of packed rows (delta.cuh), straight into pieces: q, k normalised, v as fp32
// rows, beta; optionally the normalisers for the backward.
template <typename TIO, int E>
__device__ __forceinline__ void packed_to_pieces(const unsigned char* raw, const char* row0, long long stride, float eps,
                                                 unsigned char* sq, unsigned char* sk, float* sv, float* sb,
                                                 float* dsq, float* dsk, int nt, int lane) {
  using D = DeltaChunk<TIO, E, true>;
  constexpr int LPR = E / 4, NG = 32 / LPR, K = DC / NG;
  const int grp = lane / LPR, l = lane % LPR;
#pragma unroll 2
  for (int kk = 0; kk < K; ++kk) {
    const int t = grp + kk * NG;
    const int tc = min(t, nt - 1);
    const bool in = t < nt;
    const int off = (int)(reinterpret_cast<uintptr_t>(row0 + tc * stride) & 15);
    const TIO* r = reinterpret_cast<const TIO*>(raw + tc * D::PK_PITCH + off);
    float q[4], k[4], v[4], s_q = 0.f, s_k = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      q[i] = elu_p1(to_f32(r[l * 4 + i]));
      k[i] = elu_p1(to_f32(r[E + l * 4 + i]));
      v[i] = in ? to_f32(r[2 * E + l * 4 + i]) : 0.f;
      s_q += q[i];
      s_k += k[i];
    }
#pragma unroll
    for (int o = 1; o < LPR; o <<= 1) {
      s_q += __shfl_xor_sync(0xffffffffu, s_q, o);
      s_k += __shfl_xor_sync(0xffffffffu, s_k, o);
    }
    s_q += eps;
    s_k += eps;
    const float iq = in ? __fdividef(1.f, s_q) : 0.f, ik = in ? __fdividef(1.f, s_k) : 0.f;
    uint32_t p[3][2], o[3][2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      split3(q[2 * j] * iq, q[2 * j + 1] * iq, p[0][j], p[1][j], p[2][j]);
      split3(k[2 * j] * ik, k[2 * j + 1] * ik, o[0][j], o[1][j], o[2][j]);
    }
#pragma unroll
    for (int z = 0; z < 3; ++z) {
      *reinterpret_cast<uint2*>(sq + z * D::PIECE + t * D::PITCH + l * 8) = make_uint2(p[z][0], p[z][1]);
      *reinterpret_cast<uint2*>(sk + z * D::PIECE + t * D::PITCH + l * 8) = make_uint2(o[z][0], o[z][1]);
    }
    st_vec<4>(sv + t * D::VP + l * 4, v);
    if (l == 0) {
      sb[t] = in ? fast_sigmoid(to_f32(r[3 * E])) : 0.f;
      if (dsq) { dsq[t] = s_q; dsk[t] = s_k; }
    }
  }
}

// ... of q and k only, from packed rows that lie where q's pieces and k's go.
template <typename TIO, int E>
__device__ __forceinline__ void packed_to_pieces_in_place(unsigned char* sq, unsigned char* sk, const char* row0, long long stride,
                                                          float eps, float* sb, float* norm, int nt, int lane) {
  using D = DeltaChunk<TIO, E, true>;
  constexpr int LPR = E / 4, NG = 32 / LPR, K = DC / NG;
  static_assert(DC * D::PK_PITCH <= 6 * D::PIECE, "rows fit where their pieces go");
  const int grp = lane / LPR, l = lane % LPR;
  float x[K][2][4], b[K];
#pragma unroll
  for (int kk = 0; kk < K; ++kk) {
    const int tc = min(grp + kk * NG, nt - 1), off = (int)(reinterpret_cast<uintptr_t>(row0 + tc * stride) & 15);
    const TIO* r = reinterpret_cast<const TIO*>(sq + tc * D::PK_PITCH + off);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[kk][0][i] = to_f32(r[l * 4 + i]);
      x[kk][1][i] = to_f32(r[E + l * 4 + i]);
    }
    b[kk] = l == 0 ? to_f32(r[3 * E]) : 0.f;
  }
  __syncwarp();
#pragma unroll
  for (int kk = 0; kk < K; ++kk) {
    const int t = grp + kk * NG;
    const bool in = t < nt;
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[kk][w][i] = elu_p1(x[kk][w][i]);
        s += x[kk][w][i];
      }
#pragma unroll
      for (int o = 1; o < LPR; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      s += eps;
      const float is = in ? __fdividef(1.f, s) : 0.f;
      uint32_t p[3][2];
#pragma unroll
      for (int j = 0; j < 2; ++j) split3(x[kk][w][2 * j] * is, x[kk][w][2 * j + 1] * is, p[0][j], p[1][j], p[2][j]);
#pragma unroll
      for (int z = 0; z < 3; ++z)
        *reinterpret_cast<uint2*>((w == 0 ? sq : sk) + z * D::PIECE + t * D::PITCH + l * 8) = make_uint2(p[z][0], p[z][1]);
      if (l == 0) norm[w * DC + t] = s;
    }
    if (l == 0) sb[t] = in ? fast_sigmoid(b[kk]) : 0.f;
  }
}

// lane's row address of an ldmatrix.x4 over a 16 x 16 block of piece rows (block column cb of 16 values):
// matrices in the order (rows 0-7, cols 0-7), (rows 0-7, cols 8-15), (rows 8-15, cols 0-7), (8-15, 8-15)
__device__ __forceinline__ int frag_b_off(int lane, int pitch) {
  return ((lane & 7) + (lane >> 4) * 8) * pitch + ((lane >> 3) & 1) * 16;
}
// ... and (rows 0-7, cols 0-7), (rows 8-15, cols 0-7), (rows 0-7, cols 8-15), (8-15, 8-15)
__device__ __forceinline__ int frag_a_off(int lane, int pitch) {
  return ((lane & 7) + ((lane >> 3) & 1) * 8) * pitch + (lane >> 4) * 16;
}

// C fragments (i = rows, j = columns) of X Y^T, X and Y 16 x E rows in NX and NY pieces.
template <int E, int NX, int NY>
__device__ __forceinline__ void gram(const unsigned char* X, const unsigned char* Y, int pitch, int lane,
                                     float (&c)[2][4]) {
  float hi[2][4] = {}, lo[2][4] = {};
  const int ao = frag_a_off(lane, pitch), bo = frag_b_off(lane, pitch);
  // two at a time where there are few products: 16 values of k alone wait for their loads and one another (backward, bf16:
  // E = 32 565 -> 551 us for 2368 sequences x 512 steps, E = 64 680 -> 672 for 1024); with nine, no gain and more code
  constexpr int AT_ONCE = NX * NY < 9 ? 2 : 1;
#pragma unroll AT_ONCE
  for (int ks = 0; ks < E / 16; ++ks) {
    uint32_t a[NX][4], b[NY][2][2];
#pragma unroll
    for (int p = 0; p < NX; ++p) ldsm4(a[p], X + p * DC * pitch + ao + ks * 32);
#pragma unroll
    for (int p = 0; p < NY; ++p) ldsm_b(b[p], Y + p * DC * pitch + bo + ks * 32);
    mma_tiles<NX, NY, 2>(hi, lo, a, b);
  }
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) c[n][i] = hi[n][i] + lo[n][i];
}

// A 16 x 16 matrix given as C fragments (i, j), stored as the B operand (k = j, n = i) in three pieces.
// Registers of a lane: (i = g: j low, j high), (i = g + 8: j low, j high).
__device__ __forceinline__ void store_frag(unsigned char* dst, const float (&c)[2][4], int lane) {
  uint32_t a[3][4];
  split3(c[0][0], c[0][1], a[0][0], a[1][0], a[2][0]);
  split3(c[1][0], c[1][1], a[0][1], a[1][1], a[2][1]);
  split3(c[0][2], c[0][3], a[0][2], a[1][2], a[2][2]);
  split3(c[1][2], c[1][3], a[0][3], a[1][3], a[2][3]);
#pragma unroll
  for (int p = 0; p < 3; ++p)
    *reinterpret_cast<uint4*>(dst + p * 512 + lane * 16) = make_uint4(a[p][0], a[p][1], a[p][2], a[p][3]);
}
__device__ __forceinline__ void load_frag(const unsigned char* src, int lane, uint32_t (&f)[3][2][2]) {
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const uint4 v = *reinterpret_cast<const uint4*>(src + p * 512 + lane * 16);
    f[p][0][0] = v.x; f[p][0][1] = v.y; f[p][1][0] = v.z; f[p][1][1] = v.w;
  }
}

// (I + L)^-1 - I for the strictly triangular L[i][j] = akk[i][j] b_j (j < i, or j > i with UPPER), as C
// fragments again.  One column of the inverse per lane (the two half warps do the same), by
// substitution: a finished row is subtracted from all later ones, so the chain is one multiply-add per row.
template <bool UPPER>
__device__ __forceinline__ void unit_inverse(float (&akk)[2][4], const float* sb, float* scr, int lane) {
  constexpr int TP = 20;
  const int g = lane / 4, t = lane % 4;
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
      const int j = n * 8 + 2 * t + jj;
      const float b = sb[j];
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {   // scr[j][i] = L[i][j]
        const int i = g + hh * 8;
        scr[j * TP + i] = (UPPER ? j > i : j < i) ? akk[n][2 * hh + jj] * b : 0.f;
      }
    }
  __syncwarp();
  const int c = lane & 15;
  float x[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) x[i] = i == c ? 1.f : 0.f;
#pragma unroll
  for (int s = 0; s < 15; ++s) {
    const int j = UPPER ? 15 - s : s;
#pragma unroll
    for (int i4 = 0; i4 < 4; ++i4) {
      if (UPPER ? i4 * 4 < j : i4 * 4 + 3 > j) {
        const float4 l = *reinterpret_cast<const float4*>(scr + j * TP + i4 * 4);
        const float lv[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
        for (int ii = 0; ii < 4; ++ii)
          if (UPPER ? i4 * 4 + ii < j : i4 * 4 + ii > j) x[i4 * 4 + ii] = fmaf(-lv[ii], x[j], x[i4 * 4 + ii]);
      }
    }
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if (lane < 16) scr[i * TP + c] = x[i] - (i == c ? 1.f : 0.f);
  __syncwarp();
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const float2 v = *reinterpret_cast<const float2*>(scr + (g + hh * 8) * TP + n * 8 + 2 * t);
      akk[n][2 * hh] = v.x;
      akk[n][2 * hh + 1] = v.y;
    }
  __syncwarp();
}

// ---------------------------------------------------------------------------------------
// The ring of prepared chunks, shared by forward and backward (which walks the chunks in reverse).
// ---------------------------------------------------------------------------------------
template <typename TIO, int E, int NPW, int S, bool PACKED, bool BWD>
struct DeltaRing {
  using D = DeltaChunk<TIO, E, PACKED>;
  static constexpr int NP = D::NP, NG = sizeof(TIO) == 4 ? 3 : 1;  // pieces of a q, k row; of an upstream row
  // sets of state warps (backward): products with W and with dL/dW in the same ones, or apart
  static constexpr int SW = E >= 64 ? 1 : 2;
  // Rows go straight to their slot: bf16 rows, as they are, or (IN_PLACE) fp32 and packed rows, cut there.
  static constexpr bool IN_PLACE = BWD && SW == 1 && NP == 3, DIRECT = IN_PLACE || (!PACKED && NP == 1);
  // rows of one prep warp before they are cut into pieces: packed rows, or q | k; backward: go | v_insert
  static constexpr int RG = DC * E * (int)sizeof(TIO), RI = DC * E * 4;
  static constexpr int ORG = PACKED && !IN_PLACE ? DC * D::PK_PITCH : (DIRECT ? 0 : 2 * DC * E * 4);
  static constexpr int ORI = ORG + (BWD && !DIRECT ? RG : 0);
  static constexpr int RAW = ORI + (BWD && !IN_PLACE ? RI : 0);
  // triangular scratch of one prep warp, or its place in a slot, where the inverse will be
  static constexpr bool SLOT_SCR = BWD && SW == 1;
  static constexpr int SCR = SLOT_SCR ? 0 : DC * D::TP * 4;
  // slot: q pieces | k pieces | inverse | masked q.k | beta | (backward) go, v_insert pieces, masked -go.v_insert,
  // masked v_insert.go | (packed form) normalisers of q, of k | v rows
  static constexpr int OQ = 0, OK = NP * D::PIECE, OT = 2 * NP * D::PIECE, OA = OT + D::FRAG, OB = OA + D::FRAG,
                       OG = OB + DC * 4, OI = OG + (BWD ? NG * D::PIECE : 0), OC = OI + (BWD ? 3 * D::PIECE : 0),
                       ON = OC + (BWD ? 2 * D::FRAG : 0),
                       OV = ON + (PACKED ? 2 * DC * 4 : 0);
  static constexpr int SLOT = OV + (PACKED && !IN_PLACE ? DC * D::VP * 4 : 0);   // (v: the chain warps read it themselves)
  static constexpr int BYTES = NPW * (RAW + SCR) + S * SLOT;
  static_assert(!IN_PLACE || NPW == 2, "one half each");
  static_assert(DC * D::TP * 4 <= D::FRAG, "scratch");
  static constexpr int PREP = IN_PLACE ? 2 : 1;                    // prep warps of a slot
  static constexpr int NT = 32 * ((BWD ? 1 + SW : 1) * D::NW + PREP);   // threads that meet at a slot's `empty`
  static constexpr int NM = 32 * (D::NW + PREP), NS = 32 * (SW * D::NW + 1);   // ... at `full` (chain warps), at `full_state`
  static_assert(RAW % 16 == 0 && SLOT % 16 == 0 && SCR % 16 == 0, "16-byte aligned pieces");
  // Named barriers.  The backward's chain warps and its other consumers have a `full` each: at a common one
  // the chain would wait for the warps it should run ahead of.
  // (One set of state warps has what the chain warps leave them as a sign that the slot is full.)
  static constexpr int BARS = (BWD && SW == 2 ? 3 : 2) * S;
  // (with fewer slots than prep warps, two of them would wait for the same slot on one barrier)
  static constexpr int BOTH = 14;                                  // (packed form) the two prep warps of a slot
  static_assert(S >= NPW && BARS + (BWD ? 6 : 0) <= 16, "named barriers");
  static __device__ __forceinline__ int full(int s) { return s; }
  static __device__ __forceinline__ int empty(int s) { return S + s; }
  static __device__ __forceinline__ int full_state(int s) { return 2 * S + s; }
  static __device__ __forceinline__ unsigned char* slot(unsigned char* ring, int s) {
    return ring + NPW * (RAW + SCR) + s * SLOT;
  }
};

// Prep warp pw: places pw, pw + NPW, ... in the order the chunks are walked in (BWD: from the last one).  IN_PLACE: every place, one warp
// what comes from q and k, the other what comes from the upstream rows and v_insert: a place takes half as long, and how long is
// what two slots wait for (fp32 rows, 2368 sequences x 512 steps: 1970 -> 1768 us; with three slots, bf16 rows, 148 sequences 152 -> 162: apart).
template <typename TIO, int E, int NPW, int S, bool PACKED, bool BWD, typename Params>
__device__ __forceinline__ void delta_prep_warp(const Params& p, unsigned char* ring, int pw, int lane, int n, int h) {
  using R = DeltaRing<TIO, E, NPW, S, PACKED, BWD>;
  using D = typename R::D;
  constexpr int NP = R::NP, NT = R::NT, RB = E * (int)sizeof(TIO);
  constexpr bool HALF = R::IN_PLACE;
  constexpr int STEP = HALF ? 1 : NPW;
  const int z0 = HALF ? 2 * pw : 0;   // first of its rows, and of its matrices
  const int L = p.L, nchunks = (L + DC - 1) / DC;
  unsigned char* raw = ring + pw * (R::RAW + R::SCR);
  float* scr = reinterpret_cast<float*>(raw + R::RAW);
  auto chunk_of = [&](int it) { return BWD ? nchunks - 1 - it : it; };
  constexpr int LG = E * sizeof(TIO) == 256 ? 4 : (E * sizeof(TIO) == 128 ? 3 : (E * sizeof(TIO) == 64 ? 2 : 1));
  constexpr int LGF = E == 64 ? 4 : (E == 32 ? 3 : 2);   // of fp32 rows
  auto stage = [&](int it) {
    if (it >= nchunks) return;
    const int t0 = chunk_of(it) * DC, nt = min(DC, L - t0);
    if (SRWM_BAD_ROWS(p.dbg, BWD ? 13 : 10, t0, nt, L, DC)) return;
    unsigned char* d = R::slot(ring, it % S);
    if (R::DIRECT && it >= S) bar_sync(R::empty(it % S), NT);
    if constexpr (PACKED) {
      if (!HALF || pw == 0) stage_packed_rows<D::RSB, D::PK_PITCH, 32>(HALF ? d + R::OQ : raw, p.Q.row(n, h, t0), p.Q.sl, nt, lane);
    }
    // q, k, upstream rows, v_insert: one copy of the code for all
#pragma unroll 1
    for (int z = PACKED ? 2 : z0; z < (HALF ? z0 + 2 : (BWD ? 4 : 2)); ++z) {
      const SeqView* v = z == 0 ? &p.Q : &p.K;
      unsigned char* to = R::DIRECT ? d + (z == 0 ? R::OQ : R::OK) : raw + z * DC * RB;
      int pitch = R::DIRECT && NP == 1 ? D::PITCH : RB, lg = LG;
      if constexpr (BWD) {
        if (z == 2) { v = &p.gout; to = R::DIRECT ? d + R::OG : raw + R::ORG; pitch = R::DIRECT && R::NG == 1 ? D::PITCH : RB; }
        if (z == 3) { v = &p.v_ins; to = R::IN_PLACE ? d + R::OI : raw + R::ORI; pitch = E * 4; lg = LGF; }
      }
      stage_chunk_rows(to, pitch, v->row(n, h, t0), v->sl, lg, nt, lane);
    }
  };
  TIO bt;   // (converted when it is used: a conversion here would wait for the load)
  auto beta_ld = [&](int it) {
    from_f32(bt, 0.f);
    if (PACKED || it >= nchunks || (HALF && pw != 0)) return;
    const int tt = chunk_of(it) * DC + lane;
    if (lane < DC && tt < L) bt = *reinterpret_cast<const TIO*>(p.beta.row(n, h, tt));
  };
  from_f32(bt, 0.f);
  for (int it = HALF ? -1 : pw - NPW; it < nchunks; it += STEP) {   // the first round only stages
    const bool first = it < 0;
    const int s = first ? 0 : it % S, t0 = first ? 0 : chunk_of(it) * DC, nt = min(DC, L - t0);
    unsigned char* slot = R::slot(ring, s);
    unsigned char *sq = slot + R::OQ, *sk = slot + R::OK;
    float* sb = reinterpret_cast<float*>(slot + R::OB);
    if (!first) {
      cp_async_wait<0>();
      __syncwarp();
      if (!R::DIRECT && it >= S) bar_sync(R::empty(s), NT);
      if constexpr (PACKED && HALF) {
        if (pw == 0)
          packed_to_pieces_in_place<TIO, E>(sq, sk, p.Q.row(n, h, t0), p.Q.sl, p.eps, sb, reinterpret_cast<float*>(slot + R::ON), nt, lane);
      } else if constexpr (PACKED) {
        float* norm = BWD ? reinterpret_cast<float*>(slot + R::ON) : nullptr;
        packed_to_pieces<TIO, E>(raw, p.Q.row(n, h, t0), p.Q.sl, p.eps, sq, sk, reinterpret_cast<float*>(slot + R::OV), sb,
                                 norm, BWD ? norm + DC : nullptr, nt, lane);
      } else {
        if (lane < DC && (!HALF || pw == 0)) sb[lane] = to_f32(bt);
      }
      if constexpr (R::SLOT_SCR) scr = reinterpret_cast<float*>(slot + R::OT);
      // fp32 rows to pieces: q, k (unless prepared above), v_insert, upstream rows
      if constexpr (R::IN_PLACE) {
#pragma unroll 1
        for (int z = PACKED ? (R::NG == 3 ? 2 : 3) : z0; z < z0 + 2; ++z)
          rows_to_pieces_in_place<E>(slot + (z == 0 ? R::OQ : (z == 1 ? R::OK : (z == 2 ? R::OG : R::OI))), lane);
      } else
#pragma unroll 1
      for (int z = (PACKED || R::DIRECT) ? 2 : 0; z < (BWD ? (!R::DIRECT && R::NG == 3 ? 4 : 3) : 2); ++z)
        rows_to_pieces<E>(z < 2 ? raw + z * DC * RB : raw + (z == 2 ? R::ORI : R::ORG),
                          slot + (z == 0 ? R::OQ : (z == 1 ? R::OK : (z == 2 ? R::OI : R::OG))), lane);
      if constexpr (BWD && !R::DIRECT && R::NG == 1) {
        for (int i = lane; i < DC * E / 8; i += 32) {
          const int r = i / (E / 8), b = (i % (E / 8)) * 16;
          *reinterpret_cast<uint4*>(slot + R::OG + r * D::PITCH + b) = *reinterpret_cast<const uint4*>(raw + R::ORG + r * RB + b);
        }
      }
      __syncwarp();
    }
    if constexpr (!R::DIRECT) {
      stage(it + STEP);   // the raw rows have been read
      cp_async_commit();
    }
    beta_ld(it + STEP);
    // The 16 x 16 matrices: k.k and its inverse; forward: q_i.k_j, j <= i; backward: k_i.q_j, j >= i, then
    // -go_i.v_insert_j, j > i, and v_insert_i.go_j, j >= i
    // (packed form, two warps a slot: q and k take longer, so the other warp has three of the four)
    unsigned char *sg = slot + R::OG, *si = slot + R::OI;
    if constexpr (PACKED && HALF) {
      if (!first) bar_sync(R::BOTH, 64);
    }
#pragma unroll 1
    for (int z = first ? 4 : (HALF && PACKED ? pw : (HALF ? z0 : 0)); z < (HALF ? (PACKED ? 1 + 3 * pw : z0 + 2) : (BWD ? 4 : 2)); ++z) {
      float m[2][4];
      if (z < 2 || (NP == 3 && R::NG == 3)) {
        const unsigned char *x = z == 0 ? sk : (BWD ? (z == 1 ? sk : (z == 2 ? sg : si)) : sq);
        const unsigned char *y = z == 0 ? sk : (BWD ? (z == 1 ? sq : (z == 2 ? si : sg)) : sk);
        gram<E, NP, NP>(x, y, D::PITCH, lane, m);
      } else if constexpr (BWD && !(NP == 3 && R::NG == 3)) {
        if (z == 2) gram<E, R::NG, 3>(sg, si, D::PITCH, lane, m);
        else gram<E, 3, R::NG>(si, sg, D::PITCH, lane, m);
      }
      if (z == 0) {
        unit_inverse<BWD>(m, sb, scr, lane);
      } else {
        const int g = lane / 4, t = lane % 4;
#pragma unroll
        for (int nn = 0; nn < 2; ++nn)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int d = (nn * 8 + 2 * t + (i & 1)) - (g + (i >> 1) * 8);   // column - row
            if (BWD ? d < (z == 2 ? 1 : 0) : d > 0) m[nn][i] = 0.f;
            if (BWD && z == 2) m[nn][i] = -m[nn][i];
          }
      }
      store_frag(slot + (z == 0 ? R::OT : (z == 1 ? R::OA : R::OC + (z - 2) * D::FRAG)), m, lane);
    }
    if (!first) {
      bar_arrive(R::full(s), R::NM);
      if constexpr (BWD && R::SW == 2) bar_arrive(R::full_state(s), R::NS);
    }
    if constexpr (R::DIRECT) {
      stage(it + STEP);   // waits for its slot
      cp_async_commit();
    }
  }
  cp_async_wait<0>();
}

// Rows of a sequence, one after the other (its parameters are read once: a function of its own finds them far away).
struct RowWalk {
  char* p;
  long long step;
  __device__ __forceinline__ RowWalk(const SeqView& v, int n, int h, int t, bool back) : p(v.row(n, h, t)), step(back ? -v.sl : v.sl) {}
  template <typename T>
  __device__ __forceinline__ T* next() {
    T* r = reinterpret_cast<T*>(p);
    p += step;
    return r;
  }
};

// The next row as fp32 values: plain rows, or the layers' preparation of a packed one (delta.cuh).  All lanes of a warp
// take part; lane l gives the values e = l, l + 32, ... of each.
template <typename TIO, int E, bool PACKED>
struct DeltaRow {
  static constexpr int NV = (E + 31) / 32;
  float q[NV], k[NV], v[NV], beta, s_q, s_k;
  __device__ __forceinline__ void load(RowWalk& wq, RowWalk& wk, RowWalk& wv, RowWalk& wb, float eps, int lane) {
    const TIO* r = wq.next<TIO>();
    const TIO* rk = PACKED ? r + E : wk.next<TIO>();
    const TIO* rv = PACKED ? r + 2 * E : wv.next<TIO>();
    beta = to_f32(PACKED ? r[3 * E] : *wb.next<TIO>());
    s_q = s_k = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int e = lane + 32 * i;
      q[i] = k[i] = v[i] = 0.f;
      if (e >= E) continue;
      q[i] = to_f32(r[e]); k[i] = to_f32(rk[e]); v[i] = to_f32(rv[e]);
      if constexpr (PACKED) {
        q[i] = elu_p1(q[i]); k[i] = elu_p1(k[i]);
        s_q += q[i];
        s_k += k[i];
      }
    }
    if constexpr (PACKED) {
      beta = fast_sigmoid(beta);
      s_q = allreduce_warp(s_q) + eps;
      s_k = allreduce_warp(s_k) + eps;
      const float iq = __fdividef(1.f, s_q), ik = __fdividef(1.f, s_k);
#pragma unroll
      for (int i = 0; i < NV; ++i) { q[i] *= iq; k[i] *= ik; }
    }
  }
};

// ---------------------------------------------------------------------------------------
// Forward
// ---------------------------------------------------------------------------------------
// Columns m0 .. m0 + 15 of the state once more, a step at a time: lane = column, and which half of the rows e.
template <typename TIO, int E, bool PACKED>
__device__ __noinline__ void delta_fwd_again(const DeltaFwdParams& p, int n, int h, int m0, int lane) {
  constexpr int HALF = E / 2;
  using Row = DeltaRow<TIO, E, PACKED>;
  const int m = m0 + (lane & 15), e0 = (lane >> 4) * HALF;
  const bool save = !(p.flags & 1u);
  const int L = p.L;
  const float eps = p.eps;
  RowWalk wq(p.Q, n, h, 0, false), wk(p.K, n, h, 0, false), wv(p.V, n, h, 0, false), wb(p.beta, n, h, 0, false),
      wo(p.out, n, h, 0, false), wvo(p.v_old, n, h, 0, false), wvi(p.v_ins, n, h, 0, false);
  float W[HALF], *Wg = p.W.mat(n, h);
#pragma unroll
  for (int i = 0; i < HALF; ++i) W[i] = (PACKED && (p.flags & F_ZERO_INIT)) ? 0.f : Wg[(e0 + i) * E + m];
#pragma unroll 1
  for (int t = 0; t < L; ++t) {
    Row r;
    r.load(wq, wk, wv, wb, eps, lane);
    auto at = [&](const float (&x)[Row::NV], int e) { return __shfl_sync(0xffffffffu, x[Row::NV > 1 ? e / 32 : 0], e % 32); };
    // (a lane's half may lie in the other register of the row: both are read, and one is taken)
    auto mine = [&](const float (&x)[Row::NV], int i) {
      const float a = at(x, i), b = at(x, HALF + i);
      return lane < 16 ? a : b;
    };
    const float v0 = __shfl_sync(0xffffffffu, r.v[0], m % 32), v1 = __shfl_sync(0xffffffffu, r.v[Row::NV - 1], m % 32);
    const float v = m < 32 ? v0 : v1;
    float k[HALF], vold = 0.f, o = 0.f;
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      k[i] = mine(r.k, i);
      vold = fmaf(k[i], W[i], vold);
    }
    vold += __shfl_xor_sync(0xffffffffu, vold, 16);
    const float ins = r.beta * (v - vold);
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      W[i] = fmaf(k[i], ins, W[i]);
      o = fmaf(mine(r.q, i), W[i], o);
    }
    o += __shfl_xor_sync(0xffffffffu, o, 16);
    TIO* ro = wo.next<TIO>();
    float *rvo = wvo.next<float>(), *rvi = wvi.next<float>();
    if (lane < 16) {
      from_f32(ro[m], o);
      if (save) {
        rvo[m] = vold;
        rvi[m] = ins;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < HALF; ++i) Wg[(e0 + i) * E + m] = W[i];
}

template <typename TIO, int E, int NPW, int S, int MINB, bool PACKED>
__global__ void __launch_bounds__(32 * (E / 16 + NPW), MINB) delta_fwd_chunk_kernel(const __grid_constant__ DeltaFwdParams p) {
  using D = DeltaChunk<TIO, E, PACKED>;
  using R = DeltaRing<TIO, E, NPW, S, PACKED, false>;
  constexpr int NW = D::NW, NP = D::NP, NT = R::NT;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int n = blockIdx.x / p.H, h = blockIdx.x % p.H;
  const int L = p.L, nchunks = (L + DC - 1) / DC;
  extern __shared__ __align__(16) unsigned char smem[];
  if (warp >= NW) {
    delta_prep_warp<TIO, E, NPW, S, PACKED, false>(p, smem, warp - NW, lane, n, h);
    return;
  }

  // ---- main warp: columns m0 .. m0 + 15 of the state ---------------------------------------------
  const int g = lane / 4, t = lane % 4, m0 = warp * 16;
  const bool save = !(p.flags & 1u);
  float W[E / 8][4];   // (m = m0 + g, m0 + g + 8) x (e = 8 j + 2 t, + 1)
  float* Wg = p.W.mat(n, h);
#pragma unroll
  for (int j = 0; j < E / 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      W[j][i] = (PACKED && (p.flags & F_ZERO_INIT)) ? 0.f : Wg[(8 * j + 2 * t + (i & 1)) * E + m0 + g + (i >> 1) * 8];

  // this lane's steps of a chunk: 2t, 2t+1, 2t+8, 2t+9 (columns of the 16 x 16 tiles); value (nn, i) of a
  // pair of tiles is (step nn*8 + 2t + (i&1), column g + (i>>1)*8)
  auto step_of = [&](int nn, int i) { return nn * 8 + 2 * t + (i & 1); };
  // one pointer per stream to this lane's step 2t, column m0 + g; the other steps are fixed multiples away
  const char* vp = PACKED ? nullptr : p.V.row(n, h, 2 * t) + (m0 + g) * sizeof(TIO);
  char* op = p.out.row(n, h, 2 * t) + (m0 + g) * sizeof(TIO);
  char* vop = save ? p.v_old.row(n, h, 2 * t) + (m0 + g) * 4 : nullptr;
  char* vip = save ? p.v_ins.row(n, h, 2 * t) + (m0 + g) * 4 : nullptr;
  TIO vr[2][4];   // (converted when used: a conversion here would wait for the loads)
  auto load_v = [&](int c) {
    if constexpr (!PACKED) {
      const int left = SRWM_BAD_ROWS(p.dbg, 11, c * DC, min(DC, L - c * DC), L, DC) ? 0 : L - c * DC - 2 * t;
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
          const TIO* r = reinterpret_cast<const TIO*>(vp + (nn * 8 + jj) * p.V.sl);
          from_f32(vr[nn][jj], 0.f);
          from_f32(vr[nn][2 + jj], 0.f);
          if (nn * 8 + jj < left) {
            vr[nn][jj] = r[0];
            vr[nn][2 + jj] = r[8];
          }
        }
      vp += DC * p.V.sl;
    }
  };
  load_v(0);
  float finite = 0.f;   // 0 while this warp's results are
  const int bo = frag_b_off(lane, D::PITCH), ko = frag_a_off(lane, D::PITCH);
  for (int c = 0; c < nchunks; ++c) {
    const int s = c % S, t0 = c * DC, nt = min(DC, L - t0);
    const unsigned char* slot = R::slot(smem, s);
    const unsigned char *sq = slot + R::OQ, *sk = slot + R::OK;
    bar_sync(R::full(s), R::NM);
    // K W0 and Q W0, transposed: (m x steps)
    float kq[4][4] = {}, kql[4][4] = {};   // tiles: K W0 of steps 0-7, 8-15, then Q W0
#pragma unroll
    for (int ks = 0; ks < E / 16; ++ks) {
      uint32_t a[3][4], b[NP][4][2];
      split_frag(W[2 * ks], W[2 * ks + 1], a);
#pragma unroll
      for (int z = 0; z < NP; ++z) {
        uint32_t r[2][2];
        ldsm_b(r, sk + z * D::PIECE + bo + ks * 32);
        b[z][0][0] = r[0][0]; b[z][0][1] = r[0][1]; b[z][1][0] = r[1][0]; b[z][1][1] = r[1][1];
        ldsm_b(r, sq + z * D::PIECE + bo + ks * 32);
        b[z][2][0] = r[0][0]; b[z][2][1] = r[0][1]; b[z][3][0] = r[1][0]; b[z][3][1] = r[1][1];
      }
      mma_tiles<3, NP, 4>(kq, kql, a, b);
    }
    float v[2][4];
    const float* sv = reinterpret_cast<const float*>(slot + R::OV);
#pragma unroll
    for (int nn = 0; nn < 2; ++nn)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        v[nn][i] = PACKED ? sv[step_of(nn, i) * D::VP + m0 + g + (i >> 1) * 8] : to_f32(vr[nn][i]);
    if (c + 1 < nchunks) load_v(c + 1);
    // U = (V - K W0) + ((I + L)^-1 - I) (V - K W0)
    float u[2][4], ins[2][4], vold[2][4];
    uint32_t a[3][4], f[3][2][2];
#pragma unroll
    for (int nn = 0; nn < 2; ++nn)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        vold[nn][i] = kq[nn][i] + kql[nn][i];
        u[nn][i] = v[nn][i] - vold[nn][i];
      }
    split_frag(u[0], u[1], a);
    load_frag(slot + R::OT, lane, f);
    const float* sb = reinterpret_cast<const float*>(slot + R::OB);
    {
      float hi[2][4] = {}, lo[2][4] = {};
      mma_tiles<3, 3, 2>(hi, lo, a, f);
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float dl = hi[nn][i] + lo[nn][i];
          u[nn][i] += dl;
          vold[nn][i] -= dl;
          ins[nn][i] = u[nn][i] * sb[step_of(nn, i)];
        }
    }
    split_frag(ins[0], ins[1], a);
    // W += K^T INS, transposed: INS^T (m x steps) times K (steps x e)
#pragma unroll
    for (int j4 = 0; j4 < (E + 31) / 32; ++j4) {
      constexpr int NTL = E >= 32 ? 4 : 2;
      uint32_t b[NP][NTL][2];
#pragma unroll
      for (int z = 0; z < NP; ++z)
#pragma unroll
        for (int hh = 0; hh < NTL / 2; ++hh) {
          uint32_t r[2][2];
          ldsm_bt(r, sk + z * D::PIECE + ko + (j4 * 2 + hh) * 32);
          b[z][2 * hh][0] = r[0][0]; b[z][2 * hh][1] = r[0][1];
          b[z][2 * hh + 1][0] = r[1][0]; b[z][2 * hh + 1][1] = r[1][1];
        }
      float d[NTL][4] = {};
      mma_tiles<3, NP, NTL>(d, d, a, b);
#pragma unroll
      for (int q = 0; q < NTL; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) W[j4 * 4 + q][i] += d[q][i];
    }
    // OUT = Q W0 + tril(Q K^T) INS
    load_frag(slot + R::OA, lane, f);
    float o[2][4], ol[2][4];
#pragma unroll
    for (int nn = 0; nn < 2; ++nn)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        o[nn][i] = kq[2 + nn][i];
        ol[nn][i] = kql[2 + nn][i];
      }
    mma_tiles<3, 3, 2>(o, ol, a, f);
    if (c + S < nchunks) bar_arrive(R::empty(s), NT);
    // the eight lanes of a step write 32 (16 for bf16) contiguous bytes
    const int left = SRWM_BAD_ROWS(p.dbg, 12, t0, nt, L, DC) ? 0 : nt - 2 * t;
#pragma unroll
    for (int nn = 0; nn < 2; ++nn)
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        const int k = nn * 8 + jj;
        if (k < left) {
          TIO* y = reinterpret_cast<TIO*>(op + k * p.out.sl);
          const float y0 = o[nn][jj] + ol[nn][jj], y8 = o[nn][2 + jj] + ol[nn][2 + jj];
          finite = fmaf(0.f, y0 + y8, finite);
          from_f32(y[0], y0);
          from_f32(y[8], y8);
          if (save) {
            float* vo = reinterpret_cast<float*>(vop + k * p.v_old.sl);
            float* vi = reinterpret_cast<float*>(vip + k * p.v_ins.sl);
            vo[0] = vold[nn][jj];
            vo[8] = vold[nn][2 + jj];
            vi[0] = ins[nn][jj];
            vi[8] = ins[nn][2 + jj];
          }
        }
      }
    op += DC * p.out.sl;
    vop += DC * p.v_old.sl;
    vip += DC * p.v_ins.sl;
  }
#pragma unroll
  for (int j = 0; j < E / 8; ++j) finite = fmaf(0.f, (W[j][0] + W[j][1]) + (W[j][2] + W[j][3]), finite);
  if (__any_sync(0xffffffffu, !(finite == 0.f))) {
    delta_fwd_again<TIO, E, PACKED>(p, n, h, m0, lane);
    return;
  }
#pragma unroll
  for (int j = 0; j < E / 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) Wg[(8 * j + 2 * t + (i & 1)) * E + m0 + g + (i >> 1) * 8] = W[j][i];
}

// ---------------------------------------------------------------------------------------
// Backward.  With G = dL/dW after the chunk, W the state after it, g_i the upstream rows:
//   (I + U) R = K G + triu(K Q^T) GO        U[i][j] = (k_i.k_j) b_j, j > i ;  gv_i = b_i r_i
//   gb_i = r_i.(v_i - v_old_i)
//   GQ = GO W^T - triu(GO INS^T, 1) K
//   GK = INS G^T - GV W^T + triu(INS GO^T) Q + [triu(GV INS^T) - triu(INS GV^T, 1)] K
//   G += Q^T GO - K^T GV ;  W -= K^T INS      (the state before the chunk, rebuilt)
// Only R, GV and G's update are on the chain from chunk to chunk, and they keep to columns m.  So four
// roles: chain warps own 16 columns m of G; W warps own 16 rows e of W, G warps 16 rows e of a copy of G,
// which makes GQ, GK complete sums within a warp (they contract over m; GK's two parts are added through
// shared memory), and take GV from the chain warps as bf16 pieces in shared memory; prep warps as in
// the forward.  Measured for 1024 sequences x 2048 steps, bf16, d_head 64, on the way here: one set of
// warps doing everything (partial GQ, GK exchanged, state transposed by movmatrix; 0.9 KB of spills a
// thread) 3.7 ms, W and G rows in the same warps 3.3 ms.
//
// E = 64 (DeltaRing::SW = 1).  Bound by latency: one sequence a multiprocessor, which is what the registers of 14 warps
// allow, leaves the tensor pipe and the issue slots half idle.  So two sequences, 10 warps of 96 registers each: the state warps make
// GQ and GK both; the copy of G is replaced by the pieces that the chain warps cut G into anyway, through shared memory (an
// eighth less tensor work); W and G are in tensor memory, whose 16 x 256-bit shape is the accumulators' own layout, two tiles
// at a time in registers; INS GV^T, which needs a barrier between the state warps, comes from the chain warps as four sums.
// bf16 rows, 2368 sequences x 512 steps, us: apart 1585; together, the state in registers (a quarter KB of spills) 1426; W in tensor
// memory 1344; G too 1318; a third slot 1262; INS GV^T by the chain warps 1214.  592 sequences 439 -> 357, 148 (one each) 154 -> 153.
// fp32 rows are cut in the slot that they are copied to (34 KB; two slots for two sequences): 256 sequences x 256 steps, us, register
// tiles 160 -> 123; 2368: 1011 -> 886; 148 (chunks before, too) 84 -> 78.
// Packed rows likewise; the chain warps read v themselves, and the state warps finish the rows where they are: the dot products with
// q and k go through shared memory, the values of q and k are in the operands.  256 sequences x 256 steps, us, register tiles
// 201 -> 160 (fp32), 197 -> 147 (bf16; with two of the four matrices of a slot in each prep warp, not one and three, 154).
// Not at E = 32 (bf16, 2368 sequences, 601 -> 639 with the state in registers: two sequences, 16 warps, fit as it is).
// ---------------------------------------------------------------------------------------
// Warps to roles.  A multiprocessor's four schedulers take the warps in turn: chain warps first, then G and
// W warps so that each scheduler has a like share of the tensor work, prep warps last.
template <typename TIO, int E, int NPW, bool PACKED>
struct DeltaBwdRoles {
  static constexpr int NW = E / 16, SW = DeltaRing<TIO, E, NPW, NPW, PACKED, true>::SW;
  static constexpr int WARPS = (1 + SW) * NW + NPW;
};

template <typename TIO, int E, int NPW, int S, bool PACKED>
struct DeltaChunkBwdSmem {
  using R = DeltaRing<TIO, E, NPW, S, PACKED, true>;
  static constexpr int NW = E / 16;
  static constexpr int GV = 3 * R::D::PIECE;                        // one buffer of -gv pieces, laid out like the slots'
  static constexpr int SP = 24, XP = E + 8;                         // float pitches (64-bit accesses without conflicts)
  static constexpr int OGV = (R::BYTES + 15) / 16 * 16;             // two buffers of -gv
  static constexpr int OS = OGV + 2 * GV;                           // -INS GV^T: [KH][16][SP]
  static constexpr int KH = NW >= 4 ? 2 : 1;                        // ... as KH sums over parts of m
  // (one set of state warps: -GV INS^T as NW sums, see part_at)
  static constexpr int OB = OS + (R::SW == 1 ? NW * DC * DC : KH * DC * SP) * 4;                  // partial gbeta: [2][NW][16]
  static constexpr int OK = OB + 2 * NW * DC * 4;                   // the W warps' part of gk: [NW][32 lanes][8]
  static constexpr int OX = OK + (R::SW == 2 ? NW * 32 * 8 * 4 : 0);   // packed form: gq, gk rows [2][16][XP]
  static constexpr int GP = E * R::D::PITCH;                        // a piece of dL/dW, transposed (one set of state warps)
  static constexpr int OP = OX + (PACKED ? (R::SW == 1 ? 2 * DC * NW * 4 : 2 * DC * XP * 4) : 0);   // (SW = 1: dot products [2][16][NW])
  static constexpr int OTM = OP + 3 * GP;                           // address of W and dL/dW in tensor memory
  static constexpr int TOTAL = R::SW == 1 ? OTM + 16 : OP;
  // named barriers after those of the ring
  static constexpr int GV_FULL = R::BARS, GV_EMPTY = GV_FULL + 2, IGV = GV_FULL + 4, GK = IGV + 1, ROWS = IGV + 2;
  static constexpr int GP_FULL = GK, GP_EMPTY = IGV + 2, PARTS = IGV, DOTS = IGV + 3;   // (one set of state warps)
  static constexpr int LAST = 15;                                   // all threads, once: were all results finite
  static_assert(R::SW == 1 ? (PACKED ? DOTS : GP_EMPTY) < (PACKED ? R::BOTH : LAST) : (PACKED ? ROWS : GK) < LAST, "named barriers");
  static constexpr int NGV = 32 * NW * (1 + R::SW);                 // threads that meet at a buffer of -gv
  // delta_bwd_again reuses the memory: dL/dW (rows of E + 4), two steps' five rows, four more rows
  static constexpr int AGAIN = (E * (E + 4) + 2 * (5 * E + 4) + 4 * E + 4) * 4;
  static_assert(AGAIN <= TOTAL, "the second run's rows");
};

// The sequence once more, a step at a time from W_L, which nobody has written over.  (A run that has gone to NaN altogether should
// not take an age for its last steps: four lanes share a row of W and dL/dW, in registers, and the last warp but one reads
// two steps ahead.)
template <typename TIO, int E, bool PACKED, int P, int BAR>
__device__ __noinline__ void delta_bwd_again(const DeltaBwdParams& p, int n, int h) {
  extern __shared__ __align__(16) unsigned char smem[];
  using Row = DeltaRow<TIO, E, PACKED>;
  constexpr int LD = E + 4, Q4 = E / 4, ROWS = 5 * E + 4;   // q | k | go | ins | v - v_old | beta, sums of q and k
  static_assert(P >= 4 * E + 64, "threads: four a row, a warp that fetches, one for the sums");
  const int tid = threadIdx.x, lane = tid % 32, row = tid / 4, part = (tid % 4) * Q4;
  const bool owns = tid < 4 * E, fetches = tid / 32 == P / 32 - 2, sums = tid >= P - 32;
  float *G = reinterpret_cast<float*>(smem), *rows = G + E * LD, *ru = rows + 2 * ROWS, *gv = ru + E, *gq = gv + E, *gk = gq + E,
        *gb = gk + E;
  const int last = p.L - 1;
  const float eps = p.eps;
  RowWalk wq(p.Q, n, h, last, true), wk(p.K, n, h, last, true), wv(p.V, n, h, last, true), wb(p.beta, n, h, last, true),
      wg(p.gout, n, h, last, true), wvo(p.v_old, n, h, last, true), wvi(p.v_ins, n, h, last, true), ogq(p.gQ, n, h, last, true),
      ogk(p.gK, n, h, last, true), ogv(p.gV, n, h, last, true), ogb(p.gbeta, n, h, last, true);
  auto add4 = [](float s) {
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    return s + __shfl_xor_sync(0xffffffffu, s, 2);
  };
  Row r;
  float go_r[Row::NV], vo_r[Row::NV], vi_r[Row::NV];
  auto fetch = [&]() {
    const TIO* g = wg.next<TIO>();
    const float *vo = wvo.next<float>(), *vi = wvi.next<float>();
    r.load(wq, wk, wv, wb, eps, lane);
#pragma unroll
    for (int i = 0; i < Row::NV; ++i) {
      const int e = lane + 32 * i;
      if (e >= E) continue;
      go_r[i] = to_f32(g[e]); vo_r[i] = vo[e]; vi_r[i] = vi[e];
    }
  };
  auto put = [&](int t) {
    float* d = rows + (t & 1) * ROWS;
#pragma unroll
    for (int i = 0; i < Row::NV; ++i) {
      const int e = lane + 32 * i;
      if (e >= E) continue;
      d[e] = r.q[i]; d[E + e] = r.k[i]; d[2 * E + e] = go_r[i]; d[3 * E + e] = vi_r[i]; d[4 * E + e] = r.v[i] - vo_r[i];
    }
    if (lane == 0) { d[5 * E] = r.beta; d[5 * E + 1] = r.s_q; d[5 * E + 2] = r.s_k; }
  };
  float w[Q4], x[Q4];   // this lane's share of a row of W and of dL/dW, which lies in shared memory too
  float *Wg = p.W.mat(n, h) + row * E + part, *Gs = G + row * LD + part;
  if (owns) {
#pragma unroll
    for (int i = 0; i < Q4; ++i) {
      w[i] = Wg[i];
      Gs[i] = x[i] = 0.f;
    }
  }
  if (fetches && last >= 0) {   // (an empty sequence has no rows, though its state may be anything)
    fetch();
    put(last);
    if (last > 0) fetch();
  }
  bar_sync(BAR, P);
#pragma unroll 1
  for (int t = last; t >= 0; --t) {
    const float *q = rows + (t & 1) * ROWS, *k = q + E, *go = k + E, *ins = go + E, *u = ins + E, *one = u + E;
    if (owns) {   // a row of W, a column of G
      float s = 0.f, c = 0.f, go_p[Q4], q_p[Q4], k_p[Q4];
      ld_vec<Q4>(go + part, go_p);
      ld_vec<Q4>(q + part, q_p);
      ld_vec<Q4>(k + part, k_p);
      const float go_c = go[row], q_c = q[row];
#pragma unroll
      for (int i = 0; i < Q4; ++i) {
        s = fmaf(w[i], go_p[i], s);
        c = fmaf(k_p[i], fmaf(q_p[i], go_c, G[(part + i) * LD + row]), c);
        x[i] = fmaf(q_c, go_p[i], x[i]);
      }
      s = add4(s);
      c = add4(c);
      if (tid % 4 == 0) {
        gq[row] = s;
        gv[row] = one[0] * c;
        ru[row] = c * u[row];
      }
    } else if (fetches && t > 0) {
      put(t - 1);
      if (t > 1) fetch();
    }
    bar_sync(BAR, P);
    if (owns) {
      float s = 0.f, gv_p[Q4], in_p[Q4];
      ld_vec<Q4>(gv + part, gv_p);
      ld_vec<Q4>(ins + part, in_p);
      const float k_c = k[row];
#pragma unroll
      for (int i = 0; i < Q4; ++i) {
        w[i] = fmaf(-k_c, in_p[i], w[i]);
        s = fmaf(w[i], -gv_p[i], fmaf(x[i], in_p[i], s));
        x[i] = fmaf(k_c, -gv_p[i], x[i]);
      }
      st_vec<Q4>(Gs, x);
      s = add4(s);
      if (tid % 4 == 0) gk[row] = s;
    } else if (sums) {
      float s = 0.f;
      for (int m = lane; m < E; m += 32) s += ru[m];
      s = allreduce_warp(s);
      if (lane == 0) *gb = s;
    }
    bar_sync(BAR, P);
    if (sums) {
      if constexpr (PACKED) {   // back through the preparation, see delta_bwd_state_warp
        float dq = 0.f, dk = 0.f;
        for (int e = lane; e < E; e += 32) {
          dq = fmaf(gq[e], q[e], dq);
          dk = fmaf(gk[e], k[e], dk);
        }
        dq = allreduce_warp(dq);
        dk = allreduce_warp(dk);
        const float bt = one[0], Sq = one[1], Sk = one[2], iq = __fdividef(1.f, Sq), ik = __fdividef(1.f, Sk);
        TIO* y = ogq.next<TIO>();
        for (int e = lane; e < E; e += 32) {
          const float aq = q[e] * Sq, ak = k[e] * Sk;
          from_f32(y[e], (gq[e] - dq) * iq * (aq > 1.f ? 1.f : aq));
          from_f32(y[E + e], (gk[e] - dk) * ik * (ak > 1.f ? 1.f : ak));
          from_f32(y[2 * E + e], gv[e]);
        }
        if (lane == 0) from_f32(y[3 * E], *gb * bt * (1.f - bt));
      } else {
        TIO *yq = ogq.next<TIO>(), *yk = ogk.next<TIO>(), *yv = ogv.next<TIO>(), *yb = ogb.next<TIO>();
        for (int e = lane; e < E; e += 32) {
          from_f32(yq[e], gq[e]);
          from_f32(yk[e], gk[e]);
          from_f32(yv[e], gv[e]);
        }
        if (lane == 0) from_f32(*yb, *gb);
      }
    }
    bar_sync(BAR, P);
  }
  if (owns) {
#pragma unroll
    for (int i = 0; i < Q4; ++i) {
      Wg[i] = w[i];
      if (p.gW0.base != nullptr) p.gW0.mat(n, h)[row * E + part + i] = x[i];
    }
  }
}

// The A operand of X^T for 16 columns of X, whose rows (steps) lie in shared memory.
__device__ __forceinline__ void ldsm_at(uint32_t (&a)[4], const unsigned char* x, int pitch, int lane) {
  ldsm4_t(a, x + frag_b_off(lane, pitch));
}

// Two accumulator tiles to and from tensor memory (16 lanes, 16 columns): its 16 x 256-bit shape is the tiles' own layout.
__device__ __forceinline__ void tm_ld(uint32_t addr, float (&v)[2][4]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0][0]), "=f"(v[0][1]), "=f"(v[0][2]), "=f"(v[0][3]), "=f"(v[1][0]), "=f"(v[1][1]), "=f"(v[1][2]), "=f"(v[1][3])
               : "r"(addr));
}
__device__ __forceinline__ void tm_ld_wait(float (&v)[2][4]) {   // (the values go through it: nothing uses them before)
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+f"(v[0][0]), "+f"(v[0][1]), "+f"(v[0][2]), "+f"(v[0][3]), "+f"(v[1][0]), "+f"(v[1][1]), "+f"(v[1][2]), "+f"(v[1][3])
               :: "memory");
}
__device__ __forceinline__ void tm_st(uint32_t addr, const float (&v)[2][4]) {
  asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(addr), "f"(v[0][0]), "f"(v[0][1]),
               "f"(v[0][2]), "f"(v[0][3]), "f"(v[1][0]), "f"(v[1][1]), "f"(v[1][2]), "f"(v[1][3])
               : "memory");
}
__device__ __forceinline__ void tm_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Place of (row, column) in a 16 x 16 sum: rows of pairs and columns of single values without bank conflicts.
__device__ __forceinline__ int part_at(int i, int j) { return (i * DC + j) ^ ((i & 2) << 2) ^ ((i & 4) << 2); }

template <typename TIO, int E, int NPW, int S, bool PACKED>
__device__ __forceinline__ bool delta_bwd_chain_warp(const DeltaBwdParams& p, unsigned char* smem, int warp, int lane,
                                                     int n, int h) {
  using R = DeltaRing<TIO, E, NPW, S, PACKED, true>;
  using SM = DeltaChunkBwdSmem<TIO, E, NPW, S, PACKED>;
  using D = typename R::D;
  constexpr int NW = D::NW, NP = R::NP, NG = R::NG, NT = R::NT;
  const int L = p.L, nchunks = (L + DC - 1) / DC;
  const int g = lane / 4, t = lane % 4, m0 = warp * 16;
  constexpr int TLS = E >= 32 && R::SW == 2 ? 4 : 2;   // tiles of G updated at once
  float finite = 0.f;   // 0 while this warp's results are
  // G as tiles (m = m0 + g, + 8) x (e = 8 j + 2 t, + 1), in registers or (TM) in tensor memory: two tiles at a time, `get` before use, `put` after
  // a change
  constexpr bool TM = R::SW == 1;
  float G[TM ? 2 : E / 8][4];
  uint32_t tm = 0;
  if constexpr (TM) {
    bar_sync(SM::GP_FULL, 64 * NW);   // the memory is there
    tm = *reinterpret_cast<volatile uint32_t*>(smem + SM::OTM) + E + ((uint32_t)(warp * 32) << 16);
  }
  auto get = [&](int j) {
    if constexpr (TM) {
      float(&v)[2][4] = *reinterpret_cast<float(*)[2][4]>(&G[0]);
      tm_ld(tm + j * 8, v);
      tm_ld_wait(v);
    }
  };
  auto put = [&](int j) {
    if constexpr (TM) tm_st(tm + j * 8, *reinterpret_cast<float(*)[2][4]>(&G[0]));
  };
  auto at = [](int j) { return TM ? j % 2 : j; };
#pragma unroll
  for (int j = 0; j < E / 8; ++j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) G[at(j)][i] = 0.f;
    if (j % 2) put(j - 1);
  }
  if constexpr (TM) tm_st_wait();

  // Value (nn, i) of this lane: step nn*8 + 2t + (i&1), column m0 + g + (i>>1)*8.  One pointer per stream to
  // step 2t of a chunk.
  const long long c0 = (long long)(nchunks - 1) * DC;
  auto col_ptr = [&](const SeqView& v, int es) { return v.row(n, h, 2 * t) + c0 * v.sl + (m0 + g) * es; };
  const char* vop = col_ptr(p.v_old, 4);
  // v and its gradient (packed form: a part of the rows)
  constexpr bool VROWS = !PACKED || R::IN_PLACE;
  const SeqView &vv = PACKED ? p.Q : p.V, &gvv = PACKED ? p.gQ : p.gV;
  constexpr int VOFF = PACKED ? 2 * E * (int)sizeof(TIO) : 0;
  const char* vp = VROWS ? col_ptr(vv, sizeof(TIO)) + VOFF : nullptr;
  char* gvp = VROWS ? col_ptr(gvv, sizeof(TIO)) + VOFF : nullptr;
  auto load = [&](auto (&d)[2][4], const char* ptr, long long sl, int left) {
    using T = typename std::remove_reference<decltype(d[0][0])>::type;
#pragma unroll
    for (int nn = 0; nn < 2; ++nn)
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        const T* r = reinterpret_cast<const T*>(ptr + (nn * 8 + jj) * sl);
        from_f32(d[nn][jj], 0.f);
        from_f32(d[nn][2 + jj], 0.f);
        if (nn * 8 + jj < left) {
          d[nn][jj] = r[0];
          d[nn][2 + jj] = r[8];
        }
      }
  };
  auto step_of = [&](int nn, int i) { return nn * 8 + 2 * t + (i & 1); };
  const int bo = frag_b_off(lane, D::PITCH), ko = frag_a_off(lane, D::PITCH);
  for (int it = 0; it < nchunks; ++it) {
    const int s = it % S, b = it & 1, t0 = (nchunks - 1 - it) * DC;
    const int left = SRWM_BAD_ROWS(p.dbg, 14, t0, min(DC, L - t0), L, DC) ? 0 : min(DC, L - t0) - 2 * t;
    const unsigned char* slot = R::slot(smem, s);
    const unsigned char *sq = slot + R::OQ, *sk = slot + R::OK, *sg = slot + R::OG;
    const float* sb = reinterpret_cast<const float*>(slot + R::OB);
    TIO vr[2][4];
    float vor[2][4];
    if constexpr (VROWS) load(vr, vp, vv.sl, left);
    load(vor, vop, p.v_old.sl, left);
    bar_sync(R::full(s), R::NM);

    float r[2][4];
    uint32_t a[3][4], f[3][2][2], got[NG][4];
#pragma unroll
    for (int z = 0; z < NG; ++z) ldsm_at(got[z], sg + z * D::PIECE + m0 * 2, D::PITCH, lane);
    {
      float hi[2][4] = {}, lo[2][4] = {};
#pragma unroll
      for (int ks = 0; ks < E / 16; ++ks) {
        uint32_t bk[NP][2][2];
        get(2 * ks);
        split_frag(G[at(2 * ks)], G[at(2 * ks + 1)], a);
        if constexpr (R::SW == 1) {
#pragma unroll
          for (int z = 0; z < 3; ++z) stsm4(smem + SM::OP + z * SM::GP + m0 * D::PITCH + ko + ks * 32, a[z]);
        }
#pragma unroll
        for (int z = 0; z < NP; ++z) ldsm_b(bk[z], sk + z * D::PIECE + bo + ks * 32);
        mma_tiles<3, NP, 2>(hi, lo, a, bk);
      }
      if constexpr (R::SW == 1) bar_arrive(SM::GP_FULL, 64 * NW);
      load_frag(slot + R::OA, lane, f);
      mma_tiles<NG, 3, 2>(hi, lo, got, f);
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          r[nn][i] = hi[nn][i] + lo[nn][i];
          hi[nn][i] = lo[nn][i] = 0.f;
        }
      split_frag(r[0], r[1], a);
      load_frag(slot + R::OT, lane, f);
      mma_tiles<3, 3, 2>(hi, lo, a, f);
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int i = 0; i < 4; ++i) r[nn][i] += hi[nn][i] + lo[nn][i];
    }
    float gv[2][4], gb[4];
    const float* sv = reinterpret_cast<const float*>(slot + R::OV);
#pragma unroll
    for (int nn = 0; nn < 2; ++nn)
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        float u[2];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const float v = !VROWS ? sv[step_of(nn, jj) * D::VP + m0 + g + hh * 8] : to_f32(vr[nn][2 * hh + jj]);
          u[hh] = v - vor[nn][2 * hh + jj];
          gv[nn][2 * hh + jj] = r[nn][2 * hh + jj] * sb[step_of(nn, jj)];
        }
        gb[nn * 2 + jj] = fmaf(r[nn][2 + jj], u[1], r[nn][jj] * u[0]);
      }
    finite = fmaf(0.f, ((gv[0][0] + gv[0][1]) + (gv[0][2] + gv[0][3])) + ((gv[1][0] + gv[1][1]) + (gv[1][2] + gv[1][3])), finite);
    // hand -gv over, then update G
    split_frag(gv[0], gv[1], a);
    if (it >= 2) bar_sync(SM::GV_EMPTY + b, SM::NGV);
    unsigned char* gvb = smem + SM::OGV + b * SM::GV + g * D::PITCH + (m0 + 2 * t) * 2;
    uint32_t x[3][4];   // (steps x m)
#pragma unroll
    for (int z = 0; z < 3; ++z) {
#pragma unroll
      for (int i = 0; i < 4; ++i) a[z][i] ^= 0x80008000u;
      transpose_a(a[z], x[z]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<uint32_t*>(gvb + z * D::PIECE + (i & 1) * 8 * D::PITCH + (i >> 1) * 16) = x[z][i];
    }
    // gbeta: over the eight column lanes; lane g keeps the sum of step index g & 3 (lanes 4..7 repeat 0..3)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) gb[i] += __shfl_xor_sync(0xffffffffu, gb[i], o);
    }
    if (g == 0) {
      float* xb = reinterpret_cast<float*>(smem + SM::OB) + (b * NW + warp) * DC + 2 * t;
      *reinterpret_cast<float2*>(xb) = make_float2(gb[0], gb[1]);
      *reinterpret_cast<float2*>(xb + 8) = make_float2(gb[2], gb[3]);
    }
    bar_arrive(SM::GV_FULL + b, SM::NGV);
    float pt[2][4] = {};   // -GV INS^T over this warp's columns
    if constexpr (R::SW == 1) {
      float lo[2][4] = {};
#pragma unroll
      for (int z = 0; z < 3; ++z) ldsm_b(f[z], slot + R::OI + z * D::PIECE + bo + m0 * 2);
      mma_tiles<3, 3, 2>(pt, lo, x, f);
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int i = 0; i < 4; ++i) pt[nn][i] += lo[nn][i];
    }
#pragma unroll
    for (int j4 = 0; j4 < E / 8 / TLS; ++j4) {
      constexpr int NTL = TLS;
      uint32_t bk[NP][NTL][2], bq[NP][NTL][2];
#pragma unroll
      for (int z = 0; z < NP; ++z)
#pragma unroll
        for (int hh = 0; hh < NTL / 2; ++hh) {
          uint32_t x[2][2];
          ldsm_bt(x, sk + z * D::PIECE + ko + (j4 * (TLS / 2) + hh) * 32);
          bk[z][2 * hh][0] = x[0][0]; bk[z][2 * hh][1] = x[0][1];
          bk[z][2 * hh + 1][0] = x[1][0]; bk[z][2 * hh + 1][1] = x[1][1];
          ldsm_bt(x, sq + z * D::PIECE + ko + (j4 * (TLS / 2) + hh) * 32);
          bq[z][2 * hh][0] = x[0][0]; bq[z][2 * hh][1] = x[0][1];
          bq[z][2 * hh + 1][0] = x[1][0]; bq[z][2 * hh + 1][1] = x[1][1];
        }
      float d[NTL][4] = {};
      mma_tiles<3, NP, NTL>(d, d, a, bk);
      mma_tiles<NG, NP, NTL>(d, d, got, bq);
      get(j4 * TLS);
#pragma unroll
      for (int q = 0; q < NTL; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) G[at(j4 * TLS + q)][i] += d[q][i];
      put(j4 * TLS);
    }
    if constexpr (TM) tm_st_wait();
    if (it + S < nchunks) bar_arrive(R::empty(s), NT);
    if constexpr (VROWS) {
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int jj = 0; jj < 2; ++jj)
          if (nn * 8 + jj < left) {
            TIO* y = reinterpret_cast<TIO*>(gvp + (nn * 8 + jj) * gvv.sl);
            from_f32(y[0], gv[nn][jj]);
            from_f32(y[8], gv[nn][2 + jj]);
          }
      gvp -= DC * gvv.sl;
      vp -= DC * vv.sl;
    }
    vop -= DC * p.v_old.sl;
    if constexpr (R::SW == 1) {
      // The state warps have used this chunk's G, so they are done with the sums of the chunk before.
      bar_sync(SM::GP_EMPTY, 64 * NW);
      float* st = reinterpret_cast<float*>(smem + SM::OS) + warp * DC * DC;
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
          *reinterpret_cast<float2*>(st + part_at(g + hh * 8, nn * 8 + 2 * t)) = make_float2(pt[nn][2 * hh], pt[nn][2 * hh + 1]);
      bar_arrive(SM::PARTS, 64 * NW);
    }
  }
#pragma unroll
  for (int j = 0; j < E / 8; ++j) {
    if (j % 2 == 0) get(j);
    finite = fmaf(0.f, (G[at(j)][0] + G[at(j)][1]) + (G[at(j)][2] + G[at(j)][3]), finite);
  }
  const bool ok = bar_all(SM::LAST, 32 * DeltaBwdRoles<TIO, E, NPW, PACKED>::WARPS, finite == 0.f);
  if (ok && p.gW0.base != nullptr) {
    float* Gg = p.gW0.mat(n, h);
#pragma unroll
    for (int j = 0; j < E / 8; ++j) {
      if (j % 2 == 0) get(j);
#pragma unroll
      for (int i = 0; i < 4; ++i) Gg[(8 * j + 2 * t + (i & 1)) * E + m0 + g + (i >> 1) * 8] = G[at(j)][i];
    }
  }
  if constexpr (TM) bar_arrive(SM::GP_EMPTY, 64 * NW);   // tensor memory is done with
  return ok;
}

// A 16 x 8 tile (rows = steps i, columns = steps j of half `tile`) of X Y^T over part `kp` of m, X in NX pieces.
// x: this warp's A operand rows; y: a functor giving the B operands of both tiles for 16 values of m.
template <int E, int KH, int NX, typename Y>
__device__ __forceinline__ void small_tile(const unsigned char* x, int pitch, int lane, int tile, int kp, float* out, int sp,
                                           Y y_of) {
  const int ao = frag_a_off(lane, pitch);
  float hi[1][4] = {}, lo[1][4] = {};
#pragma unroll 1
  for (int k = 0; k < E / 16 / KH; ++k) {
    const int ks = kp * (E / 16 / KH) + k;
    uint32_t a[NX][4], b[3][2][2], c[3][1][2];
#pragma unroll
    for (int z = 0; z < NX; ++z) ldsm4(a[z], x + z * DC * pitch + ao + ks * 32);
    y_of(ks, b);
#pragma unroll
    for (int z = 0; z < 3; ++z) {
      c[z][0][0] = tile ? b[z][1][0] : b[z][0][0];
      c[z][0][1] = tile ? b[z][1][1] : b[z][0][1];
    }
    mma_tiles<NX, 3, 1>(hi, lo, a, c);
  }
  const int g = lane / 4, t = lane % 4;
#pragma unroll
  for (int hh = 0; hh < 2; ++hh)
    *reinterpret_cast<float2*>(out + (g + hh * 8) * sp + tile * 8 + 2 * t) =
        make_float2(hi[0][2 * hh] + lo[0][2 * hh], hi[0][2 * hh + 1] + lo[0][2 * hh + 1]);
}

// The coefficients of the two K terms from x[i][j] = -ins_i.gv_j: c[i][j] = x[i][j] (j > i) - x[j][i] (j >= i), as B
// operands (k = j, n = i); x is the sum of KH parts.
template <int KH>
__device__ __forceinline__ void coef_frag(int lane, const float* x, int sp, int part, uint32_t (&c)[3][2][2]) {
  const int g = lane / 4, t = lane % 4;
#pragma unroll
  for (int ti = 0; ti < 2; ++ti)
#pragma unroll
    for (int tj = 0; tj < 2; ++tj) {
      const int i = g + ti * 8, j = tj * 8 + 2 * t;
      float2 d = *reinterpret_cast<const float2*>(x + i * sp + j);
      float u[2] = {x[j * sp + i], x[(j + 1) * sp + i]};
      if constexpr (KH == 2) {
        const float2 d2 = *reinterpret_cast<const float2*>(x + part + i * sp + j);
        d.x += d2.x; d.y += d2.y;
        u[0] += x[part + j * sp + i];
        u[1] += x[part + (j + 1) * sp + i];
      }
      split3(j > i ? d.x - u[0] : (j == i ? -u[0] : 0.f), j + 1 > i ? d.y - u[1] : (j + 1 == i ? -u[1] : 0.f), c[0][ti][tj],
             c[1][ti][tj], c[2][ti][tj]);
    }
}

// ... from NP sums x[i][j] = -gv_i.ins_j (part_at)
template <int NP>
__device__ __forceinline__ void coef_parts(int lane, const float* x, uint32_t (&c)[3][2][2]) {
  const int g = lane / 4, t = lane % 4;
#pragma unroll
  for (int ti = 0; ti < 2; ++ti)
#pragma unroll
    for (int tj = 0; tj < 2; ++tj) {
      const int i = g + ti * 8, j = tj * 8 + 2 * t;
      float d[2] = {}, u[2] = {};
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        const float* y = x + q * DC * DC;
        const float2 v = *reinterpret_cast<const float2*>(y + part_at(i, j));
        d[0] += v.x; d[1] += v.y;
        u[0] += y[part_at(j, i)];
        u[1] += y[part_at(j + 1, i)];
      }
      split3(j > i ? u[0] - d[0] : (j == i ? -d[0] : 0.f), j + 1 > i ? u[1] - d[1] : (j + 1 == i ? -d[1] : 0.f), c[0][ti][tj],
             c[1][ti][tj], c[2][ti][tj]);
    }
}

// Output tiles (steps x 16 rows e, transposed): value (nn, i) is step nn*8 + 2t + (i&1), e = base + (i>>1)*8.
template <typename TIO>
__device__ __forceinline__ void store_steps(char* p, long long sl, int left, const float (&v)[2][4]) {
#pragma unroll
  for (int nn = 0; nn < 2; ++nn)
#pragma unroll
    for (int jj = 0; jj < 2; ++jj)
      if (nn * 8 + jj < left) {
        TIO* y = reinterpret_cast<TIO*>(p + (nn * 8 + jj) * sl);
        from_f32(y[0], v[nn][jj]);
        from_f32(y[8], v[nn][2 + jj]);
      }
}

// State warps of the SW = 2 form.  W warps (is_g false): GQ, the W part of GK, W itself.  G warps: GK, gbeta; in the packed form
// the gradient rows.  Both multiply their state by rows of the chunk and add products of rows to it, so
// they run the same code (see the note on code size).
template <typename TIO, int E, int NPW, int S, bool PACKED>
__device__ __forceinline__ bool delta_bwd_state_warp(const DeltaBwdParams& p, unsigned char* smem, bool is_g, int warp,
                                                     int lane, int n, int h) {
  using R = DeltaRing<TIO, E, NPW, S, PACKED, true>;
  using SM = DeltaChunkBwdSmem<TIO, E, NPW, S, PACKED>;
  using D = typename R::D;
  constexpr int NW = D::NW, NP = R::NP, NG = R::NG, NT = R::NT, KS = E / 16, KH = SM::KH;
  const int L = p.L, nchunks = (L + DC - 1) / DC;
  const int g = lane / 4, t = lane % 4, e0 = warp * 16;
  float X[E / 8][4];   // W or G: (e = e0 + g, + 8) x (m = 8 j + 2 t, + 1)
  float* Wg = p.W.mat(n, h) + (e0 + g) * E + 2 * t;
#pragma unroll
  for (int j = 0; j < E / 8; ++j)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      float2 v = make_float2(0.f, 0.f);
      if (!is_g) v = *reinterpret_cast<const float2*>(Wg + hh * 8 * E + 8 * j);
      X[j][2 * hh] = v.x; X[j][2 * hh + 1] = v.y;
    }
  float finite = 0.f;
  const float sgn = is_g ? 1.f : -1.f;
  float* xs = reinterpret_cast<float*>(smem + SM::OS);
  const int bo = frag_b_off(lane, D::PITCH), ko = frag_a_off(lane, D::PITCH);
  // gq (W warps) or gk (G warps) of step 2t of a chunk, row e0 + g
  const SeqView& ov = is_g && !PACKED ? p.gK : p.gQ;
  char* op = ov.row(n, h, 2 * t) + (long long)(nchunks - 1) * DC * ov.sl + (e0 + g) * sizeof(TIO);

  for (int it = 0; it < nchunks; ++it) {
    const int s = it % S, b = it & 1, t0 = (nchunks - 1 - it) * DC;
    const int nt = SRWM_BAD_ROWS(p.dbg, 15, t0, min(DC, L - t0), L, DC) ? 0 : min(DC, L - t0), left = nt - 2 * t;
    const unsigned char* slot = R::slot(smem, s);
    const unsigned char *sq = slot + R::OQ, *sk = slot + R::OK, *sg = slot + R::OG, *si = slot + R::OI;
    const unsigned char* gvb = smem + SM::OGV + b * SM::GV;
    bar_sync(R::full_state(s), R::NS);
    uint32_t kt[NP][4], qt[NP][4];
#pragma unroll
    for (int z = 0; z < NP; ++z) {
      ldsm_at(kt[z], sk + z * D::PIECE + e0 * 2, D::PITCH, lane);
      ldsm_at(qt[z], sq + z * D::PIECE + e0 * 2, D::PITCH, lane);
    }
    bar_sync(SM::GV_FULL + b, SM::NGV);
    // -INS GV^T, for the G warps: a tile and a part of m per W warp
    if (!is_g) {
#pragma unroll 1
      for (int job = warp; job < 2 * KH; job += NW)
        small_tile<E, KH, 3>(si, D::PITCH, lane, job & 1, job >> 1, xs + (job >> 1) * DC * SM::SP, SM::SP,
                             [&](int ks, uint32_t(&x)[3][2][2]) {
#pragma unroll
                               for (int z = 0; z < 3; ++z) ldsm_b(x[z], gvb + z * D::PIECE + bo + ks * 32);
                             });
      bar_arrive(SM::IGV, 64 * NW);
    }
    // o: W: -GV W^T, G: INS G^T.  q: W: GO W^T.  X: W -= K^T INS, G += Q^T GO - K^T GV
    float o[2][4] = {}, ol[2][4] = {}, q[2][4] = {}, ql[2][4] = {};
    const unsigned char *x1 = is_g ? si : gvb, *y1 = is_g ? gvb : si;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      uint32_t a[3][4], x[3][2][2];
      split_frag(X[2 * ks], X[2 * ks + 1], a);
#pragma unroll
      for (int z = 0; z < 3; ++z) ldsm_b(x[z], x1 + z * D::PIECE + bo + ks * 32);
      mma_tiles<3, 3, 2>(o, ol, a, x);
      if (!is_g) {
        uint32_t y[NG][2][2];
#pragma unroll
        for (int z = 0; z < NG; ++z) ldsm_b(y[z], sg + z * D::PIECE + bo + ks * 32);
        mma_tiles<3, NG, 2>(q, ql, a, y);
      }
      float d[2][4] = {};
#pragma unroll
      for (int z = 0; z < 3; ++z) ldsm_bt(x[z], y1 + z * D::PIECE + ko + ks * 32);
      mma_tiles<NP, 3, 2>(d, d, kt, x);
      if (is_g) {
        uint32_t y[NG][2][2];
#pragma unroll
        for (int z = 0; z < NG; ++z) ldsm_bt(y[z], sg + z * D::PIECE + ko + ks * 32);
        mma_tiles<NP, NG, 2>(d, d, qt, y);
      }
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int i = 0; i < 4; ++i) X[2 * ks + nn][i] = fmaf(sgn, d[nn][i], X[2 * ks + nn][i]);
    }
    // the masked terms: W: gq -= triu(GO INS^T, 1) K.  G: gk += triu(INS GO^T) Q, then the two K terms
    const float* xb = reinterpret_cast<const float*>(smem + SM::OB) + b * NW * DC;
    float gb = 0.f;
    {
      uint32_t c[3][2][2];
      load_frag(slot + R::OC + (is_g ? D::FRAG : 0), lane, c);
      if (is_g) {
        mma_tiles<NP, 3, 2>(o, ol, qt, c);
        if (lane < DC) {
#pragma unroll
          for (int w = 0; w < NW; ++w) gb += xb[w * DC + lane];
        }
        bar_sync(SM::IGV, 64 * NW);
        coef_frag<KH>(lane, xs, SM::SP, DC * SM::SP, c);
        mma_tiles<NP, 3, 2>(o, ol, kt, c);
      } else {
        mma_tiles<NP, 3, 2>(q, ql, kt, c);
      }
    }
    if (!PACKED || !is_g) {
      if (it + 2 < nchunks) bar_arrive(SM::GV_EMPTY + b, SM::NGV);
      if (it + S < nchunks) bar_arrive(R::empty(s), NT);
    }
    float4* xk = reinterpret_cast<float4*>(smem + SM::OK) + warp * 64 + lane;
    float* xg = reinterpret_cast<float*>(smem + SM::OX);
    if (!is_g) {
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
        xk[nn * 32] = make_float4(o[nn][0] + ol[nn][0], o[nn][1] + ol[nn][1], o[nn][2] + ol[nn][2], o[nn][3] + ol[nn][3]);
    } else {
      bar_sync(SM::GK, 64 * NW);
#pragma unroll
      for (int nn = 0; nn < 2; ++nn) {
        const float4 v = xk[nn * 32];
        q[nn][0] = o[nn][0] + v.x; q[nn][1] = o[nn][1] + v.y; q[nn][2] = o[nn][2] + v.z; q[nn][3] = o[nn][3] + v.w;
#pragma unroll
        for (int i = 0; i < 4; ++i) ql[nn][i] = ol[nn][i];
      }
    }
#pragma unroll
    for (int nn = 0; nn < 2; ++nn)
#pragma unroll
      for (int i = 0; i < 4; ++i) q[nn][i] += ql[nn][i];
    finite = fmaf(0.f, ((q[0][0] + q[0][1]) + (q[0][2] + q[0][3])) + ((q[1][0] + q[1][1]) + (q[1][2] + q[1][3])), finite);
    if constexpr (!PACKED) {
      if (!is_g) bar_arrive(SM::GK, 64 * NW);
      store_steps<TIO>(op, ov.sl, left, q);
      op -= DC * ov.sl;
      if (is_g && warp == 0 && lane < nt) from_f32(*reinterpret_cast<TIO*>(p.gbeta.row(n, h, t0 + lane)), gb);
    } else {
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          xg[((is_g ? DC : 0) + nn * 8 + 2 * t + (i & 1)) * SM::XP + e0 + g + (i >> 1) * 8] = q[nn][i];
      if (!is_g) {
        bar_arrive(SM::GK, 64 * NW);
        continue;
      }
      // back through the layers' preparation (see delta.cuh) into the packed gradient row [gq | gk | gv | gb]
      bar_sync(SM::ROWS, 32 * NW);
      constexpr int LPR = E / 4, RG = 32 * NW / LPR;
      const int tid = warp * 32 + lane, l = tid % LPR;
      const float* norm = reinterpret_cast<const float*>(slot + R::ON);
      const float* sb = reinterpret_cast<const float*>(slot + R::OB);
#pragma unroll 1
      for (int tt = tid / LPR; tt < DC; tt += RG) {
        float qv[4] = {}, kv[4] = {}, gv[4] = {}, vq[4], vk[4], dq = 0.f, dk = 0.f;
#pragma unroll 1
        for (int z = 0; z < 3; ++z) {   // the pieces add up to the values exactly
          const int off = z * D::PIECE + tt * D::PITCH + l * 8;
          float x[4];
          ld_vec<4>(reinterpret_cast<const __nv_bfloat16*>(sq + off), x);
#pragma unroll
          for (int i = 0; i < 4; ++i) qv[i] += x[i];
          ld_vec<4>(reinterpret_cast<const __nv_bfloat16*>(sk + off), x);
#pragma unroll
          for (int i = 0; i < 4; ++i) kv[i] += x[i];
          ld_vec<4>(reinterpret_cast<const __nv_bfloat16*>(gvb + off), x);
#pragma unroll
          for (int i = 0; i < 4; ++i) gv[i] -= x[i];
        }
        ld_vec<4>(xg + tt * SM::XP + l * 4, vq);
        ld_vec<4>(xg + (DC + tt) * SM::XP + l * 4, vk);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          dq = fmaf(vq[i], qv[i], dq);
          dk = fmaf(vk[i], kv[i], dk);
        }
#pragma unroll
        for (int w = 1; w < LPR; w <<= 1) {
          dq += __shfl_xor_sync(0xffffffffu, dq, w);
          dk += __shfl_xor_sync(0xffffffffu, dk, w);
        }
        if (tt < nt) {
          const float Sq = norm[tt], Sk = norm[DC + tt];
          const float iq = __fdividef(1.f, Sq), ik = __fdividef(1.f, Sk);
          TIO* y = reinterpret_cast<TIO*>(p.gQ.row(n, h, t0 + tt));
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float aq = qv[i] * Sq, ak = kv[i] * Sk;
            from_f32(y[l * 4 + i], (vq[i] - dq) * iq * (aq > 1.f ? 1.f : aq));
            from_f32(y[E + l * 4 + i], (vk[i] - dk) * ik * (ak > 1.f ? 1.f : ak));
            from_f32(y[2 * E + l * 4 + i], gv[i]);
          }
          if (l == 0) {
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < NW; ++w) v += xb[w * DC + tt];
            const float bt = sb[tt];
            from_f32(y[3 * E], v * bt * (1.f - bt));
          }
        }
      }
      if (it + 2 < nchunks) bar_arrive(SM::GV_EMPTY + b, SM::NGV);
      if (it + S < nchunks) bar_arrive(R::empty(s), NT);
    }
  }
#pragma unroll
  for (int j = 0; j < E / 8; ++j) finite = fmaf(0.f, (X[j][0] + X[j][1]) + (X[j][2] + X[j][3]), finite);
  if (!bar_all(SM::LAST, 32 * DeltaBwdRoles<TIO, E, NPW, PACKED>::WARPS, finite == 0.f)) return false;
  if (!is_g) {   // W now holds W_0: restored in place (as the reference does)
#pragma unroll
    for (int j = 0; j < E / 8; ++j)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh)
        *reinterpret_cast<float2*>(Wg + hh * 8 * E + 8 * j) = make_float2(X[j][2 * hh], X[j][2 * hh + 1]);
  }
  return true;
}

// State warps of the SW = 1 form: 16 rows e of W each, and the same rows of GQ and GK.
template <typename TIO, int E, int NPW, int S, bool PACKED>
__device__ __forceinline__ bool delta_bwd_rows_warp(const DeltaBwdParams& p, unsigned char* smem, int warp, int lane, int n, int h) {
  using R = DeltaRing<TIO, E, NPW, S, PACKED, true>;
  using SM = DeltaChunkBwdSmem<TIO, E, NPW, S, PACKED>;
  using D = typename R::D;
  constexpr int NW = D::NW, NP = R::NP, NG = R::NG, NT = R::NT, KS = E / 16;
  const int L = p.L, nchunks = (L + DC - 1) / DC;
  const int g = lane / 4, t = lane % 4, e0 = warp * 16;
  // W in tensor memory, a row e a lane (lanes 0..15 of the warp's 32), a block of 16 columns at a time in the registers
  // (two tiles: e = e0 + g, + 8, m = 16 j + 2 t, + 1, + 8, + 9)
  float* Wg = p.W.mat(n, h) + (e0 + g) * E + 2 * t;
  uint32_t* tma = reinterpret_cast<uint32_t*>(smem + SM::OTM);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(tma))), "r"(2 * E));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  bar_sync(SM::GP_FULL, 64 * NW);
  const uint32_t tm0 = *reinterpret_cast<volatile uint32_t*>(tma), tm = tm0 + ((uint32_t)(warp * 32) << 16);
#pragma unroll
  for (int j = 0; j < E / 16; ++j) {
    float w[2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 v = *reinterpret_cast<const float2*>(Wg + (i & 1) * 8 * E + 16 * j + (i >> 1) * 8);
      w[i >> 1][(i & 1) * 2] = v.x; w[i >> 1][(i & 1) * 2 + 1] = v.y;
    }
    tm_st(tm + j * 16, w);
  }
  tm_st_wait();
  float finite = 0.f;
  float* xs = reinterpret_cast<float*>(smem + SM::OS);
  const int bo = frag_b_off(lane, D::PITCH), ko = frag_a_off(lane, D::PITCH);
  // gq and gk of step 2t of a chunk, row e0 + g
  auto row_ptr = [&](const SeqView& v) { return v.row(n, h, 2 * t) + (long long)(nchunks - 1) * DC * v.sl + (e0 + g) * sizeof(TIO); };
  const SeqView& gkv = PACKED ? p.gQ : p.gK;   // packed form: a part of the rows
  char *qp = row_ptr(p.gQ), *kp = row_ptr(gkv) + (PACKED ? E * (int)sizeof(TIO) : 0);

  for (int it = 0; it < nchunks; ++it) {
    const int s = it % S, b = it & 1, t0 = (nchunks - 1 - it) * DC;
    const int nt = SRWM_BAD_ROWS(p.dbg, 15, t0, min(DC, L - t0), L, DC) ? 0 : min(DC, L - t0), left = nt - 2 * t;
    const unsigned char* slot = R::slot(smem, s);
    const unsigned char *sq = slot + R::OQ, *sk = slot + R::OK, *sg = slot + R::OG, *si = slot + R::OI;
    const unsigned char* gvb = smem + SM::OGV + b * SM::GV;
    float o[2][4] = {}, ol[2][4] = {};   // gk
    uint32_t c[3][2][2], r[NP][4];
    bar_sync(SM::GP_FULL, 64 * NW);   // (and the slot is full)
    // INS G^T
#pragma unroll 1
    for (int ks = 0; ks < KS; ++ks) {
      uint32_t a[3][4], x[3][2][2];
#pragma unroll
      for (int z = 0; z < 3; ++z) {
        ldsm_at(a[z], smem + SM::OP + z * SM::GP + ks * DC * D::PITCH + e0 * 2, D::PITCH, lane);
        ldsm_b(x[z], si + z * D::PIECE + bo + ks * 32);
      }
      mma_tiles<3, 3, 2>(o, ol, a, x);
    }
    bar_arrive(SM::GP_EMPTY, 64 * NW);
    // triu(INS GO^T) Q
    load_frag(slot + R::OC + D::FRAG, lane, c);
#pragma unroll
    for (int z = 0; z < NP; ++z) ldsm_at(r[z], sq + z * D::PIECE + e0 * 2, D::PITCH, lane);
    mma_tiles<NP, 3, 2>(o, ol, r, c);
    bar_sync(SM::GV_FULL + b, SM::NGV);
    // -GV W^T to gk, GO W^T to gq, W -= K^T INS
    float q[2][4] = {}, ql[2][4] = {};
#pragma unroll
    for (int z = 0; z < NP; ++z) ldsm_at(r[z], sk + z * D::PIECE + e0 * 2, D::PITCH, lane);
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      uint32_t a[3][4], x[3][2][2], y[NG][2][2];
      float w[2][4];
      tm_ld(tm + ks * 16, w);
      tm_ld_wait(w);
      split_frag(w[0], w[1], a);
#pragma unroll
      for (int z = 0; z < 3; ++z) ldsm_b(x[z], gvb + z * D::PIECE + bo + ks * 32);
      mma_tiles<3, 3, 2>(o, ol, a, x);
#pragma unroll
      for (int z = 0; z < NG; ++z) ldsm_b(y[z], sg + z * D::PIECE + bo + ks * 32);
      mma_tiles<3, NG, 2>(q, ql, a, y);
      float d[2][4] = {};
#pragma unroll
      for (int z = 0; z < 3; ++z) ldsm_bt(x[z], si + z * D::PIECE + ko + ks * 32);
      mma_tiles<NP, 3, 2>(d, d, r, x);
#pragma unroll
      for (int nn = 0; nn < 2; ++nn)
#pragma unroll
        for (int i = 0; i < 4; ++i) w[nn][i] -= d[nn][i];
      tm_st(tm + ks * 16, w);
    }
    tm_st_wait();
    // gq -= triu(GO INS^T, 1) K, and the two K terms of gk
    load_frag(slot + R::OC, lane, c);
    mma_tiles<NP, 3, 2>(q, ql, r, c);
    float gb = 0.f;
    if (warp == 0 && lane < DC) {
      const float* xb = reinterpret_cast<const float*>(smem + SM::OB) + b * NW * DC;
#pragma unroll
      for (int w = 0; w < NW; ++w) gb += xb[w * DC + lane];
    }
    bar_sync(SM::PARTS, 64 * NW);
    coef_parts<NW>(lane, xs, c);
    mma_tiles<NP, 3, 2>(o, ol, r, c);
    if constexpr (!PACKED) {
      if (it + 2 < nchunks) bar_arrive(SM::GV_EMPTY + b, SM::NGV);
      if (it + S < nchunks) bar_arrive(R::empty(s), NT);
    }
#pragma unroll
    for (int nn = 0; nn < 2; ++nn)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        q[nn][i] += ql[nn][i];
        o[nn][i] += ol[nn][i];
      }
    finite = fmaf(0.f, ((q[0][0] + q[0][1]) + (q[0][2] + q[0][3])) + ((q[1][0] + q[1][1]) + (q[1][2] + q[1][3])), finite);
    finite = fmaf(0.f, ((o[0][0] + o[0][1]) + (o[0][2] + o[0][3])) + ((o[1][0] + o[1][1]) + (o[1][2] + o[1][3])), finite);
    if constexpr (PACKED) {
      // back through the layers' preparation (see delta.cuh): the rows' dot products with q and k, whose pieces as A operands
      // hold the values of this lane's places
      float xq[2][4] = {}, xk[2][4] = {};
#pragma unroll
      for (int z = 0; z < 3; ++z) {
        uint32_t y[4];
        ldsm_at(y, sq + z * D::PIECE + e0 * 2, D::PITCH, lane);
#pragma unroll
        for (int nn = 0; nn < 2; ++nn)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {   // (a bf16 value is the upper half of its fp32)
            xq[nn][2 * hh] += __uint_as_float(y[2 * nn + hh] << 16);
            xq[nn][2 * hh + 1] += __uint_as_float(y[2 * nn + hh] & 0xffff0000u);
            xk[nn][2 * hh] += __uint_as_float(r[z][2 * nn + hh] << 16);
            xk[nn][2 * hh + 1] += __uint_as_float(r[z][2 * nn + hh] & 0xffff0000u);
          }
      }
      float* dots = reinterpret_cast<float*>(smem + SM::OX);
      const float* norm = reinterpret_cast<const float*>(slot + R::ON);
      float d[8], nq[4], nk[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {   // step (i >> 1) * 8 + 2t + (i & 1)
        const int nn = i >> 1, jj = i & 1, step = nn * 8 + 2 * t + jj;
        d[i] = fmaf(q[nn][jj], xq[nn][jj], q[nn][2 + jj] * xq[nn][2 + jj]);
        d[4 + i] = fmaf(o[nn][jj], xk[nn][jj], o[nn][2 + jj] * xk[nn][2 + jj]);
        nq[i] = norm[step];
        nk[i] = norm[DC + step];
      }
      reduce_scatter<8, 8, 4>(d, lane);   // lane g has sum g over the eight
      dots[((g >> 2) * DC + (g & 2) * 4 + 2 * t + (g & 1)) * NW + warp] = d[0];
      float bt = 0.f;
      if (warp == 0 && lane < DC) bt = reinterpret_cast<const float*>(slot + R::OB)[lane];
      bar_sync(SM::DOTS, 32 * NW);
      if (it + 2 < nchunks) bar_arrive(SM::GV_EMPTY + b, SM::NGV);
      if (it + S < nchunks) bar_arrive(R::empty(s), NT);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int nn = i >> 1, jj = i & 1, step = nn * 8 + 2 * t + jj;
        float w[NW], dq = 0.f, dk = 0.f;
        ld_vec<NW>(dots + step * NW, w);
#pragma unroll
        for (int j = 0; j < NW; ++j) dq += w[j];
        ld_vec<NW>(dots + (DC + step) * NW, w);
#pragma unroll
        for (int j = 0; j < NW; ++j) dk += w[j];
        const float iq = __fdividef(1.f, nq[i]), ik = __fdividef(1.f, nk[i]);
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const float aq = xq[nn][2 * hh + jj] * nq[i], ak = xk[nn][2 * hh + jj] * nk[i];
          q[nn][2 * hh + jj] = (q[nn][2 * hh + jj] - dq) * iq * (aq > 1.f ? 1.f : aq);
          o[nn][2 * hh + jj] = (o[nn][2 * hh + jj] - dk) * ik * (ak > 1.f ? 1.f : ak);
        }
      }
      gb *= bt * (1.f - bt);
    }
    store_steps<TIO>(qp, p.gQ.sl, left, q);
    store_steps<TIO>(kp, gkv.sl, left, o);
    qp -= DC * p.gQ.sl;
    kp -= DC * gkv.sl;
    if (warp == 0 && lane < nt) {
      char* y = PACKED ? p.gQ.row(n, h, t0 + lane) + 3 * E * sizeof(TIO) : p.gbeta.row(n, h, t0 + lane);
      from_f32(*reinterpret_cast<TIO*>(y), gb);
    }
  }
#pragma unroll
  for (int j = 0; j < E / 16; ++j) {
    float w[2][4];
    tm_ld(tm + j * 16, w);
    tm_ld_wait(w);
    finite = fmaf(0.f, ((w[0][0] + w[0][1]) + (w[0][2] + w[0][3])) + ((w[1][0] + w[1][1]) + (w[1][2] + w[1][3])), finite);
  }
  const bool ok = bar_all(SM::LAST, 32 * DeltaBwdRoles<TIO, E, NPW, PACKED>::WARPS, finite == 0.f);
  if (ok) {   // W_0, in place
#pragma unroll
    for (int j = 0; j < E / 16; ++j) {
      float w[2][4];
      tm_ld(tm + j * 16, w);
      tm_ld_wait(w);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float2*>(Wg + (i & 1) * 8 * E + 16 * j + (i >> 1) * 8) = make_float2(w[i >> 1][(i & 1) * 2], w[i >> 1][(i & 1) * 2 + 1]);
    }
  }
  bar_sync(SM::GP_EMPTY, 64 * NW);
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm0), "r"(2 * E));
  return ok;
}

template <typename TIO, int E, int NPW, int S, int MINB, bool PACKED>
__global__ void __launch_bounds__(32 * DeltaBwdRoles<TIO, E, NPW, PACKED>::WARPS, MINB) delta_bwd_chunk_kernel(const __grid_constant__ DeltaBwdParams p) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int n = blockIdx.x / p.H, h = blockIdx.x % p.H;
  extern __shared__ __align__(16) unsigned char smem[];
  int role, w;   // 0 chain, 1 W, 2 G, 3 prep
  constexpr int NW = E / 16, SW = DeltaBwdRoles<TIO, E, NPW, PACKED>::SW;
  if (warp < NW) { role = 0; w = warp; }
  else if (warp < (1 + SW) * NW) { role = SW == 1 ? 1 : 1 + (warp & 1); w = (warp - NW) / SW; }
  else { role = 3; w = warp - (1 + SW) * NW; }
  constexpr int P = 32 * DeltaBwdRoles<TIO, E, NPW, PACKED>::WARPS, LAST = DeltaChunkBwdSmem<TIO, E, NPW, S, PACKED>::LAST;
  bool ok = true;
  if (role == 0) ok = delta_bwd_chain_warp<TIO, E, NPW, S, PACKED>(p, smem, w, lane, n, h);
  else if (role != 3 && SW == 1) {
    if constexpr (SW == 1) ok = delta_bwd_rows_warp<TIO, E, NPW, S, PACKED>(p, smem, w, lane, n, h);
  } else if (role != 3) {
    if constexpr (SW == 2) ok = delta_bwd_state_warp<TIO, E, NPW, S, PACKED>(p, smem, role == 2, w, lane, n, h);
  } else {
    delta_prep_warp<TIO, E, NPW, S, PACKED, true>(p, smem, w, lane, n, h);
    ok = bar_all(LAST, P, true);
  }
  if (!ok) delta_bwd_again<TIO, E, PACKED, P, LAST>(p, n, h);
}

}  // namespace srwm
