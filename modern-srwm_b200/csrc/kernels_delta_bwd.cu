// Instantiations of the delta-rule backward kernels for every compiled configuration (configs.h).
// Built twice: -DSRWM_TIO_BF16=0 (fp32 streams) and -DSRWM_TIO_BF16=1 (bf16 streams).
#include "configs.h"
#include "launch.h"

namespace srwm {
namespace {

#if SRWM_TIO_BF16
typedef __nv_bfloat16 TIO;
#else
typedef float TIO;
#endif

// The packed (layer-level) form of a call runs the LAYER instantiation of a configuration.
template <int E, int V, int P, int R, int T, bool PK, int MINB, int LAYER>
int run(const DeltaBwdParams& p, int grid, cudaStream_t s, KernelInfo* info, int describe_only, int* cuda_err) {
  if (p.flags & F_PACKED) {
    if constexpr (LAYER) {
      constexpr int smem = DeltaBwdSmem<TIO, E, P, T, true>::TOTAL;
      if (info) { info->P = P; info->R = R; info->T = T; info->smem = smem; info->id = V; }
      if (describe_only) return 0;
      static unsigned long long dev_mask_pk = 0;
      return launch_kernel(delta_bwd_kernel<TIO, E, P, R, T, PK, MINB, true>, p, grid, P, smem, s, &dev_mask_pk, cuda_err);
    } else {
      return -6;
    }
  }
  constexpr int smem = DeltaBwdSmem<TIO, E, P, T>::TOTAL;
  if (info) { info->P = P; info->R = R; info->T = T; info->smem = smem; info->id = V; }
  if (describe_only) return 0;
  static unsigned long long dev_mask = 0;
  return launch_kernel(delta_bwd_kernel<TIO, E, P, R, T, PK, MINB>, p, grid, P, smem, s, &dev_mask, cuda_err);
}

template <int E, int V, int NPF, int SF, int MF, int NPB, int SB, int MB>
int run_chunk(const DeltaBwdParams& p, int grid, cudaStream_t s, KernelInfo* info, int describe_only, int* cuda_err) {
  auto go = [&](auto packed) {
    constexpr bool PACKED = decltype(packed)::value;   // (larger slots; one named barrier more)
    constexpr bool F32 = sizeof(TIO) == 4;
    constexpr int N = PACKED ? (E == 64 ? 2 : 1) : (F32 ? NPF : NPB), S = PACKED ? 2 : (F32 ? SF : SB), MINB = PACKED || F32 ? MF : MB;
    constexpr int P = 32 * DeltaBwdRoles<TIO, E, N, PACKED>::WARPS;
    constexpr int smem = DeltaChunkBwdSmem<TIO, E, N, S, PACKED>::TOTAL;
    if (info) { info->P = P; info->R = 16; info->T = DC; info->smem = smem; info->id = V; }
    if (describe_only) return 0;
    static unsigned long long dev_mask = 0;
    return launch_kernel(delta_bwd_chunk_kernel<TIO, E, N, S, MINB, PACKED>, p, grid, P, smem, s, &dev_mask, cuda_err);
  };
  return (p.flags & F_PACKED) ? go(std::true_type()) : go(std::false_type());
}

int by_id(int E, int variant, const DeltaBwdParams& p, int grid, cudaStream_t s, KernelInfo* info, int describe_only,
          int* cuda_err) {
#define X(E_, V_, P_, R_, T_, PK_, MINB_, LAYER_) \
  if (E == E_ && variant == V_) return run<E_, V_, P_, R_, T_, PK_, MINB_, LAYER_>(p, grid, s, info, describe_only, cuda_err);
  DELTA_BWD_CONFIGS(X)
#undef X
#define C(E_, V_, NPF_, SF_, MF_, NPB_, SB_, MB_) \
  if (E == E_ && variant == V_) return run_chunk<E_, V_, NPF_, SF_, MF_, NPB_, SB_, MB_>(p, grid, s, info, describe_only, cuda_err);
  DELTA_BWD_CHUNK_CONFIGS(C)
#undef C
  return (E == 8 || E == 16 || E == 32 || E == 64) ? -6 : -3;
}

}  // namespace

// Automatic choice.  Measured, 256 steps, tile / chunk kernel:
//   E = 64 bf16  16 sequences 108 / 53 us, 592: 264 / 207, 2368: 1002 / 808   fp32: 101 / 80, 296: 160 / 166, 592: 269 / 322
//   E = 32 bf16  111 / 27, 592: 119 / 80, 2368: 337 / 296                     fp32: 101 / 39, 296: 103 / 59, 592: 105 / 113
//   E = 16 bf16  63 / 21, 592: 65 / 46, 1184: 86 / 97                         fp32: 65 / 24, 592: 68 / 62, 1184: 82 / 122
// bf16 rows at E >= 32 take the chunk kernel at every size; fp32 rows (and the packed form, whose prepared rows
// are fp32) cost it twice the tensor work, so it takes them only while all sequences are resident at once.
// Tiles at E = 64: configuration 2 (64 threads per sequence) keeps four sequences resident per
// multiprocessor and has the best throughput on full waves, but a sequence takes the same time whether its
// multiprocessor holds four sequences or three: a partial last wave costs a whole one.  So the call is
// split: whole waves on configuration 2, the sequences of the remainder on configuration 3 with twice the
// threads per sequence (shorter step latency; 432 sequences: 1.84 against 2.09 ms), launched behind
// them on the same stream.  (Four times the threads was measured too: slower at every grid size.)
// (At E = 16 the packed form has one prep warp either way.)
inline int auto_variant(int E, bool packed, int grid, int sms) {
  const bool fp32_rows = sizeof(TIO) == 4 || packed;
  if (E == 16) return !packed && (grid <= 2 * sms || (fp32_rows && grid <= 4 * sms)) ? 3 : (grid <= 4 * sms ? 2 : 1);
  if (E == 32) return !fp32_rows || grid <= 2 * sms ? 1 : 2;
  if (E == 64) return !fp32_rows || grid <= sms ? 1 : 2;
  return 1;
}

#if SRWM_TIO_BF16
int dispatch_delta_bwd_bf16(
#else
int dispatch_delta_bwd_f32(
#endif
    int E, int variant, const DeltaBwdParams& p, int grid, cudaStream_t s, KernelInfo* info, int describe_only,
    int* cuda_err, int sms) {
  const int n_sm = current_sms(sms, describe_only);
  const bool split = variant == 0 && E == 64 && !(p.flags & F_PACKED);   // configuration 3 has no packed form
  if (variant == 0) variant = auto_variant(E, (p.flags & F_PACKED) != 0, grid, n_sm);
  if (!split || variant != 2) return by_id(E, variant, p, grid, s, info, describe_only, cuda_err);
  const int wave = 4 * n_sm;                       // sequences resident at once with configuration 2
  int full = (grid / wave) * wave, rest = grid - full;
  // Beyond a few waves the multiprocessors drift apart and a single launch fills the gaps by itself
  // (8192 sequences: 13.5 ms in one launch, 13.7 ms split); a remainder that nearly fills a wave is
  // left with the whole waves as well.
  if (grid > 3 * wave || rest * 10 > wave * 9) { full = grid; rest = 0; }
  constexpr int tail_id = 3;                       // 128 threads per sequence
  if (describe_only) return by_id(E, full > 0 ? 2 : tail_id, p, grid, s, info, 1, cuda_err);
  if (full > 0) {
    const int rc = by_id(E, 2, p, full, s, info, 0, cuda_err);
    if (rc != 0 || rest == 0) return rc;
  }
  DeltaBwdParams q = p;
  q.seq0 = p.seq0 + full;
  return by_id(E, tail_id, q, rest, s, full > 0 ? nullptr : info, 0, cuda_err);
}

}  // namespace srwm
