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

// Automatic choice.  Measured, 256 steps, tile / chunk kernel, us:
//   E = 64 bf16  16 sequences 161 / 47, 592: 274 / 167, 2368: 1024 / 621
//          fp32  16: 156 / 70, 148: 159 / 78, 256: 160 / 123, 400: 226 / 184, 592: 271 / 236, 888: 404 / 345, 2368: 1011 / 886
//   E = 32 bf16  111 / 27, 592: 119 / 80, 2368: 337 / 296                     fp32: 101 / 39, 296: 103 / 59, 592: 105 / 113
//   E = 16 bf16  63 / 21, 592: 65 / 46, 1184: 86 / 97                         fp32: 65 / 24, 592: 68 / 62, 1184: 82 / 122
//   E = 64 packed  fp32  16: 126 (chunks with one sequence a multiprocessor) / 110, 148: 131 / 131, 256: 201 / 160, 400: 296 / 305,
//          2368: 1161 / 1195;  bf16  16: 119 / 105, 148: 124 / 125, 256: 197 / 147, 297: 290 / 239, 400: 293 / 275, 592: 300 / 279,
//          600: 461 / 388, 888: 471 / 416, 1184: 589 / 569, 2368: 1158 / 1134
// So the chunk kernel at E = 64, where two sequences share a multiprocessor, and with bf16 rows at 32.  fp32 rows at E = 32, and packed
// ones at 64, whose upstream rows are three pieces as well, only while all sequences are resident at once; so packed rows at 32, which
// take longer to prepare.  (At E = 16 the packed form has one prep warp either way.)
inline int auto_variant(int E, bool packed, int grid, int sms) {
  const bool fp32_rows = sizeof(TIO) == 4 || packed;
  if (E == 16) return !packed && (grid <= 2 * sms || (fp32_rows && grid <= 4 * sms)) ? 3 : (grid <= 4 * sms ? 2 : 1);
  if (E == 32) return !fp32_rows || grid <= 2 * sms ? 1 : 2;
  if (E == 64) return !packed || sizeof(TIO) == 2 || grid <= 2 * sms ? 1 : 2;
  return 1;
}

#if SRWM_TIO_BF16
int dispatch_delta_bwd_bf16(
#else
int dispatch_delta_bwd_f32(
#endif
    int E, int variant, const DeltaBwdParams& p, int grid, cudaStream_t s, KernelInfo* info, int describe_only,
    int* cuda_err, int sms) {
  if (variant == 0) variant = auto_variant(E, (p.flags & F_PACKED) != 0, grid, current_sms(sms, describe_only));
  return by_id(E, variant, p, grid, s, info, describe_only, cuda_err);
}

}  // namespace srwm
