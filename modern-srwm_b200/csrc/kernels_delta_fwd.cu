// Instantiations of the delta-rule forward kernels for every compiled configuration (configs.h).
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
int run(const DeltaFwdParams& p, int grid, cudaStream_t s, KernelInfo* info, int describe_only, int* cuda_err) {
  if (p.flags & F_PACKED) {
    if constexpr (LAYER) {
      constexpr int smem = DeltaFwdSmem<TIO, E, T, true>::TOTAL;
      if (info) { info->P = P; info->R = R; info->T = T; info->smem = smem; info->id = V; }
      if (describe_only) return 0;
      static unsigned long long dev_mask_pk = 0;
      return launch_kernel(delta_fwd_kernel<TIO, E, P, R, T, PK, MINB, true>, p, grid, P, smem, s, &dev_mask_pk, cuda_err);
    } else {
      return -6;
    }
  }
  constexpr int smem = DeltaFwdSmem<TIO, E, T>::TOTAL;
  if (info) { info->P = P; info->R = R; info->T = T; info->smem = smem; info->id = V; }
  if (describe_only) return 0;
  static unsigned long long dev_mask = 0;
  return launch_kernel(delta_fwd_kernel<TIO, E, P, R, T, PK, MINB>, p, grid, P, smem, s, &dev_mask, cuda_err);
}

template <int E, int V, int NPW, int S, int MINB>
int run_chunk(const DeltaFwdParams& p, int grid, cudaStream_t s, KernelInfo* info, int describe_only, int* cuda_err) {
  constexpr int P = 32 * (E / 16 + NPW);
  auto go = [&](auto packed) {
    constexpr bool PACKED = decltype(packed)::value;
    constexpr int smem = DeltaRing<TIO, E, NPW, S, PACKED, false>::BYTES;
    if (info) { info->P = P; info->R = 16; info->T = DC; info->smem = smem; info->id = V; }
    if (describe_only) return 0;
    static unsigned long long dev_mask = 0;
    return launch_kernel(delta_fwd_chunk_kernel<TIO, E, NPW, S, MINB, PACKED>, p, grid, P, smem, s, &dev_mask, cuda_err);
  };
  return (p.flags & F_PACKED) ? go(std::true_type()) : go(std::false_type());
}

// Automatic choice.  The chunk kernel takes a step in a third to a sixth of the tile kernel's time and keeps
// 2 (E = 64), 4 (32) or 8 (16) sequences resident per multiprocessor.  Measured, 256 steps, tile / chunk:
//   E = 64 fp32  16 sequences 66 / 33 us, 592: 123 / 102, 2368: 397 / 374    bf16: 70 / 21, 137 / 69, 439 / 251
//   E = 32 fp32  16: 75 / 20, 592: 79 / 46, 2368: 202 / 165                  bf16: 74 / 15, 81 / 31, 172 / 114
//   E = 16 fp32  16: 54 / 23, 1184: 62 / 58, 2368: 86 / 110                  bf16: 43 / 20, 54 / 49, 81 / 107
// so only at E = 16, where a chunk's fixed work (the 16 x 16 inverse) is most of it, do grids beyond one
// wave of the chunk kernel go to register tiles.
inline int auto_variant(int E, int grid, int sms) { return E == 16 && grid <= 8 * sms ? 2 : 1; }

}  // namespace

#if SRWM_TIO_BF16
int dispatch_delta_fwd_bf16(
#else
int dispatch_delta_fwd_f32(
#endif
    int E, int variant, const DeltaFwdParams& p, int grid, cudaStream_t s, KernelInfo* info, int describe_only,
    int* cuda_err, int sms) {
  if (variant == 0) variant = auto_variant(E, grid, current_sms(sms, describe_only));
#define X(E_, V_, P_, R_, T_, PK_, MINB_, LAYER_) \
  if (E == E_ && variant == V_) return run<E_, V_, P_, R_, T_, PK_, MINB_, LAYER_>(p, grid, s, info, describe_only, cuda_err);
  DELTA_FWD_CONFIGS(X)
#undef X
#define C(E_, V_, NPW_, S_, MINB_) \
  if (E == E_ && variant == V_) return run_chunk<E_, V_, NPW_, S_, MINB_>(p, grid, s, info, describe_only, cuda_err);
  DELTA_FWD_CHUNK_CONFIGS(C)
#undef C
  return (E == 8 || E == 16 || E == 32 || E == 64) ? -6 : -3;
}

}  // namespace srwm
