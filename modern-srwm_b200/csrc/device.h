// Multiprocessors of the current device, by which choices depend on the grid.
#pragma once
#include <cuda_runtime.h>

namespace srwm {

constexpr int DEFAULT_SMS = 148;

// Multiprocessor count of the current device (cached per device ordinal).
inline int current_sms(int hint, int describe_only) {
  if (hint > 0) return hint;
  if (describe_only) return DEFAULT_SMS;
  static int cache[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { (void)cudaGetLastError(); return DEFAULT_SMS; }
  int& c = cache[dev & 63];
  int v = __atomic_load_n(&c, __ATOMIC_RELAXED);
  if (v <= 0) {
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) {
      (void)cudaGetLastError();
      v = DEFAULT_SMS;
    }
    __atomic_store_n(&c, v, __ATOMIC_RELAXED);
  }
  return v;
}

// The same where a call asks several times and a small one would notice (cudaGetDevice, 30 ns each): the count of the device that
// was current at the first question, so that a question for scratch and the launch that uses it always agree.
inline int common_sms() {
  static const int v = current_sms(0, 0);
  return v;
}

}  // namespace srwm
