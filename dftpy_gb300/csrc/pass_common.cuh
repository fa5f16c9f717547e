// Host and device helpers shared by the FFT pass kernels.
#pragma once
#include "plan.h"

namespace gbct {

constexpr double kZero = 1e-30;                       // dftpy ZERO

// A scalar kernel parameter in both precisions, converted on the host: the
// FP32 kernels then run without double->float conversions, which execute on
// the FP64 pipe (a slow one on this part).
struct Sc {
  double d;
  float f;
  void set(double v) { d = v; f = (float)v; }
};
template <typename T> __device__ __forceinline__ T sc(const Sc& s) {
  if constexpr (sizeof(T) == 8) return s.d; else return s.f;
}

// Raise a kernel's dynamic shared-memory limit once to the largest size it
// has been launched with (keyed by kernel address and device).
template <typename K> inline int ct_smem(K kern, size_t bytes) {
  if (bytes <= 40 * 1024) return 0;   // 48 KB, less the kernels' static arrays
  return gb_smem_grant(reinterpret_cast<const void*>(kern), (int)bytes);
}

}  // namespace gbct
