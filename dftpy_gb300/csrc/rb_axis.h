// Axis description of the register-blocked FFT passes (fft_rb.cuh): which
// radices a length is transformed with.  Part of the plan; made on the host.
#pragma once
#include <cuda_runtime.h>

namespace gbrb {

// exact division by a small constant: q = n / d for n d < 2^32
struct FastDiv {
  unsigned d, m;
  __host__ void set(unsigned dd) {
    d = dd;
    m = d > 1 ? (unsigned)((0x100000000ull + d - 1) / d) : 0u;
  }
  __device__ __forceinline__ unsigned div(unsigned n) const { return d > 1 ? __umulhi(n, m) : n; }
};

// One axis: its length, radices in stage order and their divisors.
struct RbAxis {
  int n, nst;
  int r[8];        // radix of stage s
  int nb[8];       // n / r[s]: butterflies of a line in stage s
  int p[8];        // product of the radices before stage s
  FastDiv dnb[8], dp[8];
};

// The radices of a length in stage order (reverse: the other way round); nst = 0
// when the length has a prime factor above 7.  FP64: composite radices up to 16,
// as few stages as possible, largest first.  FP32: 8, 4, 2, 3, 5, 7 (the kernels of
// one length have their own order, in the lists of passes_rb.cuh).
RbAxis rb_axis(int n, bool f64, bool reverse);

// Lengths whose FP32 row passes form sqrt(rho) as rho rsqrt(rho); the others take
// the correctly rounded root, and every length keeps the one that it has had.  The
// G^2 kernel amplifies the root's rounding to that of the whole potential: with the
// rounded root these seven give von Weizsaecker potentials 1 to 5 % closer to the
// FP64 ones (rms over eight densities, 2.01e-5 -> 1.91e-5 at n2 = 128), in the same
// time, but other ones, up to 4.5e-5 of a 128^3 potential away from their present
// values, which is as much as those are off.
bool rb_rsqrt_length(int n);

}  // namespace gbrb
