// The FFT passes of a 3D grid on the register-blocked lines of fft_rb.cuh
// (any axis length with prime factors up to 7; other lengths run in passes.cu).
//
// Layouts and semantics are those of passes.cu.  Per pass:
//   k_rb_cols      one CTA transforms a tile of 16 (FP32) or 8 (FP64) columns =
//                  128 contiguous bytes per line element.  The first stage
//                  reads global memory into registers and the last one
//                  writes it from registers, so a column crosses shared
//                  memory once per pair of stages.  Tiles run over the columns
//                  of all outer indices back to back, so a half spectrum of
//                  n2/2 + 1 columns leaves no nearly empty last tile.
//                  CONV: axis-0 forward, kernel multiply and the inverse's
//                  first stage in the same registers.
//   k_rb_rows_fwd  prologues, R2C of row pairs.
//   k_rb_rows_inv  C2R of row pairs: the first stage reads the half spectrum
//                  straight from global memory, the last one leaves every
//                  field of a point with one thread, which runs the epilogue.
#pragma once
#include <math.h>
#include <string.h>

#include "fft_rb.cuh"
#include "gkernels.cuh"
#include "pass_common.cuh"
#include "plan.h"

// FP32 lengths with kernels of their own: the even 2, 3, 5, 7-smooth lengths
// from 24 to 400 whose radices split into two stages of at most 25, and eight of
// those that need three (196, 210, 224, 256, 280, 288, 320, 360).  294, 324, 350,
// 384, 392, odd and longer lengths run the kernels of run-time lengths.
#define GB_RB_LENGTHS_1(X) \
  X(24, GB_RB_G(8), GB_RB_G(3)) X(28, GB_RB_G(4), GB_RB_G(7)) X(30, GB_RB_G(2, 3), GB_RB_G(5)) \
  X(32, GB_RB_G(8), GB_RB_G(4)) X(36, GB_RB_G(4), GB_RB_G(3, 3)) X(40, GB_RB_G(8), GB_RB_G(5)) \
  X(42, GB_RB_G(2, 3), GB_RB_G(7)) X(48, GB_RB_G(8), GB_RB_G(2, 3)) X(50, GB_RB_G(2, 5), GB_RB_G(5)) \
  X(54, GB_RB_G(2, 3), GB_RB_G(3, 3)) X(56, GB_RB_G(8), GB_RB_G(7)) X(60, GB_RB_G(4, 3), GB_RB_G(5)) \
  X(64, GB_RB_G(8), GB_RB_G(8)) X(70, GB_RB_G(2, 5), GB_RB_G(7)) X(72, GB_RB_G(8), GB_RB_G(3, 3)) \
  X(80, GB_RB_G(8), GB_RB_G(2, 5)) X(84, GB_RB_G(4, 3), GB_RB_G(7)) X(90, GB_RB_G(2, 3), GB_RB_G(3, 5)) \
  X(96, GB_RB_G(8), GB_RB_G(4, 3)) X(98, GB_RB_G(2, 7), GB_RB_G(7))
#define GB_RB_LENGTHS_2(X) \
  X(100, GB_RB_G(4, 5), GB_RB_G(5)) X(108, GB_RB_G(4, 3), GB_RB_G(3, 3)) X(112, GB_RB_G(8), GB_RB_G(2, 7)) \
  X(120, GB_RB_G(8), GB_RB_G(3, 5)) X(126, GB_RB_G(2, 3, 3), GB_RB_G(7)) X(128, GB_RB_G(8), GB_RB_G(4, 4)) \
  X(140, GB_RB_G(4, 5), GB_RB_G(7)) X(144, GB_RB_G(8, 2), GB_RB_G(3, 3)) \
  X(150, GB_RB_G(2, 3), GB_RB_G(5, 5)) X(160, GB_RB_G(8), GB_RB_G(4, 5)) \
  X(162, GB_RB_G(2, 3, 3), GB_RB_G(3, 3))
#define GB_RB_LENGTHS_3(X) \
  X(168, GB_RB_G(8), GB_RB_G(3, 7)) X(180, GB_RB_G(4, 3), GB_RB_G(3, 5)) X(192, GB_RB_G(8), GB_RB_G(8, 3)) \
  X(200, GB_RB_G(8), GB_RB_G(5, 5)) X(216, GB_RB_G(8, 3), GB_RB_G(3, 3)) \
  X(240, GB_RB_G(8, 2), GB_RB_G(3, 5)) X(250, GB_RB_G(2, 5), GB_RB_G(5, 5))
#define GB_RB_LENGTHS_4(X) \
  X(252, GB_RB_G(4, 3), GB_RB_G(3, 7)) X(270, GB_RB_G(2, 3, 3), GB_RB_G(3, 5)) \
  X(300, GB_RB_G(4, 3), GB_RB_G(5, 5)) X(336, GB_RB_G(8, 2), GB_RB_G(3, 7)) \
  X(378, GB_RB_G(2, 3, 3), GB_RB_G(3, 7)) X(400, GB_RB_G(8, 2), GB_RB_G(5, 5))
#define GB_RB_LENGTHS3(X) \
  X(196, GB_RB_G(4), GB_RB_G(7), GB_RB_G(7)) X(210, GB_RB_G(2, 3), GB_RB_G(5), GB_RB_G(7)) \
  X(224, GB_RB_G(8), GB_RB_G(4), GB_RB_G(7)) X(256, GB_RB_G(8), GB_RB_G(8), GB_RB_G(4)) \
  X(280, GB_RB_G(8), GB_RB_G(5), GB_RB_G(7)) X(288, GB_RB_G(8), GB_RB_G(4), GB_RB_G(3, 3)) \
  X(320, GB_RB_G(8), GB_RB_G(8), GB_RB_G(5)) X(360, GB_RB_G(8), GB_RB_G(5), GB_RB_G(3, 3))

#ifndef GB_RB_GROUP
#define GB_RB_GROUP 0
#endif
#define GB_RB_CAT2(a, b) a##b
#define GB_RB_CAT(a, b) GB_RB_CAT2(a, b)

namespace gbrb {

using gbct::Sc;
using gbct::kZero;
using gbct::sc;

// element j of a line in shared memory: one complex value of padding per 128
// bytes, so the stride-radix writes of a first stage spread over the banks
template <typename T> __device__ __forceinline__ int sidx(int j) {
  constexpr int S = sizeof(T) == 4 ? 4 : 3;
  return j + (j >> S);
}
template <typename T> __host__ __device__ inline int line_pitch(int n) {
  constexpr int S = sizeof(T) == 4 ? 4 : 3;
  return n + (n >> S) + 1;
}

// ---- FP64 elementary functions from single-precision seeds -------------------
// x^(-1/6), x in the float range: one third-order (Halley-type) step on the
// seed, y (1 + r/6 + 7 r^2/72) with r = 1 - x y^6 (|r| < 1e-5, so the next term
// is below 1e-16)
__device__ __forceinline__ double rroot6(double x) {
  const double y = (double)rsqrtf(cbrtf((float)x));
  const double y2 = y * y;
  const double r = fma(-x, y2 * y2 * y2, 1.0);
  return fma(y * r, fma(r, 7.0 / 72.0, 1.0 / 6.0), y);
}

// The roots of a positive density that the terms are made of: x^(1/3), x^(-1/3),
// x^(-1/2) and (FP64) x^(-1/6), from single-precision seeds.  x^(1/3), x^(-1/3) and
// x^(-1/6) each end in a correction by r = 1 - x y0^6, a third of whose roundings
// reaches them, so they are good to about one rounding themselves, and the terms to
// no more than library calls of cbrt, sqrt and division gave them (rms error of the
// potentials in 2^-53, 24 x 20 x 84: Thomas-Fermi 1.0, LDA 0.6; library 1.2, 0.7;
// powers of one x^(-1/6), 14 FP64 operations against 17, 1.6 and 1.7).  x^(-1/2), a
// product of two (0.8 rms), only ever meets a convolution's result, whose error is
// thousands of roundings.
template <typename T> struct Roots { T c, z3, z2, y; };
__device__ __forceinline__ Roots<double> roots(double x) {
  const double y0 = (double)rsqrtf(cbrtf((float)x));     // (its square is exact)
  const double y2 = y0 * y0, c0 = x * (y2 * y2), r = fma(-c0, y2, 1.0);
  Roots<double> q;
  q.z3 = fma(y2 * r, fma(r, 2.0 / 9.0, 1.0 / 3.0), y2);
  q.c = fma(c0 * r, fma(r, 5.0 / 9.0, 2.0 / 3.0), c0);
  q.y = fma(y0 * r, fma(r, 7.0 / 72.0, 1.0 / 6.0), y0);
  q.z2 = q.y * q.z3;
  return q;
}
__device__ __forceinline__ Roots<float> roots(float x) {
  const float a = rcbrtf(x), b = rsqrtf(x);
  const float a2 = a * a, c = x * a2, s = x * b;
  Roots<float> q;
  q.z3 = a;
  q.z2 = fmaf(b * fmaf(-s, b, 1.0f), 0.5f, b);
  q.c = fmaf(fmaf(-(c * c), c, x), a2 * (1.0f / 3.0f), c);
  q.y = 0.0f;
  return q;
}
// x^(1/2) and x^(5/6) of the forward rows.  FP64: from x^(-1/6); one more Newton
// step for the square root, whose rounding the G^2 kernel amplifies.
template <typename T> struct Powers { T sq, p56; };
__device__ __forceinline__ Powers<double> powers(double x) {
  const double y = rroot6(x), z2 = y * y * y, s = x * z2;
  return Powers<double>{fma(0.5 * z2, fma(-s, s, x), s), x * y};
}
__device__ __forceinline__ Powers<float> powers(float x) {
  const Roots<float> r = roots(x);
  return Powers<float>{x * rsqrtf(x), x * r.z2 * r.c};
}

// ---- forward rows ---------------------------------------------------------------
struct RowsFwd {
  const void* in[GB_RB_FIELDS];   // per field (the derived kinds read in[0])
  void* out[GB_RB_FIELDS];
  int nrows, n2h, ld2, nf, lp;
  int op[GB_RB_FIELDS];
  int b56, rsq;           // rsq: sqrt(rho) as rho rsqrt(rho) (FP32)
  Sc beta, beta2, half, rho0, inv0;
  RbAxis ax;
  FastDiv dn, dnh;
  const void* tw;
  // PK_WGC, FP64: keep rho^beta and rho^beta2 / take rho^beta from an earlier launch
  void *pw_out, *pw2_out;
  const void* pw_in;
};

template <typename T>
__device__ __noinline__ T pow_general(T x, T b) { return pow(x, b); }
template <typename T>
__device__ __noinline__ T sqrt_call(T x) { return sqrt(x); }

// x^b.  FP64: exp(b ln x), one logarithm for both exponents where two powers
// of a density are wanted; its relative error, |b ln x| ulp, is below 1e-14 for
// x >= 1e-30.
__device__ __forceinline__ float pow_of(float x, float b) { return powf(x, b); }
__device__ __forceinline__ double pow_of(double x, double b) { return exp(b * log(x)); }

// Prologues of the forward rows.  A kernel per kind: a plain transform holds
// none of the root arithmetic (the compiler would compute it ahead of the
// branch, at 12 FP64 operations a point).
// PK_WGC: the three fields rho^e, u rho^e, u^2 rho^e of one exponent.
enum { PK_PLAIN = 0, PK_ROOTS = 1, PK_GENERAL = 2, PK_WGC = 3 };

// the values of one density that the derived fields are made of
template <typename T> struct Derived { T rho, sq, b, u; };
template <typename T, int KIND>
__device__ __forceinline__ Derived<T> derived(const RowsFwd& a, T rho) {
  Derived<T> d;
  d.rho = d.sq = d.b = d.u = rho;
  if constexpr (KIND == PK_WGC) {
    const T rc = rho > (T)kZero ? rho : (T)kZero;
    d.u = (rc - sc<T>(a.rho0)) * sc<T>(a.inv0);
    if constexpr (sizeof(T) == 8) {
      if (!a.pw_in) {
        const T l = log(rc);
        d.b = exp(sc<T>(a.beta) * l);
        if (a.pw2_out) d.sq = exp(sc<T>(a.beta2) * l);      // kept for the other exponent's fields
      }
    } else {
      d.b = pow_of(rc, sc<T>(a.beta));
    }
  } else if constexpr (KIND != PK_PLAIN) {
    const T kz = (T)kZero;
    const T rc = rho < kz ? kz : rho;                    // a NaN stays one in the powers
    const Powers<T> r = powers(rc);
    d.sq = r.sq;
    if (sizeof(T) == 4 && !a.rsq) d.sq = sqrt(rc);
    if (!(rho >= kz)) d.sq = sqrt_call<T>(rho > (T)0 ? rho : kz);
    if constexpr (KIND == PK_ROOTS) d.b = r.p56;
    else d.b = pow_general<T>(rc, sc<T>(a.beta));
  }
  return d;
}
template <typename T, int KIND>
__device__ __forceinline__ T field_of(int op, const Derived<T>& d) {
  if constexpr (KIND == PK_PLAIN) return d.rho;
  if constexpr (KIND == PK_WGC) return op == OP_WGC0 ? d.b : (op == OP_WGC1 ? d.u * d.b : d.u * d.u * d.b);
  T v = d.rho;
  if (op == OP_SQRT) v = d.sq;
  else if (op == OP_POWB) v = d.b;
  return v;
}
// one derived field alone (FP32: the roots of a field cost less than passing
// every field through shared memory)
template <typename T>
__device__ __forceinline__ T field_direct(int op, T rho, bool rsq) {
  const T kz = (T)kZero;
  if (op == OP_SQRT) {
    const T rc = rho > (T)0 ? rho : kz;
    return rsq && rc >= kz ? rc * rsqrtf(rc) : sqrtf(rc);
  }
  if (op == OP_POWB) {
    const T rc = rho < kz ? kz : rho;
    return powers(rc).p56;
  }
  return rho;
}

// transform of all lines of the CTA between two shared buffers (line pitch
// ls); returns the buffer with the result.  FIRST = false: the first stage's
// results are in b already.
template <int DIR, bool FIRST, typename T, typename AX>
__device__ __forceinline__ cpx<T>* lines(cpx<T>* a, cpx<T>* b, int ls, int nl, const AX& ax,
                                         const cpx<T>* __restrict__ tw) {
  const int tid = threadIdx.x, nthr = blockDim.x, n = ax.n();
  if constexpr (FIRST) {
    ax.first([&](auto rc) {
      constexpr int R = decltype(rc)::R;
      const int nb = ax.nbf();
      for (int t0 = tid; t0 < nl * nb; t0 += nthr) {
        const int l = ax.div_nbf(t0), i = t0 - l * nb;
        cpx<T> u[R];
        const cpx<T>* src = a + l * ls;
#pragma unroll
        for (int t = 0; t < R; ++t) u[t] = src[sidx<T>(i + t * nb)];
        stage_first<DIR, T>(rc, u, tw, n);
        cpx<T>* dst = b + l * ls;
#pragma unroll
        for (int t = 0; t < R; ++t) dst[sidx<T>(i * R + t)] = u[t];
      }
    });
  }
  __syncthreads();
  cpx<T>* x = a;
  a = b;
  b = x;
  ax.middle([&](auto rc, auto nb, auto p, auto div_nb, auto div_p) {
    constexpr int R = decltype(rc)::R;
    for (int t0 = tid; t0 < nl * nb; t0 += nthr) {
      const int l = div_nb(t0), i = t0 - l * nb;
      const int k = i - p * div_p(i);
      cpx<T> u[R];
      load_stage<DIR, T>(rc, u, a + l * ls, tw, i, k, nb, p, n, sidx<T>);
      cpx<T>* dst = b + l * ls;
      const int j0 = (i - k) * R + k;
#pragma unroll
      for (int t = 0; t < R; ++t) dst[sidx<T>(j0 + t * p)] = u[t];
    }
    __syncthreads();
    cpx<T>* y = a;
    a = b;
    b = y;
  });
  if (ax.nst() < 2) return a;
  ax.last([&](auto rc) {
    constexpr int R = decltype(rc)::R;
    const int nb = ax.nbl();
    for (int t0 = tid; t0 < nl * nb; t0 += nthr) {
      const int l = ax.div_nbl(t0), i = t0 - l * nb;
      cpx<T> u[R];
      // the last stage writes the elements that it read
      cpx<T>* x = a + l * ls;
      load_stage<DIR, T>(rc, u, x, tw, i, i, nb, nb, n, sidx<T>);
#pragma unroll
      for (int t = 0; t < R; ++t) x[sidx<T>(i + t * nb)] = u[t];
    }
  });
  __syncthreads();
  return a;
}

// forward rows whose first stage reads global memory: FP32, fields of rho,
// sqrt(rho) and rho^(5/6), a first radix whose inputs fit in registers beside
// a field's butterfly
template <typename T, int KIND, typename AX> constexpr bool direct_rows() {
  if constexpr (sizeof(T) == 4 && AX::kFixed && KIND != PK_GENERAL)
    return AX::n() / AX::nbf() <= (KIND == PK_PLAIN ? 16 : KIND == PK_ROOTS ? 12 : 8);
  else return false;
}
template <typename T, int KIND, typename AX> constexpr bool kDirect = direct_rows<T, KIND, AX>();
// ... and that then needs one shared buffer only (two stages)
template <typename T, int KIND, typename AX> constexpr bool one_buffer() {
  if constexpr (direct_rows<T, KIND, AX>()) return AX::nst() == 2;
  else return false;
}

template <typename T, typename AX = AxRun<T>> struct RowCta {
  static constexpr int NT = sizeof(T) == 4 ? 128 : 96;      // threads of a row CTA, at most
  static constexpr int MINB = sizeof(T) == 8 || !AX::kFixed ? 4 : 7;   // resident CTAs per SM to allocate registers for
};

template <typename T, int KIND, typename AX>
__global__ void __launch_bounds__(RowCta<T>::NT, (RowCta<T, AX>::MINB)) k_rb_rows_fwd(const __grid_constant__ RowsFwd a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const AX ax(a.ax);
  const int n = ax.n(), lp = a.lp, ls = line_pitch<T>(n), nl = a.nf * lp;
  cpx<T>* A = reinterpret_cast<cpx<T>*>(smem_raw);
  cpx<T>* B = one_buffer<T, KIND, AX>() ? A : A + nl * ls;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int base = blockIdx.x * 2 * lp;
  const cpx<T>* tw = reinterpret_cast<const cpx<T>*>(a.tw);
  cpx<T>* res;
  if constexpr (kDirect<T, KIND, AX>) {
    // FP32: the first stage reads the rows from global memory and derives its
    // field in registers
    const bool rsq = a.rsq != 0;
    ax.first([&](auto rc) {
      constexpr int R = decltype(rc)::R;
      constexpr int nb = AX::nbf();
      for (int t0 = tid; t0 < lp * nb; t0 += nthr) {
        const int l = ax.div_nbf(t0), i = t0 - l * nb;
        const int ra = base + 2 * l;
        const int64_t off = (int64_t)ra * n + i;
        T x0[R], x1[R], b0[KIND == PK_WGC ? R : 1], b1[KIND == PK_WGC ? R : 1];
        auto load = [&](const void* p) {
          const T* src = reinterpret_cast<const T*>(p) + off;
#pragma unroll
          for (int t = 0; t < R; ++t) {
            x0[t] = ra < a.nrows ? __ldg(src + t * nb) : (T)0;
            x1[t] = ra + 1 < a.nrows ? __ldg(src + n + t * nb) : (T)0;
          }
        };
        load(a.in[0]);
        if constexpr (KIND == PK_WGC) {
#pragma unroll
          for (int t = 0; t < R; ++t) {
            const Derived<T> d0 = derived<T, KIND>(a, x0[t]), d1 = derived<T, KIND>(a, x1[t]);
            x0[t] = d0.u; b0[t] = d0.b;
            x1[t] = d1.u; b1[t] = d1.b;
          }
        }
        for (int f = 0; f < a.nf; ++f) {
          const int op = a.op[f];
          cpx<T> u[R];
          if constexpr (KIND == PK_WGC) {
#pragma unroll
            for (int t = 0; t < R; ++t) {
              const Derived<T> d0{x0[t], x0[t], b0[t], x0[t]}, d1{x1[t], x1[t], b1[t], x1[t]};
              u[t] = cpx<T>{field_of<T, KIND>(op, d0), field_of<T, KIND>(op, d1)};
            }
          } else if (op == OP_RHO || KIND == PK_PLAIN) {
            if (KIND == PK_PLAIN && f > 0 && a.in[f] != a.in[f - 1]) load(a.in[f]);
#pragma unroll
            for (int t = 0; t < R; ++t) u[t] = cpx<T>{x0[t], x1[t]};
          } else if (op == OP_SQRT) {
#pragma unroll
            for (int t = 0; t < R; ++t) u[t] = cpx<T>{field_direct<T>(OP_SQRT, x0[t], rsq), field_direct<T>(OP_SQRT, x1[t], rsq)};
          } else {
#pragma unroll
            for (int t = 0; t < R; ++t) u[t] = cpx<T>{field_direct<T>(OP_POWB, x0[t], rsq), field_direct<T>(OP_POWB, x1[t], rsq)};
          }
          stage_first<-1, T>(rc, u, tw, AX::n());
          cpx<T>* dst = B + (f * lp + l) * ls;
#pragma unroll
          for (int t = 0; t < R; ++t) dst[sidx<T>(i * R + t)] = u[t];
        }
      }
    });
    res = lines<-1, false, T>(A, B, ls, nl, ax, tw);
  } else {
#pragma unroll 2
    for (int idx = tid; idx < lp * n; idx += nthr) {
      const int l = AX::kFixed ? idx / n : (int)a.dn.div(idx), j = idx - l * n;
      const int ra = base + 2 * l;
      const bool ok0 = ra < a.nrows, ok1 = ra + 1 < a.nrows;
      const int64_t off = (int64_t)ra * n + j;
      cpx<T>* o = A + l * ls + sidx<T>(j);
      if constexpr (KIND == PK_PLAIN) {
        for (int f = 0; f < a.nf; ++f) {
          const T* src = reinterpret_cast<const T*>(a.in[f]) + off;
          o[f * lp * ls] = cpx<T>{ok0 ? __ldg(src) : (T)0, ok1 ? __ldg(src + n) : (T)0};
        }
      } else {
        const T* src = reinterpret_cast<const T*>(a.in[0]) + off;
        Derived<T> d0 = derived<T, KIND>(a, ok0 ? __ldg(src) : (T)0);
        Derived<T> d1 = derived<T, KIND>(a, ok1 ? __ldg(src + n) : (T)0);
        if constexpr (KIND == PK_WGC && sizeof(T) == 8) {
          if (a.pw_in) {
            const T* pw = reinterpret_cast<const T*>(a.pw_in) + off;
            if (ok0) d0.b = pw[0];
            if (ok1) d1.b = pw[n];
          }
          if (a.pw_out) {
            T* pw = reinterpret_cast<T*>(a.pw_out) + off;
            if (ok0) pw[0] = d0.b;
            if (ok1) pw[n] = d1.b;
          }
          if (a.pw2_out) {
            T* pw = reinterpret_cast<T*>(a.pw2_out) + off;
            if (ok0) pw[0] = d0.sq;
            if (ok1) pw[n] = d1.sq;
          }
        }
        for (int f = 0; f < a.nf; ++f)
          o[f * lp * ls] = cpx<T>{field_of<T, KIND>(a.op[f], d0), field_of<T, KIND>(a.op[f], d1)};
      }
    }
    __syncthreads();
    res = lines<-1, true, T>(A, B, ls, nl, ax, tw);
  }
  const T half = sc<T>(a.half);
  const int nh = AX::kFixed ? n / 2 + 1 : a.n2h;
  for (int f = 0; f < a.nf; ++f) {
    cpx<T>* o = reinterpret_cast<cpx<T>*>(a.out[f]);
    const cpx<T>* src = res + f * lp * ls;
    for (int idx = tid; idx < lp * nh; idx += nthr) {
      const int l = AX::kFixed ? idx / nh : (int)a.dnh.div(idx), k = idx - l * nh;
      const int ra = base + 2 * l;
      if (ra >= a.nrows) continue;
      const cpx<T> Z = src[l * ls + sidx<T>(k)];
      const cpx<T> Zc = src[l * ls + sidx<T>(k == 0 ? 0 : n - k)];
      cpx<T>* q = o + (int64_t)ra * a.ld2 + k;
      cpx<T> va = {Z.x + Zc.x, Z.y - Zc.y}, vb = {Z.y + Zc.y, Zc.x - Z.x};
      if (half != (T)1) {
        va = c_scale(va, half);
        vb = c_scale(vb, half);
      }
      q[0] = va;
      if (ra + 1 < a.nrows) q[a.ld2] = vb;
    }
  }
}

// ---- inverse rows ----------------------------------------------------------------
struct RowsInv {
  const void* in[GB_RB_FIELDS];
  int nrows, n2h, ld2, nf, lp;
  RbAxis ax;
  const void* tw;
  void* out;
  int64_t ostride;
  Sc scale;
  EvalDesc ev;
  Sc tf_v, tf_vl, tf_e, vw_y, half_vw, two_alpha, inv_two_alpha, wt_beta;
  int b56;
  const void* rho;
  const void* vloc;
  void* pot;
  double* partials;
  int base;             // the fused terms are wanted (else the WGC term alone)
  int add;              // add to pot
  // WGC term: its fields X0..X2 (Y0..Y2) are the line fields from slot wslot on
  int wgc, wslot, two;
  Sc w_rho0, w_inv0, w_a, w_b;
  const void *pa, *pb;  // FP64: rho^a and rho^b of the forward rows
  void* wstore[6];      // FP64: copies of the fields and of the potential (delta-evaluation reference)
  void* vstore;
};

// a call, so that the compiler cannot compute the logarithm of the r_s < 1
// branch for every point (35 FP64 operations)
static __device__ __noinline__ double log_call(double x) { return log(x); }
static __device__ __forceinline__ float log_call(float x) { return logf(x); }

// Perdew-Zunger 1981 LDA given the density's roots: potential and (want_e)
// energy per particle
template <typename T>
__device__ __forceinline__ void pz_lda(const Roots<T>& r, T& eps, T& pot, bool want_e) {
  const T a = (T)0.0311, b = (T)-0.048, c = (T)0.0020, d = (T)-0.0116;
  const T g = (T)-0.1423, b1 = (T)1.0529, b2 = (T)0.3334;
  const T cx = (T)0.98474502184269654115;                 // (3/pi)^(1/3)
  const T rc = r.c;
  const T rs = (T)0.62035049089940001667 * r.z3;          // (3/(4 pi))^(1/3) / rho^(1/3)
  pot = -cx * rc;
  eps = (T)(-0.75) * cx * rc;
  if (rs < (T)1) {
    const T lr = log_call(rs);
    pot += lr * (a + (T)(2.0 / 3.0) * c * rs) + b - (T)(1.0 / 3.0) * a + (T)(1.0 / 3.0) * ((T)2 * d - c) * rs;
    if (want_e) eps += a * lr + b + c * rs * lr + d * rs;
  } else {
    T sq;
    if constexpr (sizeof(T) == 8) sq = 0.78762331789974326286 * r.y;   // sqrt(0.62035...) rho^(-1/6)
    else sq = sqrt(rs);
    const T inv = rcp_nr((T)1 + b1 * sq + b2 * rs);
    pot += (g + ((T)(7.0 / 6.0) * g * b1) * sq + ((T)(4.0 / 3.0) * g * b2 * rs)) * (inv * inv);
    if (want_e) eps += g * inv;
  }
}

// A thread's sum of one energy term over its points (the 2 rl points of a row
// pair's butterfly, up to 32, rarely of a second one), in double across threads.
// FP32: the running sum and the sum of its rounding errors, and products of two
// fields with theirs, so that n points add an error of n^2 2^-49 at most where
// 24-bit sums had n 2^-24 (measured: 1e-9 of the total); doubles would take the
// FP64 pipe 12 operations a point.
template <typename T> struct ESum;
template <> struct ESum<double> {
  double s;
  __device__ __forceinline__ void init() { s = 0.0; }
  __device__ __forceinline__ void add(double x) { s += x; }
  __device__ __forceinline__ void add_product(double x, double y) { s += x * y; }
  __device__ __forceinline__ void add(const ESum& o) { s += o.s; }
  __device__ __forceinline__ double value() const { return s; }
};
template <> struct ESum<float> {
  float s, c;
  __device__ __forceinline__ void init() { s = c = 0.0f; }
  __device__ __forceinline__ void add(float x) {
    const float t = __fadd_rn(s, x), z = __fsub_rn(t, s);
    c += __fsub_rn(s, __fsub_rn(t, z)) + __fsub_rn(x, z);
    s = t;
  }
  __device__ __forceinline__ void add_product(float x, float y) {
    const float p = __fmul_rn(x, y);
    add(p);
    c += __fmaf_rn(x, y, -p);
  }
  __device__ __forceinline__ void add(const ESum& o) {
    add(o.s);
    c += o.c;
  }
  __device__ __forceinline__ double value() const { return (double)s + (double)c; }
};

// the pointwise terms at rho <= 1e-30 (the reference's clamps), out of line
template <typename T>
__device__ __noinline__ void point_tiny(const RowsInv& a, T rho, T w, T kc, T vh, T vl, bool want_e, T* pot_out,
                                        ESum<T>* es) {
  const EvalDesc& ev = a.ev;
  T pot = (T)0;
  const T kz = (T)kZero;
  if (ev.tf) {
    pot += sc<T>(a.tf_v) * cbrt(rho * rho);
    if (want_e) {
      T r5 = rho * rho;
      r5 = r5 * rho; r5 = r5 * rho; r5 = r5 * rho;
      es[0].add(cbrt(r5) * sc<T>(a.tf_e));
    }
  }
  if (ev.vw) {
    const T v = (T)0.5 * w * (rho > (T)0 ? (T)1 / fmax(sqrt(rho), kz) : (T)1e15);
    pot += v * sc<T>(a.vw_y);
    if (want_e && rho > (T)0) es[1].add(rho * v * sc<T>(a.vw_y));
  }
  if (ev.wt) {
    const T rb = a.b56 ? sqrt(kz) * cbrt(kz) / kz : pow(kz, sc<T>(a.wt_beta)) / kz;
    const T v = sc<T>(a.two_alpha) * rb * kc;
    pot += v;
    if (want_e) es[2].add(v * rho * sc<T>(a.inv_two_alpha));
  }
  if (ev.xc) {
    T rc = cbrt(rho);
    if (rc < kz) rc = kz;
    const T inv = (T)1 / rc;
    T vx, eps;
    Roots<T> r;
    r.c = rc;
    r.z3 = inv;
    r.z2 = (T)0;
    r.y = sqrt(inv);
    pz_lda<T>(r, eps, vx, want_e);
    pot += vx;
    if (want_e) es[3].add(eps * rho);
  }
  if (ev.hartree) {
    pot += vh;
    if (want_e) es[4].add_product((T)0.5 * vh, rho);
  }
  if (ev.pp) {
    pot += vl;
    if (want_e) es[5].add_product(vl, rho);
  }
  *pot_out = pot;
}

// potential at one point from its density and convolution results; energy
// densities added to es
template <typename T, bool WANT_E>
__device__ __forceinline__ T point(const RowsInv& a, T rho, T w, T kc, T vh, T vl, ESum<T>* es) {
  const EvalDesc& ev = a.ev;
  if (!(rho > (T)kZero)) {
    T p;
    ESum<T> e6[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) e6[q].init();
    point_tiny<T>(a, rho, w, kc, vh, vl, WANT_E, &p, e6);
    if constexpr (WANT_E) {
#pragma unroll
      for (int q = 0; q < 6; ++q) es[q].add(e6[q]);
    }
    return p;
  }
  const Roots<T> r = roots(rho);
  T pot = (T)0;
  if (ev.tf) {
    const T r23 = rho * r.z3;                           // rho^(2/3)
    if constexpr (sizeof(T) == 4) pot = fma(sc<T>(a.tf_v), r23, sc<T>(a.tf_vl) * r23);
    else pot += sc<T>(a.tf_v) * r23;
    if (WANT_E) es[0].add(rho * r23 * sc<T>(a.tf_e));
  }
  if (ev.vw) {
    const T v = w * r.z2 * sc<T>(a.half_vw);
    pot += v;
    if (WANT_E) es[1].add(rho * v);
  }
  if (ev.wt) {
    // rho^(beta - 1)
    const T rb = a.b56 ? (sizeof(T) == 8 ? r.y : r.c * r.z2) : pow_general<T>(rho, sc<T>(a.wt_beta)) / rho;
    const T v = sc<T>(a.two_alpha) * rb * kc;
    pot += v;
    if (WANT_E) es[2].add(v * rho * sc<T>(a.inv_two_alpha));
  }
  if (ev.xc) {
    T eps, vx;
    pz_lda<T>(r, eps, vx, WANT_E);
    pot += vx;
    if (WANT_E) es[3].add(eps * rho);
  }
  if (ev.hartree) {
    pot += vh;
    if (WANT_E) es[4].add_product((T)0.5 * vh, rho);
  }
  if (ev.pp) {
    pot += vl;
    if (WANT_E) es[5].add_product(vl, rho);
  }
  return pot;
}

// the WGC term at one point from its six fields (FP64: and the powers A, B of
// the forward rows): potential; energy density added to es[2]
template <typename T, bool WANT_E>
__device__ __forceinline__ T wgc_point(const RowsInv& a, T rho, T A, T B, T X0, T X1, T X2, T Y0, T Y1, T Y2,
                                       ESum<T>* es) {
  const T rc = rho > (T)kZero ? rho : (T)kZero;
  const T inv0 = sc<T>(a.w_inv0), u = (rc - sc<T>(a.w_rho0)) * inv0;
  if constexpr (sizeof(T) == 4) A = pow_of(rc, sc<T>(a.w_a));
  const T ir = rcp_nr(rc);
  const T sx = X0 + u * X1 + u * u * X2, tx = X1 + (T)2 * u * X2;
  if (WANT_E) es[2].add(A * sx);
  T v = A * (sc<T>(a.w_a) * ir * sx + inv0 * tx);
  if (a.two) {
    if constexpr (sizeof(T) == 4) B = pow_of(rc, sc<T>(a.w_b));
    const T sy = Y0 + u * Y1 + u * u * Y2, ty = Y1 + (T)2 * u * Y2;
    v += B * (sc<T>(a.w_b) * ir * sy + inv0 * ty);
  } else {
    v *= (T)2;
  }
  return v;
}

// inputs i + t nb of a row pair's inverse transform from its two half spectra
template <int R, typename T>
__device__ __forceinline__ void inverse_row_inputs(cpx<T>* u, const cpx<T>* pa, int ld2, bool ok0, bool ok1, int i,
                                                   int nb, int n) {
#pragma unroll
  for (int t = 0; t < R; ++t) {
    const int j = i + t * nb;
    // j > n/2, and j in {0, n/2}, whose imaginary parts do not count
    bool up, edge;
    if constexpr (R % 2 == 0) {
      up = t > R / 2 || (t == R / 2 && i > 0);
      edge = t % (R / 2) == 0 && i == 0;
    } else {
      up = 2 * j > n;
      edge = j == 0 || 2 * j == n;
    }
    const int k = up ? n - j : j;
    cpx<T> va = {(T)0, (T)0}, vb = {(T)0, (T)0};
    if (ok0) va = pa[k];
    if (ok1) vb = pa[ld2 + k];
    if (edge) { va.y = (T)0; vb.y = (T)0; }
    u[t] = up ? cpx<T>{va.x + vb.y, vb.x - va.y} : cpx<T>{va.x - vb.y, va.y + vb.x};
  }
}

enum { RI_STORE = 0, RI_EVAL = 1, RI_EVAL_E = 2 };

template <typename T, int MODE, typename AX>
__global__ void __launch_bounds__(RowCta<T>::NT, (RowCta<T, AX>::MINB)) k_rb_rows_inv(const __grid_constant__ RowsInv a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const AX ax(a.ax);
  const int n = ax.n(), lp = a.lp, ls = line_pitch<T>(n), nl = a.nf * lp;
  cpx<T>* A = reinterpret_cast<cpx<T>*>(smem_raw);
  cpx<T>* B = A + nl * ls;                               // used by three or more stages
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int base = blockIdx.x * 2 * lp;
  const cpx<T>* tw = reinterpret_cast<const cpx<T>*>(a.tw);
  // first stage: line element j of a row pair is X_a[j] + i X_b[j] for
  // j <= n/2 and the conjugates' combination above
  ax.first([&](auto rc) {
    constexpr int R = decltype(rc)::R;
    const int nb = ax.nbf();
    for (int t0 = tid; t0 < nl * nb; t0 += nthr) {
      const int line = ax.div_nbf(t0), i = t0 - line * nb;
      const int f = line / lp, l = line - f * lp;
      const int ra = base + 2 * l;
      cpx<T> u[R];
      const cpx<T>* pa = reinterpret_cast<const cpx<T>*>(a.in[f]) + (int64_t)ra * a.ld2;
      const bool ok0 = ra < a.nrows, ok1 = ra + 1 < a.nrows;
      inverse_row_inputs<R, T>(u, pa, a.ld2, ok0, ok1, i, nb, n);
      stage_first<1, T>(rc, u, tw, n);
      cpx<T>* dst = A + line * ls;
#pragma unroll
      for (int t = 0; t < R; ++t) dst[sidx<T>(i * R + t)] = u[t];
    }
  });
  __syncthreads();
  cpx<T>* cur = A;
  cpx<T>* oth = B;
  ax.middle([&](auto rc, auto nb, auto p, auto div_nb, auto div_p) {
    constexpr int R = decltype(rc)::R;
    for (int t0 = tid; t0 < nl * nb; t0 += nthr) {
      const int line = div_nb(t0), i = t0 - line * nb;
      const int k = i - p * div_p(i);
      cpx<T> u[R];
      load_stage<1, T>(rc, u, cur + line * ls, tw, i, k, nb, p, n, sidx<T>);
      cpx<T>* dst = oth + line * ls;
      const int j0 = (i - k) * R + k;
#pragma unroll
      for (int t = 0; t < R; ++t) dst[sidx<T>(j0 + t * p)] = u[t];
    }
    __syncthreads();
    cpx<T>* x = cur;
    cur = oth;
    oth = x;
  });
  // last stage: a thread transforms butterfly i of every field of a row pair
  // in place (its own elements), so the points i + t nb are complete in it
  const int nb = ax.nbl(), rl = ax.rl();
  ESum<T> es[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) es[c].init();
  for (int t0 = tid; t0 < lp * nb; t0 += nthr) {
    const int l = ax.div_nbl(t0), i = t0 - l * nb;
    const int ra = base + 2 * l;
    if (ra >= a.nrows) continue;
    const bool ok1 = ra + 1 < a.nrows;
    if (ax.nst() > 1) {
      ax.last([&](auto rc) {
        constexpr int R = decltype(rc)::R;
        for (int f = 0; f < a.nf; ++f) {
          cpx<T>* src = cur + (f * lp + l) * ls;
          cpx<T> u[R];
          load_stage<1, T>(rc, u, src, tw, i, i, nb, nb, n, sidx<T>);
#pragma unroll
          for (int t = 0; t < R; ++t) src[sidx<T>(i + t * nb)] = u[t];
        }
      });
    }
    const cpx<T>* fld = cur + l * ls;
    if constexpr (MODE == RI_STORE) {
      T* out = reinterpret_cast<T*>(a.out);
      const T scl = sc<T>(a.scale);
      for (int f = 0; f < a.nf; ++f) {
        T* o = out + f * a.ostride + (int64_t)ra * n + i;
        for (int t = 0; t < rl; ++t) {
          const cpx<T> z = fld[f * lp * ls + sidx<T>(i + t * nb)];
          o[t * nb] = z.x * scl;
          if (ok1) o[t * nb + n] = z.y * scl;
        }
      }
    } else {
      const EvalDesc& ev = a.ev;
      const int64_t g0 = (int64_t)ra * n + i;
      const T* rp = reinterpret_cast<const T*>(a.rho) + g0;
      const T* vp = reinterpret_cast<const T*>(a.vloc) + g0;
      T* pp = reinterpret_cast<T*>(a.pot) + g0;
      const int fs = lp * ls;
      // density and v_loc of the next point pair are in flight while this
      // one's terms are formed
      T r0 = __ldg(rp), r1 = ok1 ? __ldg(rp + n) : (T)1, v0 = (T)0, v1 = (T)0;
      if (ev.pp) {
        v0 = __ldg(vp);
        if (ok1) v1 = __ldg(vp + n);
      }
#pragma unroll 1
      for (int t = 0; t < rl; ++t) {
        const int j = t * nb;
        const int o = sidx<T>(i + j);
        T nr0 = (T)1, nr1 = (T)1, nv0 = (T)0, nv1 = (T)0;
        if (t + 1 < rl) {
          nr0 = __ldg(rp + j + nb);
          if (ok1) nr1 = __ldg(rp + j + nb + n);
          if (ev.pp) {
            nv0 = __ldg(vp + j + nb);
            if (ok1) nv1 = __ldg(vp + j + nb + n);
          }
        }
        cpx<T> w = {(T)0, (T)0}, kc = {(T)0, (T)0}, vh = {(T)0, (T)0};
        if (ev.vw) w = fld[ev.slot_vw * fs + o];
        if (ev.wt) kc = fld[ev.slot_wt * fs + o];
        if (ev.hartree) vh = fld[ev.slot_h * fs + o];
        if constexpr (sizeof(T) == 8) {
          if (ev.cout) {
            // copy of the convolution results (delta-evaluation reference)
            T* c = reinterpret_cast<T*>(ev.cout) + g0 + j;
            if (ev.vw) { c[ev.slot_vw * ev.cstride] = w.x; if (ok1) c[ev.slot_vw * ev.cstride + n] = w.y; }
            if (ev.wt) { c[ev.slot_wt * ev.cstride] = kc.x; if (ok1) c[ev.slot_wt * ev.cstride + n] = kc.y; }
            if (ev.hartree) { c[ev.slot_h * ev.cstride] = vh.x; if (ok1) c[ev.slot_h * ev.cstride + n] = vh.y; }
          }
        }
        constexpr bool E = MODE == RI_EVAL_E;
        T p0 = (T)0, p1 = (T)0;
        if (a.base) {
          p0 = point<T, E>(a, r0, w.x, kc.x, vh.x, v0, es);
          if (ok1) p1 = point<T, E>(a, r1, w.y, kc.y, vh.y, v1, es);
        }
        if (a.add) {
          p0 += pp[j];
          if (ok1) p1 += pp[j + n];
        }
        if (a.wgc) {
          cpx<T> x[3], y[3];
          const int ys = a.two ? 3 : 0;
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            x[q] = fld[(a.wslot + q) * fs + o];
            y[q] = fld[(a.wslot + ys + q) * fs + o];
          }
          T A0 = (T)0, B0 = (T)0, A1 = (T)0, B1 = (T)0;
          if constexpr (sizeof(T) == 8) {
            const T *qa = reinterpret_cast<const T*>(a.pa) + g0 + j, *qb = reinterpret_cast<const T*>(a.pb) + g0 + j;
            A0 = qa[0]; B0 = qb[0];
            if (ok1) { A1 = qa[n]; B1 = qb[n]; }
            if (a.vstore) {
#pragma unroll
              for (int q = 0; q < 3; ++q) {
                T* c = reinterpret_cast<T*>(a.wstore[q]) + g0 + j;
                c[0] = x[q].x;
                if (ok1) c[n] = x[q].y;
                if (a.two) {
                  c = reinterpret_cast<T*>(a.wstore[3 + q]) + g0 + j;
                  c[0] = y[q].x;
                  if (ok1) c[n] = y[q].y;
                }
              }
            }
          }
          const T w0 = wgc_point<T, E>(a, r0, A0, B0, x[0].x, x[1].x, x[2].x, y[0].x, y[1].x, y[2].x, es);
          T w1 = (T)0;
          if (ok1) w1 = wgc_point<T, E>(a, r1, A1, B1, x[0].y, x[1].y, x[2].y, y[0].y, y[1].y, y[2].y, es);
          if constexpr (sizeof(T) == 8) {
            if (a.vstore) {
              T* c = reinterpret_cast<T*>(a.vstore) + g0 + j;
              c[0] = w0;
              if (ok1) c[n] = w1;
            }
          }
          p0 += w0;
          p1 += w1;
        }
        pp[j] = p0;
        if (ok1) pp[j + n] = p1;
        r0 = nr0;
        r1 = nr1;
        v0 = nv0;
        v1 = nv1;
      }
    }
  }
  if constexpr (MODE != RI_EVAL_E) return;
  __shared__ double red[8][6];
  const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const double v = warp_sum(es[c].value());
    if (lane == 0) red[warp][c] = v;
  }
  __syncthreads();
  if (tid < 6) {
    KSum t;
    t.init();
    for (int w = 0; w < (nthr + 31) / 32; ++w) t.add(red[w][tid]);
    a.partials[(int64_t)blockIdx.x * GB_NE + tid] = t.value();
  }
}

// ---- columns -------------------------------------------------------------------
struct Cols {
  void* data[GB_RB_FIELDS];
  int64_t stride, ostride;
  unsigned ncol;          // columns over all outer indices (pitch ld2 each)
  int n2h;
  FastDiv dld;
  RbAxis ax, inv;         // the axis; the same radices in reverse order (CONV)
  const void* tw;
  Sc scale;
  Sc coef[GB_MAX_FIELDS];
  Sc bg[9];
  int type[GB_MAX_FIELDS];
  const void* arr[GB_MAX_FIELDS];
  int n0, n1, n2, full;
  const void* K;          // WGC: K0, K1, Kq, Kx (API layout), kstride values each
  int64_t kstride;
  const void* src;        // inverse: read one field from here instead
  int64_t sstride, sostride;
};

template <typename T> struct ColTile { static constexpr int TB = 128 / (2 * (int)sizeof(T)); };

// reciprocal-space kernel along one axis-0 column (i1, k2)
template <typename T> struct ColKernel {
  T b0, b1, b2;           // axis-0 reciprocal vector
  T ux, uy, uz;           // m1 b1 + m2 b2
  T px, py, pz;           // the same at the conjugate partner (-i1, -k2)
  int sym;                // 0: no partner average, 1: at i0 = n0/2, 2: at every i0
  int n0;

  __device__ __forceinline__ void init(const Cols& a, int i1, int k2) {
    n0 = a.n0;
    const bool ny1 = (a.n1 & 1) == 0 && 2 * i1 == a.n1, ny2 = (a.n2 & 1) == 0 && 2 * k2 == a.n2;
    const T m1 = (T)gbk::ffreq(i1, a.n1), m2 = (T)(a.full ? gbk::ffreq(k2, a.n2) : k2);
    const T q1 = ny1 ? m1 : -m1, q2 = a.full ? (ny2 ? m2 : -m2) : m2;
    b0 = sc<T>(a.bg[0]); b1 = sc<T>(a.bg[1]); b2 = sc<T>(a.bg[2]);
    ux = m1 * sc<T>(a.bg[3]) + m2 * sc<T>(a.bg[6]);
    uy = m1 * sc<T>(a.bg[4]) + m2 * sc<T>(a.bg[7]);
    uz = m1 * sc<T>(a.bg[5]) + m2 * sc<T>(a.bg[8]);
    px = q1 * sc<T>(a.bg[3]) + q2 * sc<T>(a.bg[6]);
    py = q1 * sc<T>(a.bg[4]) + q2 * sc<T>(a.bg[7]);
    pz = q1 * sc<T>(a.bg[5]) + q2 * sc<T>(a.bg[8]);
    const bool plane = a.full || k2 == 0 || ny2;
    sym = plane ? ((ny1 || (a.full && ny2)) ? 2 : 1) : 0;
  }
  static __device__ __forceinline__ T gg(T x, T y, T z) { return x * x + y * y + z * z; }
  static __device__ __forceinline__ T val(bool hart, T g) {
    if (!hart) return g;
    return g > (T)0 ? (T)(4.0 * 3.14159265358979323846) * rcp_nr(g) : (T)0;
  }
  // K at axis-0 index j, averaged with the conjugate partner's on Nyquist planes
  __device__ __forceinline__ T at(bool hart, int j) const {
    const T m0 = (T)gbk::ffreq(j, n0);
    T k = val(hart, gg(m0 * b0 + ux, m0 * b1 + uy, m0 * b2 + uz));
    const bool ny0 = 2 * j == n0;
    if (sym == 2 || (sym == 1 && ny0)) {
      const T q0 = ny0 ? m0 : -m0;
      k = (k + val(hart, gg(q0 * b0 + px, q0 * b1 + py, q0 * b2 + pz))) * (T)0.5;
    }
    return k;
  }
};

// ---- LWT --------------------------------------------------------------------------
// Linear interpolation between the knots k_i of the kernel: a point with k_F in
// interval e has weight t at the interval's right knot and 1 - t at its left one.
// The passes take a batch of knots and run through them with the shared memory of
// one: all knots of a batch at once left four row CTAs (one column CTA) on an SM
// (360^3 FP32, per knot: inverse rows 363 -> 292 us, forward rows 180 -> 131 us,
// forward columns 274 -> 128 us).
struct LwtRows {
  const void* in[GB_RB_FIELDS];
  void* out[GB_RB_FIELDS];
  const void *kf, *ra;
  void *out1, *out3;
  int first, m, below;
  int nrows, n2h, ld2, lp;
  RbAxis ax;
  FastDiv dnh;
  const void* tw;
  Sc half;
  Sc lo[GB_LWT_BATCH + 1], hi[GB_LWT_BATCH + 1], inv[GB_LWT_BATCH + 1];
  Sc kl, kl_e, inv_kl;
};

// weights of one knot of the batch, without branches (the loads of k_F around them
// stay in flight together)
template <typename T> struct LwtWeight {
  T lo0, hi0, inv0, lo1, hi1, inv1, kl, kl_e, inv_kl;
  __device__ __forceinline__ LwtWeight(const LwtRows& a, int q) {
    lo0 = sc<T>(a.lo[q]); hi0 = sc<T>(a.hi[q]); inv0 = sc<T>(a.inv[q]);
    lo1 = sc<T>(a.lo[q + 1]); hi1 = sc<T>(a.hi[q + 1]); inv1 = sc<T>(a.inv[q + 1]);
    kl = sc<T>(a.kl); inv_kl = sc<T>(a.inv_kl);
    kl_e = q == 0 && a.below ? sc<T>(a.kl_e) : -(T)HUGE_VAL;
  }
  // low: count the points below the first knot
  __device__ __forceinline__ T at(T kf, bool low) const {
    T w = low && kf < kl_e ? (kf - kl) * inv_kl : (T)0;
    w = kf > lo1 && kf < hi1 ? (T)1 - (kf - lo1) * inv1 : w;
    return kf > lo0 && kf < hi0 ? (kf - lo0) * inv0 : w;
  }
};

// out1 (out3) (+)= sum over the batch of weight x inverse rows of the knot's field
// (its derivative field).  The transformed fields never reach memory; a point has
// its interval's two knots only, so the sums are added in memory where the weight is
// not zero (from the batch's second knot on, in L2).
template <typename T, typename AX>
__global__ void __launch_bounds__(RowCta<T>::NT, (RowCta<T, AX>::MINB)) k_rb_lwt_rows_inv(const __grid_constant__ LwtRows a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const AX ax(a.ax);
  const int n = ax.n(), lp = a.lp, ls = line_pitch<T>(n), nk = a.out3 ? 2 : 1, nl = nk * lp;
  cpx<T>* A = reinterpret_cast<cpx<T>*>(smem_raw);
  cpx<T>* B = A + nl * ls;                               // three or more stages
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int base = blockIdx.x * 2 * lp;
  const cpx<T>* tw = reinterpret_cast<const cpx<T>*>(a.tw);
  const int nb = ax.nbl(), rl = ax.rl();
#pragma unroll 1
  for (int q = 0; q < a.m; ++q) {
    const LwtWeight<T> wq(a, q);
    ax.first([&](auto rc) {
      constexpr int R = decltype(rc)::R;
      const int nbf = ax.nbf();
      for (int t0 = tid; t0 < nl * nbf; t0 += nthr) {
        const int line = ax.div_nbf(t0), i = t0 - line * nbf;
        const int f = line >= lp, l = line - f * lp;
        const int ra = base + 2 * l;
        cpx<T> u[R];
        const cpx<T>* pa = reinterpret_cast<const cpx<T>*>(a.in[q + f * a.m]) + (int64_t)ra * a.ld2;
        inverse_row_inputs<R, T>(u, pa, a.ld2, ra < a.nrows, ra + 1 < a.nrows, i, nbf, n);
        stage_first<1, T>(rc, u, tw, n);
        cpx<T>* dst = A + line * ls;
#pragma unroll
        for (int t = 0; t < R; ++t) dst[sidx<T>(i * R + t)] = u[t];
      }
    });
    __syncthreads();
    cpx<T>* cur = A;
    cpx<T>* oth = B;
    ax.middle([&](auto rc, auto nbm, auto p, auto div_nb, auto div_p) {
      constexpr int R = decltype(rc)::R;
      for (int t0 = tid; t0 < nl * nbm; t0 += nthr) {
        const int line = div_nb(t0), i = t0 - line * nbm;
        const int k = i - p * div_p(i);
        cpx<T> u[R];
        load_stage<1, T>(rc, u, cur + line * ls, tw, i, k, nbm, p, n, sidx<T>);
        cpx<T>* dst = oth + line * ls;
        const int j0 = (i - k) * R + k;
#pragma unroll
        for (int t = 0; t < R; ++t) dst[sidx<T>(j0 + t * p)] = u[t];
      }
      __syncthreads();
      cpx<T>* x = cur;
      cur = oth;
      oth = x;
    });
    for (int t0 = tid; t0 < lp * nb; t0 += nthr) {
      const int l = ax.div_nbl(t0), i = t0 - l * nb;
      const int ra = base + 2 * l;
      if (ra >= a.nrows) continue;
      const bool ok1 = ra + 1 < a.nrows;
      const T* kp = reinterpret_cast<const T*>(a.kf) + (int64_t)ra * n + i;
      const int second = ok1 ? n : 0;
      const bool store = a.first && q == 0;
      // C points t, t + 1, .. of field f: every load before the first store
      auto add = [&](auto cc, int t, int f, auto&& z) {
        constexpr int C = decltype(cc)::value;
        T* o = reinterpret_cast<T*>(f ? a.out3 : a.out1) + (int64_t)ra * n + i;
        T w0[C], w1[C], s0[C], s1[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
          // below the knots there is no derivative term
          w0[c] = wq.at(__ldg(kp + (t + c) * nb), f == 0);
          w1[c] = wq.at(__ldg(kp + (t + c) * nb + second), f == 0);
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
          s0[c] = !store && w0[c] != (T)0 ? o[(t + c) * nb] : (T)0;
          s1[c] = !store && w1[c] != (T)0 ? o[(t + c) * nb + second] : (T)0;
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const cpx<T> v = z(t + c);
          if (store || w0[c] != (T)0) o[(t + c) * nb] = s0[c] + w0[c] * v.x;
          if (ok1 && (store || w1[c] != (T)0)) o[(t + c) * nb + n] = s1[c] + w1[c] * v.y;
        }
      };
      if (ax.nst() > 1) {
        ax.last([&](auto rc) {
          constexpr int R = decltype(rc)::R;
          // 4 or so: 360^3 FP32, three knots 877 us, 904 with 2 (registers for 7 CTAs;
          // without spills, at 5 CTAs, 1026)
          constexpr int C = R % 4 == 0 ? 4 : R % 3 == 0 ? 3 : R % 5 == 0 ? 5 : R % 7 == 0 ? 7 : 2;
          for (int f = 0; f < nk; ++f) {
            cpx<T> u[R];
            load_stage<1, T>(rc, u, cur + (f * lp + l) * ls, tw, i, i, nb, nb, n, sidx<T>);
#pragma unroll
            for (int t = 0; t < R; t += C) add(std::integral_constant<int, C>{}, t, f, [&](int k) { return u[k]; });
          }
        });
      } else {
        for (int f = 0; f < nk; ++f)
          for (int t = 0; t < rl; ++t)
            add(std::integral_constant<int, 1>{}, t, f,
                [&](int k) { return cur[(f * lp + l) * ls + sidx<T>(i + k * nb)]; });
      }
    }
    __syncthreads();                                     // the next knot overwrites the buffers
  }
}

// spectra along axis 2 of weight x ra for every knot of the batch
template <typename T, typename AX>
__global__ void __launch_bounds__(RowCta<T>::NT, (RowCta<T, AX>::MINB)) k_rb_lwt_rows_fwd(const __grid_constant__ LwtRows a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const AX ax(a.ax);
  const int n = ax.n(), lp = a.lp, ls = line_pitch<T>(n);
  cpx<T>* A = reinterpret_cast<cpx<T>*>(smem_raw);
  cpx<T>* B = ax.nst() > 2 ? A + lp * ls : A;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int base = blockIdx.x * 2 * lp;
  const cpx<T>* tw = reinterpret_cast<const cpx<T>*>(a.tw);
  const T* kf = reinterpret_cast<const T*>(a.kf);
  const T* fac = reinterpret_cast<const T*>(a.ra);
  const int nh = AX::kFixed ? n / 2 + 1 : a.n2h;
#pragma unroll 1
  for (int q = 0; q < a.m; ++q) {
    const LwtWeight<T> wq(a, q);
    ax.first([&](auto rc) {
      constexpr int R = decltype(rc)::R;
      const int nb = ax.nbf();
      for (int t0 = tid; t0 < lp * nb; t0 += nthr) {
        const int l = ax.div_nbf(t0), i = t0 - l * nb;
        const int ra = base + 2 * l;
        const bool ok0 = ra < a.nrows, ok1 = ra + 1 < a.nrows;
        const int64_t off = (int64_t)ra * n + i;
        cpx<T> u[R];
#pragma unroll
        for (int t = 0; t < R; ++t) u[t] = cpx<T>{ok0 ? __ldg(kf + off + t * nb) : (T)0, ok1 ? __ldg(kf + off + n + t * nb) : (T)0};
#pragma unroll
        for (int t = 0; t < R; ++t) {
          const T w0 = ok0 ? wq.at(u[t].x, true) : (T)0, w1 = ok1 ? wq.at(u[t].y, true) : (T)0;
          u[t].x = w0 != (T)0 ? w0 * __ldg(fac + off + t * nb) : (T)0;
          u[t].y = w1 != (T)0 ? w1 * __ldg(fac + off + n + t * nb) : (T)0;
        }
        stage_first<-1, T>(rc, u, tw, n);
        cpx<T>* dst = B + l * ls;
#pragma unroll
        for (int t = 0; t < R; ++t) dst[sidx<T>(i * R + t)] = u[t];
      }
    });
    const cpx<T>* res = lines<-1, false, T>(A, B, ls, lp, ax, tw);
    const T half = sc<T>(a.half);
    cpx<T>* o = reinterpret_cast<cpx<T>*>(a.out[q]);
    for (int idx = tid; idx < lp * nh; idx += nthr) {
      const int l = AX::kFixed ? idx / nh : (int)a.dnh.div(idx), k = idx - l * nh;
      const int ra = base + 2 * l;
      if (ra >= a.nrows) continue;
      const cpx<T> Z = res[l * ls + sidx<T>(k)];
      const cpx<T> Zc = res[l * ls + sidx<T>(k == 0 ? 0 : n - k)];
      cpx<T>* w = o + (int64_t)ra * a.ld2 + k;
      w[0] = c_scale(cpx<T>{Z.x + Zc.x, Z.y - Zc.y}, half);
      if (ra + 1 < a.nrows) w[a.ld2] = c_scale(cpx<T>{Z.y + Zc.y, Zc.x - Z.x}, half);
    }
    __syncthreads();                                     // the next knot overwrites the buffers
  }
}

// Columns along axis 0.  Inverse: field f = ifft(K_f S), the product formed as the
// pass loads S (the fields of one column tile are neighbouring CTAs: the tile
// comes from HBM once).  Forward: out (+)= sum_f K_f fft(in_f), added through L2 as
// each field's last stage ends.
struct LwtCols {
  const void* in[GB_RB_FIELDS];
  void* out[GB_RB_FIELDS];
  const void* K[GB_RB_FIELDS];
  int64_t stride, ostride, kst;
  unsigned ncol;
  int n2h, nf, first;
  FastDiv dld;
  RbAxis ax;
  const void* tw;
};

// columns of a tile.  The sums read and write memory field after field: half the
// tile, and twice the CTAs on an SM, for three-stage lines (360^3 FP32, three
// fields: 466 -> 385 us; the inverse pass 549 -> 573 us, so it keeps the whole one)
template <typename T, int DIR, typename AX> constexpr int lwt_tb() {
  if constexpr (sizeof(T) == 4 && AX::kFixed && DIR < 0) return AX::nst() > 2 ? 8 : ColTile<T>::TB;
  else return ColTile<T>::TB;
}

template <typename T, int DIR, typename AX>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 400 : 256) k_rb_lwt(const __grid_constant__ LwtCols a) {
  constexpr int TB = lwt_tb<T, DIR, AX>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const AX ax(a.ax);
  const int n = ax.n();
  cpx<T>* A = reinterpret_cast<cpx<T>*>(smem_raw);
  const int c = threadIdx.x % TB, i0 = threadIdx.x / TB, ni = blockDim.x / TB;
  const unsigned tile = DIR > 0 ? blockIdx.x / a.nf : blockIdx.x;
  const unsigned col = tile * TB + c;
  const int outer = a.dld.div(col), k2 = col - outer * a.dld.d;
  const bool ok = col < a.ncol && k2 < a.n2h;
  const int64_t off = outer * a.ostride + k2, koff = (int64_t)outer * a.n2h + k2;
  const cpx<T>* tw = reinterpret_cast<const cpx<T>*>(a.tw);
  const int64_t st = a.stride, kst = a.kst;
  auto sx = [&](int j) { return j * TB + c; };
  const int f_lo = DIR > 0 ? blockIdx.x - tile * a.nf : 0, f_hi = DIR > 0 ? f_lo + 1 : a.nf;
#pragma unroll 1
  for (int f = f_lo; f < f_hi; ++f) {
    const cpx<T>* g = reinterpret_cast<const cpx<T>*>(a.in[DIR > 0 ? 0 : f]) + off;
    const T* K = reinterpret_cast<const T*>(a.K[f]) + koff;
    ax.first([&](auto rc) {
      constexpr int R = decltype(rc)::R;
      const int nb = ax.nbf();
      for (int i = i0; i < nb; i += ni) {
        cpx<T> u[R];
#pragma unroll
        for (int t = 0; t < R; ++t) {
          const int j = i + t * nb;
          u[t] = ok ? g[j * st] : cpx<T>{(T)0, (T)0};
          if (DIR > 0) u[t] = c_scale(u[t], ok ? __ldg(K + j * kst) : (T)0);
        }
        stage_first<DIR, T>(rc, u, tw, n);
#pragma unroll
        for (int t = 0; t < R; ++t) A[sx(i * R + t)] = u[t];
      }
    });
    __syncthreads();
    cpx<T>* cur = A;
    cpx<T>* oth = A + n * TB;
    ax.middle([&](auto rc, auto nb, auto p, auto, auto div_p) {
      constexpr int R = decltype(rc)::R;
      for (int i = i0; i < nb; i += ni) {
        const int k = i - p * div_p(i);
        cpx<T> u[R];
        load_stage<DIR, T>(rc, u, cur, tw, i, k, nb, p, n, sx);
        const int j0 = (i - k) * R + k;
#pragma unroll
        for (int t = 0; t < R; ++t) oth[sx(j0 + t * p)] = u[t];
      }
      __syncthreads();
      cpx<T>* y = cur;
      cur = oth;
      oth = y;
    });
    cpx<T>* o = reinterpret_cast<cpx<T>*>(a.out[DIR > 0 ? f : 0]) + off;
    ax.last([&](auto rc) {
      constexpr int R = decltype(rc)::R;
      const int nb = ax.nbl();
      for (int i = i0; i < nb; i += ni) {
        cpx<T> u[R];
        load_stage<DIR, T>(rc, u, cur, tw, i, i, nb, nb, n, sx);
        if (!ok) continue;
#pragma unroll
        for (int t = 0; t < R; ++t) {
          const int j = i + t * nb;
          if (DIR < 0) {
            u[t] = c_scale(u[t], __ldg(K + j * kst));
            if (f > 0 || !a.first) {
              const cpx<T> s = o[j * st];
              u[t] = cpx<T>{s.x + u[t].x, s.y + u[t].y};
            }
          }
          o[j * st] = u[t];
        }
      }
    });
    if (DIR < 0) __syncthreads();                        // the next field overwrites the buffers
  }
}

template <typename T, int DIR, bool CONV, typename AX, typename AXI>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 400 : 256) k_rb_cols(const __grid_constant__ Cols a) {
  constexpr int TB = ColTile<T>::TB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const AX ax(a.ax);
  const AXI axi(a.inv);
  const int n = ax.n(), nst = ax.nst();
  cpx<T>* A = reinterpret_cast<cpx<T>*>(smem_raw);
  cpx<T>* B = A + n * TB;
  const int c = threadIdx.x % TB, i0 = threadIdx.x / TB, ni = blockDim.x / TB;
  const unsigned col = blockIdx.x * TB + c;
  const int outer = a.dld.div(col), k2 = col - outer * a.dld.d;
  const bool ok = col < a.ncol && k2 < a.n2h;
  const int f = blockIdx.y;
  cpx<T>* g = reinterpret_cast<cpx<T>*>(a.data[f]) + outer * a.ostride + k2;
  const cpx<T>* tw = reinterpret_cast<const cpx<T>*>(a.tw);
  const int64_t st = a.stride;
  const cpx<T>* gs = g;
  int64_t ss = st;
  if (DIR > 0 && !CONV && a.src) {
    gs = reinterpret_cast<const cpx<T>*>(a.src) + outer * a.sostride + k2;
    ss = a.sstride;
  }
  ColKernel<T> ker;
  int type = KER_NONE;
  T coef = (T)1;
  const T* karr = nullptr;
  if constexpr (CONV) {
    type = a.type[f];
    coef = sc<T>(a.coef[f]);
    if (type == KER_HARTREE || type == KER_G2) ker.init(a, outer, k2);
    // the API table layout [n0][n1][n2h]
    if (type == KER_ARRAY) karr = reinterpret_cast<const T*>(a.arr[f]) + (int64_t)outer * a.n2h + k2;
  }
  const int64_t kst = (int64_t)a.n1 * a.n2h;
  auto kmul = [&](int j, cpx<T> v) {
    T k = (T)1;
    if (type == KER_ARRAY) k = ok ? __ldg(karr + j * kst) : (T)0;
    else if (type != KER_NONE) k = ker.at(type == KER_HARTREE, j);
    return c_scale(v, k * coef);
  };
  const T scl = sc<T>(a.scale);
  constexpr int D0 = CONV ? -1 : DIR;
  if (nst == 1) {
    if (i0 > 0) return;
    ax.first([&](auto rc) {
      constexpr int R = decltype(rc)::R;
      cpx<T> u[R];
#pragma unroll
      for (int t = 0; t < R; ++t) u[t] = ok ? gs[t * ss] : cpx<T>{(T)0, (T)0};
      stage_first<D0, T>(rc, u, tw, n);
      if constexpr (CONV) {
#pragma unroll
        for (int t = 0; t < R; ++t) u[t] = kmul(t, u[t]);
        stage_first<1, T>(rc, u, tw, n);
      }
      if (ok) {
#pragma unroll
        for (int t = 0; t < R; ++t) g[t * st] = c_scale(u[t], scl);
      }
    });
    return;
  }
  auto sx = [&](int j) { return j * TB + c; };
  ax.first([&](auto rc) {
    constexpr int R = decltype(rc)::R;
    const int nb = ax.nbf();
    for (int i = i0; i < nb; i += ni) {
      cpx<T> u[R];
#pragma unroll
      for (int t = 0; t < R; ++t) u[t] = ok ? gs[(i + t * nb) * ss] : cpx<T>{(T)0, (T)0};
      stage_first<D0, T>(rc, u, tw, n);
#pragma unroll
      for (int t = 0; t < R; ++t) A[sx(i * R + t)] = u[t];
    }
  });
  __syncthreads();
  cpx<T>* cur = A;
  cpx<T>* oth = B;
  auto middle = [&](const auto& x, auto dir) {
    constexpr int D = decltype(dir)::value;
    x.middle([&](auto rc, auto nb, auto p, auto, auto div_p) {
      constexpr int R = decltype(rc)::R;
      for (int i = i0; i < nb; i += ni) {
        const int k = i - p * div_p(i);
        cpx<T> u[R];
        load_stage<D, T>(rc, u, cur, tw, i, k, nb, p, n, sx);
        const int j0 = (i - k) * R + k;
#pragma unroll
        for (int t = 0; t < R; ++t) oth[sx(j0 + t * p)] = u[t];
      }
      __syncthreads();
      cpx<T>* y = cur;
      cur = oth;
      oth = y;
    });
  };
  middle(ax, std::integral_constant<int, D0>{});
  ax.last([&](auto rc) {
    constexpr int R = decltype(rc)::R;
    const int nb = ax.nbl();
    for (int i = i0; i < nb; i += ni) {
      cpx<T> u[R];
      load_stage<D0, T>(rc, u, cur, tw, i, i, nb, nb, n, sx);
      if constexpr (CONV) {
#pragma unroll
        for (int t = 0; t < R; ++t) u[t] = kmul(i + t * nb, u[t]);
        stage_first<1, T>(rc, u, tw, n);
#pragma unroll
        for (int t = 0; t < R; ++t) oth[sx(i * R + t)] = u[t];
      } else if (ok) {
        if (scl != (T)1) {
#pragma unroll
          for (int t = 0; t < R; ++t) u[t] = c_scale(u[t], scl);
        }
#pragma unroll
        for (int t = 0; t < R; ++t) g[(i + t * nb) * st] = u[t];
      }
    }
  });
  if constexpr (CONV) {
    __syncthreads();
    cpx<T>* x = cur;
    cur = oth;
    oth = x;
    middle(axi, std::integral_constant<int, 1>{});
    axi.last([&](auto rc) {
      constexpr int R = decltype(rc)::R;
      const int nb = axi.nbl();
      for (int i = i0; i < nb; i += ni) {
        cpx<T> u[R];
        load_stage<1, T>(rc, u, cur, tw, i, i, nb, nb, n, sx);
        if (ok) {
#pragma unroll
          for (int t = 0; t < R; ++t) g[(i + t * nb) * st] = u[t];
        }
      }
    });
  }
}

// WGC term along axis 0: forward transforms of the three fields F0..F2 of one
// exponent (blockIdx.y), X0 = K0 F0 + K1/6 F1 + Kq F2, X1 = K1/6 F0 + Kx F1,
// X2 = Kq F0, and the inverse transforms, in one pass over the spectra.  The
// forward results stay in shared memory; each output is combined in the
// registers of its inverse's first stage.  blockDim.y = 3: the fields, then the
// outputs, side by side; 1: one after the other.  Three column buffers and,
// per side, one (two for three or more stages).
// FP32: one field's butterflies (128 to 256 threads) leave the SM waiting on the
// loads of each stage: 96^3, six fields, 42.7 us; side by side 24.4 us
// FP64: bound by the FP64 pipe either way.
template <typename T> constexpr int kWgcThreads = sizeof(T) == 4 ? 768 : 256;
template <typename T, typename AX, typename AXI>
__global__ void __launch_bounds__(kWgcThreads<T>) k_rb_wgc(const __grid_constant__ Cols a) {
  constexpr int TB = ColTile<T>::TB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const AX ax(a.ax);
  const AXI axi(a.inv);
  const int n = ax.n();
  cpx<T>* S = reinterpret_cast<cpx<T>*>(smem_raw);
  const int f0 = threadIdx.y, nf = blockDim.y;
  cpx<T>* D = S + (3 + f0) * n * TB;
  cpx<T>* E = D + nf * n * TB;                           // three or more stages
  const int c = threadIdx.x % TB, i0 = threadIdx.x / TB, ni = blockDim.x / TB;
  const unsigned col = blockIdx.x * TB + c;
  const int outer = a.dld.div(col), k2 = col - outer * a.dld.d;
  const bool ok = col < a.ncol && k2 < a.n2h;
  const int64_t off = outer * a.ostride + k2;
  const cpx<T>* tw = reinterpret_cast<const cpx<T>*>(a.tw);
  const int64_t st = a.stride;
  auto sx = [&](int j) { return j * TB + c; };
  auto field = [&](int f) { return reinterpret_cast<cpx<T>*>(a.data[3 * blockIdx.y + f]) + off; };
  // middle stages of one column buffer: cur -> oth -> cur ...; the result's buffer
  auto middle = [&](const auto& x, auto dir, cpx<T>* cur, cpx<T>* oth) {
    constexpr int DR = decltype(dir)::value;
    x.middle([&](auto rc, auto nb, auto p, auto, auto div_p) {
      constexpr int R = decltype(rc)::R;
      for (int i = i0; i < nb; i += ni) {
        const int k = i - p * div_p(i);
        cpx<T> u[R];
        load_stage<DR, T>(rc, u, cur, tw, i, k, nb, p, n, sx);
        const int j0 = (i - k) * R + k;
#pragma unroll
        for (int t = 0; t < R; ++t) oth[sx(j0 + t * p)] = u[t];
      }
      __syncthreads();
      cpx<T>* y = cur;
      cur = oth;
      oth = y;
    });
    return cur;
  };
#pragma unroll 1
  for (int f = f0; f < 3; f += nf) {
    const cpx<T>* g = field(f);
    cpx<T>* s = S + f * n * TB;
    ax.first([&](auto rc) {
      constexpr int R = decltype(rc)::R;
      const int nb = ax.nbf();
      for (int i = i0; i < nb; i += ni) {
        cpx<T> u[R];
#pragma unroll
        for (int t = 0; t < R; ++t) u[t] = ok ? g[(i + t * nb) * st] : cpx<T>{(T)0, (T)0};
        stage_first<-1, T>(rc, u, tw, n);
#pragma unroll
        for (int t = 0; t < R; ++t) s[sx(i * R + t)] = u[t];
      }
    });
  }
  __syncthreads();
  const int nbl = ax.nbl();
#pragma unroll 1
  for (int f = f0; f < 3; f += nf) {
    cpx<T>* s = S + f * n * TB;
    const cpx<T>* cur = s;
    if (ax.nst() > 2) cur = middle(ax, std::integral_constant<int, -1>{}, s, D);
    ax.last([&](auto rc) {
      constexpr int R = decltype(rc)::R;
      for (int i = i0; i < nbl; i += ni) {
        cpx<T> u[R];
        load_stage<-1, T>(rc, u, cur, tw, i, i, nbl, nbl, n, sx);
#pragma unroll
        for (int t = 0; t < R; ++t) s[sx(i + t * nbl)] = u[t];
      }
    });
    __syncthreads();      // D is read before the next field's middle stages write it, S written before it is combined
  }
  const T* K = reinterpret_cast<const T*>(a.K) + (int64_t)outer * a.n2h + k2;
  const int64_t kst = (int64_t)a.n1 * a.n2h;
  const T scl = sc<T>(a.scale), sc6 = scl * (T)(1.0 / 6.0);
#pragma unroll 1
  for (int o = f0; o < 3; o += nf) {
    ax.last([&](auto rc) {
      constexpr int R = decltype(rc)::R;
      for (int i = i0; i < nbl; i += ni) {
        cpx<T> u[R];
#pragma unroll
        for (int t = 0; t < R; ++t) {
          const int j = i + t * nbl;
          const T* kj = K + j * kst;
          // coefficients of F0, F1, F2
          T q0 = (T)0, q1 = (T)0, q2 = (T)0;
          if (ok) {
            if (o == 0) {
              q0 = __ldg(kj) * scl;
              q1 = __ldg(kj + a.kstride) * sc6;
              q2 = __ldg(kj + 2 * a.kstride) * scl;
            } else if (o == 1) {
              q0 = __ldg(kj + a.kstride) * sc6;
              q1 = __ldg(kj + 3 * a.kstride) * scl;
            } else {
              q0 = __ldg(kj + 2 * a.kstride) * scl;
            }
          }
          const cpx<T> g0 = S[sx(j)];
          cpx<T> v = {q0 * g0.x, q0 * g0.y};
          if (o < 2) {
            const cpx<T> g1 = S[n * TB + sx(j)];
            v = cpx<T>{v.x + q1 * g1.x, v.y + q1 * g1.y};
          }
          if (o == 0) {
            const cpx<T> g2 = S[2 * n * TB + sx(j)];
            v = cpx<T>{v.x + q2 * g2.x, v.y + q2 * g2.y};
          }
          u[t] = v;
        }
        stage_first<1, T>(rc, u, tw, n);
#pragma unroll
        for (int t = 0; t < R; ++t) D[sx(i * R + t)] = u[t];
      }
    });
    __syncthreads();
    const cpx<T>* cur = middle(axi, std::integral_constant<int, 1>{}, D, E);
    cpx<T>* g = field(o);
    axi.last([&](auto rc) {
      constexpr int R = decltype(rc)::R;
      const int nb = axi.nbl();
      for (int i = i0; i < nb; i += ni) {
        cpx<T> u[R];
        load_stage<1, T>(rc, u, cur, tw, i, i, nb, nb, n, sx);
        if (ok) {
#pragma unroll
          for (int t = 0; t < R; ++t) g[(i + t * nb) * st] = u[t];
        }
      }
    });
    __syncthreads();
  }
}

// ---- host side --------------------------------------------------------------------
// what the launch shapes need to know of an axis type
struct AxisInfo { int n, nst, nbf, nbl, nbmax; };
template <typename AX> inline AxisInfo axis_info(const RbAxis& a) {
  AxisInfo x;
  if constexpr (AX::kFixed) {
    x = AxisInfo{AX::n(), AX::nst(), AX::nbf(), AX::nbl(), AX::nbf() > AX::nbl() ? AX::nbf() : AX::nbl()};
  } else {
    x = AxisInfo{a.n, a.nst, a.nb[0], a.nb[a.nst - 1], 0};
    for (int s = 0; s < a.nst; ++s) x.nbmax = a.nb[s] > x.nbmax ? a.nb[s] : x.nbmax;
  }
  return x;
}

template <typename K> inline int launch_check(const char* what) {
  gb_count_launch();
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : gb_set_error(GBOFDFT_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

// f(axis type, reversed axis type) for a length.  The FP32 lengths listed
// above have kernels with every index folded at compile time: no radix switch, no
// index arithmetic between a thread's loads (128^3, three fields: a column pass
// 12.5 -> 9.4 us, the convolution 34 -> 16 us).  FP64 passes wait for the FP64
// pipe, and the kernels with run-time lengths are as fast.  Each translation unit
// holds one group of lengths (GB_RB_GROUP); group 0 holds every other length.
// 1: the length belongs to another group.
template <typename A, typename B> struct AxPair { using ax = A; using inv = B; };
// inverse rows: the order whose last radix is the smaller (a thread ends with
// that many points of a row pair)
template <typename P, bool FIXED> struct InverseOrder { using type = typename P::ax; };
template <typename P> struct InverseOrder<P, true> {
  using type = std::conditional_t<(P::ax::rl() <= P::inv::rl()), typename P::ax, typename P::inv>;
};
template <typename P> using inverse_order = typename InverseOrder<P, P::ax::kFixed>::type;
#define GB_RB_G(...) Rad<__VA_ARGS__>
template <typename T, typename F> static int by_axis(const RbAxis& ax, F&& f) {
#define GB_RB_TWO(LEN, A, B)                                                \
  case LEN:                                                                 \
    static_assert(Ax2<A, B>::N == LEN, "the radices make another length");  \
    return f(AxPair<Ax2<A, B>, Ax2<B, A>>{});
#define GB_RB_THREE(LEN, A, B, C)                                              \
  case LEN:                                                                    \
    static_assert(Ax3<A, B, C>::N == LEN, "the radices make another length");  \
    return f(AxPair<Ax3<A, B, C>, Ax3<C, B, A>>{});
#define GB_RB_OTHER(N, ...) case N: return 1;
  if constexpr (sizeof(T) == 4) {
    switch (ax.n) {
#if GB_RB_GROUP == 0
      GB_RB_LENGTHS_1(GB_RB_OTHER) GB_RB_LENGTHS_2(GB_RB_OTHER) GB_RB_LENGTHS_3(GB_RB_OTHER)
      GB_RB_LENGTHS_4(GB_RB_OTHER) GB_RB_LENGTHS3(GB_RB_OTHER)
#elif GB_RB_GROUP == 1
      GB_RB_LENGTHS_1(GB_RB_TWO)
#elif GB_RB_GROUP == 2
      GB_RB_LENGTHS_2(GB_RB_TWO)
#elif GB_RB_GROUP == 3
      GB_RB_LENGTHS_3(GB_RB_TWO)
#elif GB_RB_GROUP == 4
      GB_RB_LENGTHS_4(GB_RB_TWO)
      GB_RB_LENGTHS3(GB_RB_THREE)
#endif
      default: break;
    }
  }
#undef GB_RB_TWO
#undef GB_RB_THREE
#undef GB_RB_OTHER
#if GB_RB_GROUP == 0
  return f(AxPair<AxRun<T>, AxRun<T>>{});
#else
  return 1;
#endif
}

constexpr size_t kMaxSmem = 227 * 1024;   // longer lines take the run-time-radix passes (return 1)
constexpr int kSMs = 152;

// Row pairs and threads of a row CTA.  Every candidate is rated by the lanes
// that its stages keep busy (a warp instruction costs the same with idle
// lanes) and by how evenly the CTAs divide over the SMs; shared memory lets
// four CTAs be resident.
struct RowShape { int lp, threads; };
template <typename T> inline RowShape row_shape(const AxisInfo& ax, int nf, int nbuf, int nrows) {
  const int lines = nf > 0 ? nf : 1;
  const size_t per = sizeof(cpx<T>) * (size_t)line_pitch<T>(ax.n) * lines * nbuf;
  const int nbl = ax.nbl, nbf = ax.nbf;
  RowShape best{1, 32};
  double rate = -1.0;
  for (int lp = 1; lp <= RowCta<T>::NT && (lp == 1 || lp * per <= 56 * 1024); ++lp) {
    int th = (lp * nbl + 31) / 32 * 32;
    if (th > RowCta<T>::NT) {
      if (lp > 1) break;
      th = RowCta<T>::NT;
    }
    auto busy = [&](int tasks) { return tasks / (double)((tasks + th - 1) / th * th); };
    const double lanes = 0.5 * busy(lp * nbl) + 0.5 * busy(lines * lp * nbf);
    const double ctas = (double)((nrows + 2 * lp - 1) / (2 * lp));
    const double waves = ctas / kSMs, even = waves / ceil(waves);
    // fewer than 8 warps on an SM, or CTAs of one warp, leave latencies exposed
    const double warps = waves * th / 32.0;
    const double r = lanes * even * (th < 64 ? 0.9 : 1.0) * (warps < 8.0 ? warps / 8.0 : 1.0);
    if (r > rate + 1e-9) {
      rate = r;
      best = RowShape{lp, th};
    }
  }
  return best;
}

template <typename T>
static int rows_fwd(gbofdft_plan* p, const RbFwd& d, cudaStream_t st) {
  RowsFwd a;
  memset(&a, 0, sizeof(a));
  a.ax = p->rb[2];
  if (a.ax.nst == 0) return 1;
  const int nf = d.nf;
  const int* ops = d.op;
  for (int f = 0; f < GB_RB_FIELDS; ++f) {
    a.in[f] = f < nf ? d.in[f] : nullptr;
    a.out[f] = f < nf ? d.out[f] : nullptr;
    a.op[f] = f < nf ? ops[f] : OP_RHO;
  }
  a.nrows = p->n[0] * p->n[1]; a.n2h = p->n2h; a.ld2 = d.ld2; a.nf = nf;
  a.b56 = fabs(d.beta - 5.0 / 6.0) < 1e-15;
  a.rsq = rb_rsqrt_length(p->n[2]);
  a.beta.set(d.beta);
  a.beta2.set(d.beta2);
  a.half.set(0.5 * d.scale);
  a.rho0.set(d.rho0);
  a.inv0.set(d.rho0 > 0.0 ? 1.0 / d.rho0 : 0.0);
  a.pw_out = d.pw_out; a.pw2_out = d.pw2_out; a.pw_in = d.pw_in;
  a.tw = p->tw[2];
  a.dn.set(p->n[2]);
  a.dnh.set(p->n2h);
  int kind = PK_PLAIN;
  for (int f = 0; f < nf; ++f) {
    if (ops[f] >= OP_WGC0) kind = PK_WGC;
    else if (ops[f] == OP_SQRT || (ops[f] == OP_POWB && a.b56)) kind = kind > PK_ROOTS ? kind : PK_ROOTS;
    else if (ops[f] != OP_RHO) kind = PK_GENERAL;
  }
  auto go = [&](auto kern, const AxisInfo& x, int nbuf) -> int {
    const RowShape sh = row_shape<T>(x, nf, nbuf, a.nrows);
    a.lp = sh.lp;
    const size_t sm = nbuf * sizeof(cpx<T>) * (size_t)nf * a.lp * line_pitch<T>(x.n);
    if (sm > kMaxSmem) return 1;
    if (int rc = gbct::ct_smem(kern, sm)) return rc;
    kern<<<(a.nrows + 2 * a.lp - 1) / (2 * a.lp), sh.threads, sm, st>>>(a);
    return launch_check<T>("rb_rows_fwd");
  };
  return by_axis<T>(a.ax, [&](auto x) {
    using AX = typename decltype(x)::ax;
    const AxisInfo xi = axis_info<AX>(a.ax);
    if (kind == PK_GENERAL) return go(k_rb_rows_fwd<T, PK_GENERAL, AX>, xi, 2);
    if (kind == PK_WGC) return go(k_rb_rows_fwd<T, PK_WGC, AX>, xi, one_buffer<T, PK_WGC, AX>() ? 1 : 2);
    if (kind == PK_ROOTS) return go(k_rb_rows_fwd<T, PK_ROOTS, AX>, xi, one_buffer<T, PK_ROOTS, AX>() ? 1 : 2);
    return go(k_rb_rows_fwd<T, PK_PLAIN, AX>, xi, one_buffer<T, PK_PLAIN, AX>() ? 1 : 2);
  });
}

template <typename T>
static int rows_inv(gbofdft_plan* p, const RbInv& d, int64_t* nblk_out, cudaStream_t st) {
  RowsInv a;
  memset(&a, 0, sizeof(a));
  a.ax = p->rb[2];
  if (a.ax.nst == 0) return 1;
  const int nf = d.nf;
  const EvalDesc* ev = d.ev;
  for (int f = 0; f < nf; ++f) a.in[f] = d.in[f];
  a.nrows = p->n[0] * p->n[1]; a.n2h = p->n2h; a.ld2 = d.ld2; a.nf = nf;
  a.tw = p->tw[2];
  a.out = d.out; a.ostride = d.ostride; a.scale.set(d.scale);
  const int nrows = a.nrows;
  auto go = [&](auto kern, const AxisInfo& x) -> int {
    const int nbuf = x.nst > 2 ? 2 : 1;
    const RowShape sh = row_shape<T>(x, nf, nbuf, nrows);
    a.lp = sh.lp;
    const int nblk = (nrows + 2 * sh.lp - 1) / (2 * sh.lp);
    if (nblk_out) *nblk_out = nblk;
    const size_t sm = nbuf * sizeof(cpx<T>) * (size_t)nf * a.lp * line_pitch<T>(x.n);
    if (sm > kMaxSmem) return 1;
    if (int rc = gbct::ct_smem(kern, sm)) return rc;
    kern<<<nblk, sh.threads, sm, st>>>(a);
    return launch_check<T>("rb_rows_inv");
  };
  if (!ev)
    return by_axis<T>(a.ax, [&](auto x) {
      using AX = inverse_order<decltype(x)>;
      return go(k_rb_rows_inv<T, RI_STORE, AX>, axis_info<AX>(a.ax));
    });
  a.ev = *ev; a.rho = d.rho; a.vloc = d.vloc; a.pot = d.pot; a.partials = d.partials;
  a.base = ev->tf || ev->vw || ev->wt || ev->xc || ev->hartree || ev->pp;
  a.add = d.add;
  if (d.wgc) {
    a.wgc = 1;
    a.wslot = d.wslot;
    a.two = d.two;
    a.w_rho0.set(d.wgc->rho0);
    a.w_inv0.set(1.0 / d.wgc->rho0);
    a.w_a.set(d.wgc->alpha);
    a.w_b.set(d.wgc->beta);
    a.pa = d.pa; a.pb = d.pb;
    for (int i = 0; i < 6; ++i) a.wstore[i] = d.wstore[i];
    a.vstore = d.vstore;
  }
  const double ctf = 2.87123400018819181594;    // (3/10)(3 pi^2)^(2/3)
  a.tf_v.set(4.78539000031365302657 * ev->tf_x);   // (5/3) ctf
  a.tf_vl.set(a.tf_v.d - (double)a.tf_v.f);        // (FP32: the rest of it)
  a.tf_e.set(ctf * ev->tf_x);
  a.vw_y.set(ev->vw_y);
  a.half_vw.set(0.5 * ev->vw_y);
  a.two_alpha.set(2.0 * ev->wt_alpha);
  a.inv_two_alpha.set(ev->wt_alpha != 0.0 ? 1.0 / (2.0 * ev->wt_alpha) : 0.0);
  a.wt_beta.set(ev->wt_beta);
  a.b56 = fabs(ev->wt_beta - 5.0 / 6.0) < 1e-15;
  return by_axis<T>(a.ax, [&](auto x) {
    using AX = inverse_order<decltype(x)>;
    const AxisInfo xi = axis_info<AX>(a.ax);
    return d.calc_e ? go(k_rb_rows_inv<T, RI_EVAL_E, AX>, xi) : go(k_rb_rows_inv<T, RI_EVAL, AX>, xi);
  });
}

// Butterflies of a column side by side.  FP64: one per thread of the stage with
// the most (idle warps cost nothing on the FP64 pipe).  FP32: as many as keep
// the threads of every stage busy, the last stage weighed with wl.
template <typename T> inline int column_threads(const AxisInfo& x, int cap, double wl) {
  const int rounds = (x.nbmax + cap - 1) / cap;
  int ni = (x.nbmax + rounds - 1) / rounds;
  if (sizeof(T) == 4) {
    double best = -1.0;
    for (int c = x.nbl < x.nbf ? x.nbl : x.nbf; c <= x.nbmax && c <= cap; ++c) {
      auto busy = [&](int nb) { return nb / (double)((nb + c - 1) / c * c); };
      const double r = busy(x.nbf) + wl * busy(x.nbl) + 1e-3 * c;
      if (r > best) {
        best = r;
        ni = c;
      }
    }
  }
  return ni;
}

// LWT columns along axis 0
template <typename T>
static int lwt_cols(gbofdft_plan* p, const RbLwt& d, cudaStream_t st) {
  LwtCols a;
  memset(&a, 0, sizeof(a));
  a.ax = p->rb[0];
  if (a.ax.nst < 2) return 1;
  for (int f = 0; f < d.nf; ++f) {
    a.in[f] = d.in[f];
    a.out[f] = d.out[f];
    a.K[f] = d.K[f];
  }
  a.stride = (int64_t)p->n[1] * d.ld2;
  a.kst = (int64_t)p->n[1] * p->n2h;
  a.ostride = d.ld2;
  a.ncol = (unsigned)p->n[1] * d.ld2; a.n2h = p->n2h; a.nf = d.nf; a.first = d.first;
  a.dld.set(d.ld2);
  a.tw = p->tw[0];
  return by_axis<T>(a.ax, [&](auto x) {
    using AX = typename decltype(x)::ax;
    const AxisInfo xi = axis_info<AX>(a.ax);
    auto go = [&](auto kern, auto tb, unsigned nf) -> int {
      constexpr int TB = decltype(tb)::value;
      const size_t sm = (xi.nst > 2 ? 2 : 1) * sizeof(cpx<T>) * (size_t)TB * xi.n;
      if (sm > kMaxSmem) return 1;
      if (int rc = gbct::ct_smem(kern, sm)) return rc;
      const int threads = TB * column_threads<T>(xi, (sizeof(T) == 4 ? 400 : 256) / TB, 1.0);
      kern<<<(a.ncol + TB - 1) / TB * nf, threads, sm, st>>>(a);
      return launch_check<T>("rb_lwt");
    };
    if (d.dir > 0) return go(k_rb_lwt<T, 1, AX>, std::integral_constant<int, lwt_tb<T, 1, AX>()>{}, d.nf);
    return go(k_rb_lwt<T, -1, AX>, std::integral_constant<int, lwt_tb<T, -1, AX>()>{}, 1);
  });
}

// LWT rows: inverse (d.out1) or forward
template <typename T>
static int lwt_rows(gbofdft_plan* p, const RbLwtRows& d, cudaStream_t st) {
  LwtRows a;
  memset(&a, 0, sizeof(a));
  a.ax = p->rb[2];
  if (a.ax.nst == 0) return 1;
  const LwtKnots& k = *d.knots;
  const int inverse = d.out1 != nullptr, nk = inverse && d.out3 ? 2 : 1;
  for (int f = 0; f < (inverse ? nk : 0) * k.m; ++f) a.in[f] = d.in[f];
  for (int f = 0; f < (inverse ? 0 : k.m); ++f) a.out[f] = d.out[f];
  a.kf = d.kf; a.ra = d.ra; a.out1 = d.out1; a.out3 = d.out3; a.first = d.first;
  a.m = k.m; a.below = k.below;
  a.nrows = p->n[0] * p->n[1]; a.n2h = p->n2h; a.ld2 = d.ld2;
  a.dnh.set(p->n2h);
  a.tw = p->tw[2];
  a.half.set(0.5 * d.scale);
  for (int e = 0; e <= k.m; ++e) {
    a.lo[e].set(k.lo[e]);
    a.hi[e].set(k.hi[e]);
    a.inv[e].set(k.inv[e]);
  }
  a.kl.set(k.kl); a.kl_e.set(k.kl_e); a.inv_kl.set(k.inv_kl);
  auto go = [&](auto kern, const AxisInfo& x) -> int {
    const int nbuf = x.nst > 2 ? 2 : 1;
    const RowShape sh = row_shape<T>(x, nk, nbuf, a.nrows);
    a.lp = sh.lp;
    const size_t sm = nbuf * sizeof(cpx<T>) * (size_t)nk * a.lp * line_pitch<T>(x.n);
    if (sm > kMaxSmem) return 1;
    if (int rc = gbct::ct_smem(kern, sm)) return rc;
    kern<<<(a.nrows + 2 * a.lp - 1) / (2 * a.lp), sh.threads, sm, st>>>(a);
    return launch_check<T>("rb_lwt_rows");
  };
  return by_axis<T>(a.ax, [&](auto x) {
    using P = decltype(x);
    if (inverse) return go(k_rb_lwt_rows_inv<T, inverse_order<P>>, axis_info<inverse_order<P>>(a.ax));
    return go(k_rb_lwt_rows_fwd<T, typename P::ax>, axis_info<typename P::ax>(a.ax));
  });
}

// WGC: the WGC kernel on groups of three fields, else plain columns or (kd) the convolution
template <typename T, bool WGC>
static int cols(gbofdft_plan* p, const RbCols& d, cudaStream_t st) {
  Cols a;
  memset(&a, 0, sizeof(a));
  const int axis = d.axis, nf = d.nf, dir = d.dir, ld2 = d.ld2;
  const KerDesc* kd = d.kd;
  a.ax = p->rb[axis];
  if (a.ax.nst == 0) return 1;
  a.inv = p->rbi[axis];
  const int outer = p->n[axis == 1 ? 0 : 1];
  for (int f = 0; f < nf; ++f) a.data[f] = d.data[f];
  a.stride = axis == 1 ? ld2 : (int64_t)p->n[1] * ld2;
  a.ostride = axis == 1 ? (int64_t)p->n[1] * ld2 : ld2;
  a.ncol = (unsigned)outer * ld2; a.n2h = p->n2h; a.dld.set(ld2);
  a.tw = p->tw[axis]; a.scale.set(d.scale);
  a.n0 = p->n[0]; a.n1 = p->n[1]; a.n2 = p->n[2]; a.full = p->full;
  for (int i = 0; i < 9; ++i) a.bg[i].set(p->bg[i]);
  if (kd)
    for (int f = 0; f < nf; ++f) {
      a.type[f] = kd->type[f];
      a.arr[f] = kd->arr[f];
      a.coef[f].set(kd->coef[f]);
    }
  a.K = d.K;
  a.kstride = p->NG;
  a.src = d.src;
  a.sstride = axis == 1 ? d.src_ld : (int64_t)p->n[1] * d.src_ld;
  a.sostride = axis == 1 ? (int64_t)p->n[1] * d.src_ld : d.src_ld;
  constexpr int TB = ColTile<T>::TB;
  const dim3 grid((a.ncol + TB - 1) / TB, WGC ? nf / 3 : nf);
  auto go = [&](auto kern, const AxisInfo& x) -> int {
    auto smem = [&](int fy) {
      const int nbuf = WGC ? 3 + fy * (x.nst > 2 ? 2 : 1) : x.nst < 2 ? 0 : (kd || x.nst > 2 ? 2 : 1);
      return nbuf * sizeof(cpx<T>) * (size_t)TB * x.n;
    };
    const int fy = WGC && sizeof(T) == 4 && smem(3) <= kMaxSmem ? 3 : 1;
    const int cap = WGC ? kWgcThreads<T> / (TB * fy) : (sizeof(T) == 4 ? 400 : 256) / TB;
    // the last stage of the convolution continues with the inverse's first
    const int ni = column_threads<T>(x, cap, kd || WGC ? 2.0 : 1.0);
    const size_t sm = smem(fy);
    if (sm > kMaxSmem) return 1;
    if (int rc = gbct::ct_smem(kern, sm)) return rc;
    kern<<<grid, dim3(TB * ni, fy), sm, st>>>(a);
    return launch_check<T>("rb_cols");
  };
  return by_axis<T>(a.ax, [&](auto x) {
    using AX = typename decltype(x)::ax;
    using AXI = typename decltype(x)::inv;
    const AxisInfo xi = axis_info<AX>(a.ax);
    if constexpr (WGC) {
      if (xi.nst < 2) return 1;
      return go(k_rb_wgc<T, AX, AXI>, xi);
    } else {
      if (kd) return go(k_rb_cols<T, -1, true, AX, AXI>, xi);
      return dir < 0 ? go(k_rb_cols<T, -1, false, AX, AXI>, xi) : go(k_rb_cols<T, 1, false, AX, AXI>, xi);
    }
  });
}

}  // namespace gbrb

// Instantiate the launchers of one precision and group of lengths (row and
// column passes in translation units of their own: they compile in parallel).
#define GB_RB_NAME(base, SUF) GB_RB_CAT(GB_RB_CAT(base##_##SUF, _g), GB_RB_GROUP)
#define GB_RB_DEFINE_FWD(T, SUF)                                                                                \
  int GB_RB_NAME(gb_rb_rows_fwd, SUF)(gbofdft_plan* p, const RbFwd& d, cudaStream_t st) {                      \
    return gbrb::rows_fwd<T>(p, d, st);                                                                        \
  }
#define GB_RB_DEFINE_INV(T, SUF)                                                                                \
  int GB_RB_NAME(gb_rb_rows_inv, SUF)(gbofdft_plan* p, const RbInv& d, int64_t* nblk, cudaStream_t st) {       \
    return gbrb::rows_inv<T>(p, d, nblk, st);                                                                  \
  }
#define GB_RB_DEFINE_COLS(T, SUF)                                                                               \
  int GB_RB_NAME(gb_rb_cols, SUF)(gbofdft_plan* p, const RbCols& d, cudaStream_t st) {                         \
    return gbrb::cols<T, false>(p, d, st);                                                                     \
  }
#define GB_RB_DEFINE_WGC(T, SUF)                                                                                \
  int GB_RB_NAME(gb_rb_wgc, SUF)(gbofdft_plan* p, const RbCols& d, cudaStream_t st) {                          \
    return gbrb::cols<T, true>(p, d, st);                                                                      \
  }
#define GB_RB_DEFINE_LWT(T, SUF)                                                                                \
  int GB_RB_NAME(gb_rb_lwt, SUF)(gbofdft_plan* p, const RbLwt& d, cudaStream_t st) {                           \
    return gbrb::lwt_cols<T>(p, d, st);                                                                        \
  }                                                                                                             \
  int GB_RB_NAME(gb_rb_lwt_rows, SUF)(gbofdft_plan* p, const RbLwtRows& d, cudaStream_t st) {                  \
    return gbrb::lwt_rows<T>(p, d, st);                                                                        \
  }
