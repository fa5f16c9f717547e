// Register-blocked FFT stages for lines of any 2, 3, 5, 7-smooth length.
//
// A line of length n is a Stockham transform with few large radices (two
// stages for most lengths up to 400, three above): every thread holds whole
// butterflies of a stage in registers, so a line crosses shared memory once
// between two stages instead of once per small radix.  The radices are
// compile-time codelets (below); which of them a length uses is decided on
// the host (RbAxis) and selected in the kernel by a branch that is uniform
// over the CTA, so one kernel serves every length.
//
// Composite radices whose factors are coprime (6, 10, 12, 14, 15) use
// the Good-Thomas prime-factor index maps: no twiddle factors inside.
//
// Stage s (radix r, p = product of the radices before it), butterfly i in
// [0, n/r), k = i % p:
//   u_t = in[i + t n/r] w^(t k), w = exp(DIR 2 pi i / (p r));  v = DFT_r(u);
//   out[(i - k) r + k + t p] = v_t.
// For the last stage p = n/r, so k = i and butterfly i reads and produces the
// elements i + t n/r: an inverse transform whose first radix is that r can
// continue in the same registers (the convolution pass does).
#pragma once
#include <type_traits>

#include "fft_core.cuh"
#include "rb_axis.h"

namespace gbrb {

using gbfft::dft2;
using gbfft::dft4;

constexpr int inv_mod(int a, int m) {
  for (int x = 1; x < m; ++x)
    if ((a * x) % m == 1) return x;
  return 1;
}

// The codelets are written so that multiplications land in fused
// multiply-adds (a +- s b in one instruction each): on the FP64 pipe, which
// bounds the FP64 passes, every instruction counts the same.

// a + DIR i s b and a - DIR i s b
template <int DIR, typename T>
__device__ __forceinline__ void rot_pair(cpx<T> a, cpx<T> b, T s, cpx<T>& p, cpx<T>& m) {
  const T d = DIR < 0 ? s : -s;
  p = cpx<T>{fma(d, b.y, a.x), fma(-d, b.x, a.y)};
  m = cpx<T>{fma(-d, b.y, a.x), fma(d, b.x, a.y)};
}

template <int DIR, typename T>
__device__ __forceinline__ void dft3(cpx<T>* u) {
  const cpx<T> t = c_add(u[1], u[2]), d = c_sub(u[1], u[2]);
  const cpx<T> m = {fma((T)-0.5, t.x, u[0].x), fma((T)-0.5, t.y, u[0].y)};
  u[0] = c_add(u[0], t);
  rot_pair<DIR, T>(m, d, (T)GB_S3, u[1], u[2]);
}

template <int DIR, typename T>
__device__ __forceinline__ void dft5(cpx<T>* u) {
  const T q = (T)0.55901699437494742410;                    // sqrt(5) / 4
  const T r = (T)0.61803398874989484820;                    // sin(4 pi / 5) / sin(2 pi / 5)
  const cpx<T> t1 = c_add(u[1], u[4]), t2 = c_add(u[2], u[3]);
  const cpx<T> t3 = c_sub(u[1], u[4]), t4 = c_sub(u[2], u[3]);
  const cpx<T> s = c_add(t1, t2), d = c_sub(t1, t2);
  const cpx<T> m = {fma((T)-0.25, s.x, u[0].x), fma((T)-0.25, s.y, u[0].y)};
  const cpx<T> a1 = {fma(q, d.x, m.x), fma(q, d.y, m.y)}, a2 = {fma(-q, d.x, m.x), fma(-q, d.y, m.y)};
  const cpx<T> b1 = {fma(r, t4.x, t3.x), fma(r, t4.y, t3.y)}, b2 = {fma(r, t3.x, -t4.x), fma(r, t3.y, -t4.y)};
  u[0] = c_add(u[0], s);
  rot_pair<DIR, T>(a1, b1, (T)GB_S5A, u[1], u[4]);
  rot_pair<DIR, T>(a2, b2, (T)GB_S5A, u[2], u[3]);
}

template <int DIR, typename T>
__device__ __forceinline__ void dft7(cpx<T>* u) {
  // cos / sin (2 pi j / 7), j = 1, 2, 3; the sines as ratios to s1
  const T c1 = (T)0.62348980185873353053, c2 = (T)-0.22252093395631440429, c3 = (T)-0.90096886790241912624;
  const T s1 = (T)0.78183148246802980871, r2 = (T)1.24697960371746706106, r3 = (T)0.55495813208737119142;
  const cpx<T> p1 = c_add(u[1], u[6]), p2 = c_add(u[2], u[5]), p3 = c_add(u[3], u[4]);
  const cpx<T> m1 = c_sub(u[1], u[6]), m2 = c_sub(u[2], u[5]), m3 = c_sub(u[3], u[4]);
  const cpx<T> a1 = {u[0].x + c1 * p1.x + c2 * p2.x + c3 * p3.x, u[0].y + c1 * p1.y + c2 * p2.y + c3 * p3.y};
  const cpx<T> a2 = {u[0].x + c2 * p1.x + c3 * p2.x + c1 * p3.x, u[0].y + c2 * p1.y + c3 * p2.y + c1 * p3.y};
  const cpx<T> a3 = {u[0].x + c3 * p1.x + c1 * p2.x + c2 * p3.x, u[0].y + c3 * p1.y + c1 * p2.y + c2 * p3.y};
  const cpx<T> b1 = {m1.x + r2 * m2.x + r3 * m3.x, m1.y + r2 * m2.y + r3 * m3.y};
  const cpx<T> b2 = {r2 * m1.x - r3 * m2.x - m3.x, r2 * m1.y - r3 * m2.y - m3.y};
  const cpx<T> b3 = {r3 * m1.x - m2.x + r2 * m3.x, r3 * m1.y - m2.y + r2 * m3.y};
  u[0] = c_add(u[0], c_add(p1, c_add(p2, p3)));
  rot_pair<DIR, T>(a1, b1, s1, u[1], u[6]);
  rot_pair<DIR, T>(a2, b2, s1, u[2], u[5]);
  rot_pair<DIR, T>(a3, b3, s1, u[3], u[4]);
}

template <int DIR, typename T>
__device__ __forceinline__ void dft8(cpx<T>* u) {
  const T h = (T)GB_R2;
  cpx<T> b[4], c[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    b[k] = c_add(u[k], u[k + 4]);
    c[k] = c_sub(u[k], u[k + 4]);
  }
  // odd outputs: DFT4 of c_k exp(DIR i pi k / 4); the sqrt(1/2) of k = 1, 3
  // goes into the last additions
  const cpx<T> c1 = c_add(c[1], c_rot<DIR>(c[1])), c2 = c_rot<DIR>(c[2]), c3 = c_sub(c_rot<DIR>(c[3]), c[3]);
  const cpx<T> a = c_add(c[0], c2), d = c_sub(c[0], c2), s = c_add(c1, c3), e = c_sub(c1, c3);
  dft4<DIR, T>(b);
#pragma unroll
  for (int k = 0; k < 4; ++k) u[2 * k] = b[k];
  u[1] = cpx<T>{fma(h, s.x, a.x), fma(h, s.y, a.y)};
  u[5] = cpx<T>{fma(-h, s.x, a.x), fma(-h, s.y, a.y)};
  rot_pair<DIR, T>(d, e, h, u[3], u[7]);
}

// a + w b and a - w b in six fused operations
template <typename T>
__device__ __forceinline__ void tw_pair(cpx<T> a, cpx<T> b, T wx, T wy, cpx<T>& p, cpx<T>& m) {
  p = cpx<T>{fma(wx, b.x, fma(-wy, b.y, a.x)), fma(wx, b.y, fma(wy, b.x, a.y))};
  m = cpx<T>{fma((T)2, a.x, -p.x), fma((T)2, a.y, -p.y)};
}

// 16 = 2 x 8: DFT8 of the even and of the odd inputs, then radix-2
// butterflies with exp(DIR 2 pi i k / 16)
template <int DIR, typename T>
__device__ __forceinline__ void dft16(cpx<T>* u) {
  const T c = (T)0.92387953251128675613, s = (T)0.38268343236508977173, h = (T)GB_R2;   // pi / 8
  const T d = DIR < 0 ? (T)-1 : (T)1;
  cpx<T> e[8], o[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    e[k] = u[2 * k];
    o[k] = u[2 * k + 1];
  }
  dft8<DIR, T>(e);
  dft8<DIR, T>(o);
  u[0] = c_add(e[0], o[0]);
  u[8] = c_sub(e[0], o[0]);
  tw_pair<T>(e[1], o[1], c, d * s, u[1], u[9]);
  tw_pair<T>(e[2], o[2], h, d * h, u[2], u[10]);
  tw_pair<T>(e[3], o[3], s, d * c, u[3], u[11]);
  u[4] = c_add(e[4], c_rot<DIR>(o[4]));
  u[12] = c_sub(e[4], c_rot<DIR>(o[4]));
  tw_pair<T>(e[5], o[5], -s, d * c, u[5], u[13]);
  tw_pair<T>(e[6], o[6], -h, d * h, u[6], u[14]);
  tw_pair<T>(e[7], o[7], -c, d * s, u[7], u[15]);
}

// 9 = 3 x 3: u[m + 3 j] -> DFT3 over j, twiddles w9^(m k), DFT3 over m
template <int DIR, typename T>
__device__ __forceinline__ void dft9(cpx<T>* u) {
  const T d = DIR < 0 ? (T)-1 : (T)1;
  // exp(DIR 2 pi i j / 9), j = 1, 2, 4
  const cpx<T> w1 = {(T)0.76604444311897803520, d * (T)0.64278760968653932632};
  const cpx<T> w2 = {(T)0.17364817766693034885, d * (T)0.98480775301220805937};
  const cpx<T> w4 = {(T)-0.93969262078590838405, d * (T)0.34202014332566873304};
  cpx<T> q[3][3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
#pragma unroll
    for (int j = 0; j < 3; ++j) q[m][j] = u[m + 3 * j];
    dft3<DIR, T>(q[m]);
  }
  q[1][1] = c_mul(q[1][1], w1);
  q[1][2] = c_mul(q[1][2], w2);
  q[2][1] = c_mul(q[2][1], w2);
  q[2][2] = c_mul(q[2][2], w4);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    cpx<T> e[3] = {q[0][k], q[1][k], q[2][k]};
    dft3<DIR, T>(e);
#pragma unroll
    for (int j = 0; j < 3; ++j) u[k + 3 * j] = e[j];
  }
}

template <int DIR, typename T, int R>
__device__ __forceinline__ void dft(cpx<T>* u);

// Good-Thomas: n = A n_a + B n_b mod AB -> inputs (B n_a + A n_b) mod AB,
// outputs k with k = k_a mod A and k = k_b mod B
template <int DIR, typename T, int A, int B>
__device__ __forceinline__ void dft_pfa(cpx<T>* u) {
  constexpr int N = A * B;
  constexpr int EA = B * inv_mod(B % A, A), EB = A * inv_mod(A % B, B);
  cpx<T> q[A][B];
#pragma unroll
  for (int a = 0; a < A; ++a) {
#pragma unroll
    for (int b = 0; b < B; ++b) q[a][b] = u[(B * a + A * b) % N];
    dft<DIR, T, B>(q[a]);
  }
#pragma unroll
  for (int b = 0; b < B; ++b) {
    cpx<T> e[A];
#pragma unroll
    for (int a = 0; a < A; ++a) e[a] = q[a][b];
    dft<DIR, T, A>(e);
#pragma unroll
    for (int a = 0; a < A; ++a) u[(EA * a + EB * b) % N] = e[a];
  }
}

template <int DIR, typename T, int R>
__device__ __forceinline__ void dft(cpx<T>* u) {
  if constexpr (R == 2) dft2<DIR, T>(u);
  else if constexpr (R == 3) dft3<DIR, T>(u);
  else if constexpr (R == 4) dft4<DIR, T>(u);
  else if constexpr (R == 5) dft5<DIR, T>(u);
  else if constexpr (R == 6) dft_pfa<DIR, T, 2, 3>(u);
  else if constexpr (R == 7) dft7<DIR, T>(u);
  else if constexpr (R == 8) dft8<DIR, T>(u);
  else if constexpr (R == 9) dft9<DIR, T>(u);
  else if constexpr (R == 10) dft_pfa<DIR, T, 2, 5>(u);
  else if constexpr (R == 12) dft_pfa<DIR, T, 3, 4>(u);
  else if constexpr (R == 14) dft_pfa<DIR, T, 2, 7>(u);
  else if constexpr (R == 15) dft_pfa<DIR, T, 3, 5>(u);
  else if constexpr (R == 16) dft16<DIR, T>(u);
  else static_assert(R == 2, "radix not implemented");
}

// ---- stages ----------------------------------------------------------------
// A stage's butterfly is one of two kinds.
//
// Pfa<R> (FP64): the codelets above, fewest operations.
//
// Rad<Q...> (FP32): the radices Q one after the other on the same registers,
// each with its table twiddles -- exactly the operations of a transform that
// makes one pass per radix Q, so the rounding does not depend on how many of
// them a stage joins.  That matters in FP32: rho and sqrt(rho) have a mean as
// large as their variation, every partial sum carries it, its rounding is the
// noise of all high-G coefficients, and the G^2 kernel makes that noise the
// error of the potential.  A length's radices therefore stay what they are
// (8, 4, 2, 3, 5, 7; the lists of passes_rb.cuh have 128 as 8, 4, 4 and 360 as
// 8, 5, 3, 3).
template <int R_> struct Pfa { static constexpr int R = R_; };
template <int Q, int... Qs> struct Rad {
  static constexpr int R = Q * Rad<Qs...>::R;
};
template <int Q> struct Rad<Q> {
  static constexpr int R = Q;
};

template <int DIR, typename T, int R>
__device__ __forceinline__ void dft_small(cpx<T>* u) {
  if constexpr (R == 2) dft2<DIR, T>(u);
  else if constexpr (R == 3) gbfft::dft3<DIR, T>(u);
  else if constexpr (R == 4) dft4<DIR, T>(u);
  else if constexpr (R == 5) gbfft::dft5<DIR, T>(u);
  else if constexpr (R == 7) dft7<DIR, T>(u);
  else if constexpr (R == 8) gbfft::dft8<DIR, T>(u);
  else static_assert(R == 2, "radix not implemented");
}

// v w (v conj(w) for the inverse), each pair of products as one rounded
// product and one fused multiply-add, spelt out: the rounding must not depend
// on how the compiler pairs them
template <int DIR>
__device__ __forceinline__ float2 tw_mul(float2 a, float2 b) {
  if constexpr (DIR > 0) b.y = -b.y;
  return float2{__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.y, b.x, __fmul_rn(a.x, b.y))};
}

// Radix 7 as the plain sum over its inputs in order, the stage's twiddle (step
// e) and the DFT's (step n / 7) looked up together.  Forward transforms keep it with
// their radices, for the rounding of the mean; inverse ones take the cheaper codelet,
// since nothing amplifies their rounding.
template <int DIR, typename T>
__device__ __forceinline__ void dft7_direct(cpx<T>* u, const cpx<T>* __restrict__ tw, int e, int n) {
  cpx<T> o[7];
#pragma unroll
  for (int q = 0; q < 7; ++q) {
    cpx<T> acc = u[0];
#pragma unroll
    for (int t = 1; t < 7; ++t) {
      int m = t * e + ((t * q) % 7) * (n / 7);
      if (m >= n) m -= n;
      acc = c_add(acc, tw_mul<DIR>(u[t], __ldg(tw + m)));
    }
    o[q] = acc;
  }
#pragma unroll
  for (int q = 0; q < 7; ++q) u[q] = o[q];
}

// u in Stockham input order (element i + t n/R), out in output order (t p);
// k = i mod p; ONE: k = 0, no twiddles in the first radix
template <int DIR, typename T, bool ONE, int Q, int... Qs>
__device__ __forceinline__ void rad_dft(Rad<Q, Qs...>, cpx<T>* u, const cpx<T>* __restrict__ tw, int k, int p, int n) {
  constexpr int M = Rad<Q, Qs...>::R / Q;
  if constexpr (Q == 7 && M == 1 && DIR < 0) {
    dft7_direct<DIR, T>(u, tw, ONE ? 0 : k * (n / (p * Q)), n);
    return;
  }
  cpx<T> y[M][Q];
  const int step = ONE ? 0 : k * (n / (p * Q));
#pragma unroll
  for (int t = 0; t < Q; ++t) {
    cpx<T> w = {(T)1, (T)0};
    if (!ONE && t > 0) w = __ldg(tw + t * step);
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const cpx<T> v = u[m + t * M];
      y[m][t] = ONE || t == 0 ? v : tw_mul<DIR>(v, w);
    }
  }
#pragma unroll
  for (int m = 0; m < M; ++m) dft_small<DIR, T, Q>(y[m]);
  if constexpr (M == 1) {
#pragma unroll
    for (int t = 0; t < Q; ++t) u[t] = y[0][t];
  } else {
#pragma unroll
    for (int t = 0; t < Q; ++t) {
      cpx<T> z[M];
#pragma unroll
      for (int m = 0; m < M; ++m) z[m] = y[m][t];
      if (ONE && t == 0) rad_dft<DIR, T, true>(Rad<Qs...>{}, z, tw, 0, p * Q, n);
      else rad_dft<DIR, T, false>(Rad<Qs...>{}, z, tw, k + t * p, p * Q, n);
#pragma unroll
      for (int m = 0; m < M; ++m) u[t + Q * m] = z[m];
    }
  }
}

// first stage of a line (p = 1) / a later one, on the butterfly's registers
template <int DIR, typename T, int R>
__device__ __forceinline__ void stage_first(Pfa<R>, cpx<T>* u, const cpx<T>*, int) { dft<DIR, T, R>(u); }
template <int DIR, typename T, int... Q>
__device__ __forceinline__ void stage_first(Rad<Q...> r, cpx<T>* u, const cpx<T>* tw, int n) {
  rad_dft<DIR, T, true>(r, u, tw, 0, 1, n);
}
template <int DIR, typename T, int R>
__device__ __forceinline__ void stage_next(Pfa<R>, cpx<T>* u, const cpx<T>* __restrict__ tw, int k, int p, int n) {
  const int step = k * (n / (p * R));
#pragma unroll
  for (int t = 1; t < R; ++t) {
    const cpx<T> w = __ldg(tw + t * step);
    u[t] = DIR < 0 ? c_mul(u[t], w) : c_mulc(u[t], w);
  }
  dft<DIR, T, R>(u);
}
template <int DIR, typename T, int... Q>
__device__ __forceinline__ void stage_next(Rad<Q...> r, cpx<T>* u, const cpx<T>* tw, int k, int p, int n) {
  rad_dft<DIR, T, false>(r, u, tw, k, p, n);
}

// How a kernel sees its axis.  AxRun: any length, run-time strides, the radix
// of a stage selected by a branch that is uniform over the CTA.  Ax2, Ax3: the
// length G0 x G1 (x G2) with every index folded at compile time.
template <typename T> struct AxRun {
  static constexpr bool kFixed = false;
  const RbAxis& a;
  __device__ __forceinline__ explicit AxRun(const RbAxis& x) : a(x) {}
  __device__ __forceinline__ int n() const { return a.n; }
  __device__ __forceinline__ int nst() const { return a.nst; }
  __device__ __forceinline__ int nbf() const { return a.nb[0]; }
  __device__ __forceinline__ int nbl() const { return a.nb[a.nst - 1]; }
  __device__ __forceinline__ int rl() const { return a.r[a.nst - 1]; }
  __device__ __forceinline__ int div_nbf(int x) const { return a.dnb[0].div(x); }
  __device__ __forceinline__ int div_nbl(int x) const { return a.dnb[a.nst - 1].div(x); }
  template <typename F> static __device__ __forceinline__ void pick(int r, F&& f) {
    if constexpr (sizeof(T) == 4) {
      switch (r) {
        case 2: f(Rad<2>{}); break;
        case 3: f(Rad<3>{}); break;
        case 4: f(Rad<4>{}); break;
        case 5: f(Rad<5>{}); break;
        case 7: f(Rad<7>{}); break;
        case 8: f(Rad<8>{}); break;
        default: break;
      }
    } else {
      switch (r) {
        case 2: f(Pfa<2>{}); break;
        case 3: f(Pfa<3>{}); break;
        case 4: f(Pfa<4>{}); break;
        case 5: f(Pfa<5>{}); break;
        case 6: f(Pfa<6>{}); break;
        case 7: f(Pfa<7>{}); break;
        case 8: f(Pfa<8>{}); break;
        case 9: f(Pfa<9>{}); break;
        case 10: f(Pfa<10>{}); break;
        case 12: f(Pfa<12>{}); break;
        case 14: f(Pfa<14>{}); break;
        case 15: f(Pfa<15>{}); break;
        case 16: f(Pfa<16>{}); break;
        default: break;
      }
    }
  }
  template <typename F> __device__ __forceinline__ void first(F&& f) const { pick(a.r[0], f); }
  template <typename F> __device__ __forceinline__ void last(F&& f) const { pick(a.r[a.nst - 1], f); }
  // stages between the first and the last: f(butterfly, nb, p, i -> line division)
  template <typename F> __device__ __forceinline__ void middle(F&& f) const {
#pragma unroll 1
    for (int s = 1; s < a.nst - 1; ++s)
      pick(a.r[s], [&](auto rc) {
        const FastDiv dn = a.dnb[s], dp = a.dp[s];
        f(rc, a.nb[s], a.p[s], [=](int x) { return (int)dn.div(x); }, [=](int x) { return (int)dp.div(x); });
      });
  }
};

template <typename G0, typename G1> struct Ax2 {
  static constexpr bool kFixed = true;
  __device__ __forceinline__ explicit Ax2(const RbAxis&) {}
  static constexpr int N = G0::R * G1::R;
  static __host__ __device__ __forceinline__ constexpr int n() { return N; }
  static __host__ __device__ __forceinline__ constexpr int nst() { return 2; }
  static __host__ __device__ __forceinline__ constexpr int nbf() { return G1::R; }
  static __host__ __device__ __forceinline__ constexpr int nbl() { return G0::R; }
  static __host__ __device__ __forceinline__ constexpr int rl() { return G1::R; }
  static __device__ __forceinline__ int div_nbf(int x) { return (unsigned)x / (unsigned)nbf(); }
  static __device__ __forceinline__ int div_nbl(int x) { return (unsigned)x / (unsigned)nbl(); }
  template <typename F> __device__ __forceinline__ void first(F&& f) const { f(G0{}); }
  template <typename F> __device__ __forceinline__ void last(F&& f) const { f(G1{}); }
  template <typename F> __device__ __forceinline__ void middle(F&&) const {}
};

template <typename G0, typename G1, typename G2> struct Ax3 {
  static constexpr bool kFixed = true;
  __device__ __forceinline__ explicit Ax3(const RbAxis&) {}
  static constexpr int N = G0::R * G1::R * G2::R;
  static __host__ __device__ __forceinline__ constexpr int n() { return N; }
  static __host__ __device__ __forceinline__ constexpr int nst() { return 3; }
  static __host__ __device__ __forceinline__ constexpr int nbf() { return N / G0::R; }
  static __host__ __device__ __forceinline__ constexpr int nbl() { return N / G2::R; }
  static __host__ __device__ __forceinline__ constexpr int rl() { return G2::R; }
  static __device__ __forceinline__ int div_nbf(int x) { return (unsigned)x / (unsigned)nbf(); }
  static __device__ __forceinline__ int div_nbl(int x) { return (unsigned)x / (unsigned)nbl(); }
  template <typename F> __device__ __forceinline__ void first(F&& f) const { f(G0{}); }
  template <typename F> __device__ __forceinline__ void last(F&& f) const { f(G2{}); }
  template <typename F> __device__ __forceinline__ void middle(F&& f) const {
    f(G1{}, std::integral_constant<int, N / G1::R>{}, std::integral_constant<int, G0::R>{},
      [](int x) { return (int)((unsigned)x / (unsigned)(N / G1::R)); },
      [](int x) { return (int)((unsigned)x / (unsigned)G0::R); });
  }
};

// Butterfly i of a later stage from shared memory (element j at idx(j)),
// transformed in u.
template <int DIR, typename T, typename RC, typename IDX>
__device__ __forceinline__ void load_stage(RC rc, cpx<T>* u, const cpx<T>* __restrict__ s,
                                           const cpx<T>* __restrict__ tw, int i, int k, int nb, int p, int n, IDX idx) {
#pragma unroll
  for (int t = 0; t < RC::R; ++t) u[t] = s[idx(i + t * nb)];
  stage_next<DIR, T>(rc, u, tw, k, p, n);
}

}  // namespace gbrb
