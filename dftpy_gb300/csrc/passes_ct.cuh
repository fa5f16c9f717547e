// FP32 row passes of compile-time length for the plane pipeline and the delta
// evaluations, for the grid sizes of the workloads; a launcher returns 1 when the
// size has no specialisation, 0 on success, or an error.  Spectra are plane-major:
// element k2 of row r at k2 * nrows + r, consecutive threads on consecutive rows of
// one k2.
#pragma once
#include <math.h>
#include <string.h>
#include <type_traits>

#include "fft_ct.cuh"
#include "gkernels.cuh"
#include "pass_common.cuh"
#include "plan.h"

namespace gbct {

template <typename F>
__host__ inline bool ct_dispatch(int n, F&& f) {
  switch (n) {
    case 32: f(std::integral_constant<int, 32>{}); return true;
    case 64: f(std::integral_constant<int, 64>{}); return true;
    case 96: f(std::integral_constant<int, 96>{}); return true;
    case 128: f(std::integral_constant<int, 128>{}); return true;
    case 160: f(std::integral_constant<int, 160>{}); return true;
    case 256: f(std::integral_constant<int, 256>{}); return true;
    case 360: f(std::integral_constant<int, 360>{}); return true;
    default: return false;
  }
}

// Launch-shape parameters (overridable at build time for tuning sweeps)
#ifndef GB_CT_RP_F32
#define GB_CT_RP_F32 4
#endif
#ifndef GB_CT_ROWS_MINB
#define GB_CT_ROWS_MINB 1
#endif
#ifndef GB_CT_PF_F32
#define GB_CT_PF_F32 4      // density / v_loc values prefetched per thread in the FP32 evaluation epilogue (measured best)
#endif

constexpr int kRowPairs = GB_CT_RP_F32;         // row pairs per CTA (per field)
// threads of a row-pass CTA: TPL per line, one line per (field, row pair)
template <int N> constexpr int rows_threads_max() { return Tpl<N>::value * kRowPairs * GB_MAX_FIELDS; }

// ---- pointwise functions -----------------------------------------------------
// x^(1/2), x^(5/6) and friends for x >= 1e-30 (the reference's clamps)
__device__ __forceinline__ float sqrt_pos(float x) { return x * rsqrtf(x); }

__device__ __forceinline__ float pow_beta_ct(float x, bool b56, float beta) {
  if (b56) {
    const float z3 = rcbrtf(x), z2 = rsqrtf(x);
    return (x * z2) * (x * z3 * z3);         // x^(1/2) x^(1/3)
  }
  return powf(x, beta);
}

__device__ __forceinline__ float prologue_ct(int op, float rho, bool b56, float beta) {
  if (op == OP_SQRT) return sqrt_pos(rho > 0.0f ? rho : (float)kZero);
  if (op == OP_POWB) return pow_beta_ct(rho < (float)kZero ? (float)kZero : rho, b56, beta);
  return rho;
}

// ---- rows forward ---------------------------------------------------------------
// One CTA: RP row pairs of the input, all nf derived fields transformed at
// once (line = field * RP + pair; TPL threads per line).
struct CtRowsFwd {
  const void* in;
  void* out;
  int64_t fstride;
  int nrows, nf;
  int op[GB_MAX_FIELDS];
  int b56;            // beta == 5/6
  Sc beta;
  const void* tw;
};

template <int N>
__global__ void __launch_bounds__(rows_threads_max<N>(), GB_CT_ROWS_MINB) k_ct_rows_fwd(CtRowsFwd a) {
  constexpr int RP = kRowPairs, TPL = Tpl<N>::value, NP = Pad<float, N>::NP, NH = N / 2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nl = a.nf * RP;
  cpx<float>* tw = reinterpret_cast<cpx<float>*>(smem_raw);
  cpx<float>* A = tw + N;
  cpx<float>* B = A + nl * NP;
  float* R = reinterpret_cast<float*>(B + nl * NP);      // [2 RP][N] real input rows
  const int tid = threadIdx.x, l = tid / TPL, lane = tid % TPL;
  const int64_t base = (int64_t)blockIdx.x * 2 * RP;
  const cpx<float>* twg = reinterpret_cast<const cpx<float>*>(a.tw);
  for (int i = tid; i < N; i += blockDim.x) tw[i] = twg[i];
  const float* in = reinterpret_cast<const float*>(a.in);
  // input rows: batches of independent loads ahead of their stores
  constexpr int NE = 2 * RP * N, UNR = 4;
#pragma unroll 1
  for (int b0 = 0; b0 < NE; b0 += UNR * (int)blockDim.x) {
    float v[UNR];
#pragma unroll
    for (int u = 0; u < UNR; ++u) {
      const int idx = b0 + u * (int)blockDim.x + tid;
      const int64_t row = base + idx / N;
      v[u] = (idx < NE && row < a.nrows) ? __ldg(in + row * N + idx % N) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < UNR; ++u) {
      const int idx = b0 + u * (int)blockDim.x + tid;
      if (idx < NE) R[idx] = v[u];
    }
  }
  __syncthreads();
  const bool b56 = a.b56 != 0;
  const float beta = sc<float>(a.beta);
  // fields in an unrolled outer loop: the field's prologue op is a
  // compile-time parameter index, and every index split below is by a
  // compile-time constant
#pragma unroll
  for (int f = 0; f < GB_MAX_FIELDS; ++f) {
    if (f >= a.nf) break;
    const int op = a.op[f];
    for (int idx = tid; idx < RP * N; idx += blockDim.x) {
      const int l2 = idx / N, j = idx % N;
      const int64_t ra = base + 2 * l2;
      const float x0 = ra < a.nrows ? prologue_ct(op, R[(2 * l2) * N + j], b56, beta) : 0.0f;
      const float x1 = ra + 1 < a.nrows ? prologue_ct(op, R[(2 * l2 + 1) * N + j], b56, beta) : 0.0f;
      A[sw<float, NP>(f * RP + l2, j)] = cpx<float>{x0, x1};
    }
  }
  __syncthreads();
  cpx<float>* res = fft<-1, float, N>(A, B, tw, l, lane, true);
  cpx<float>* out = reinterpret_cast<cpx<float>*>(a.out);
#pragma unroll
  for (int f = 0; f < GB_MAX_FIELDS; ++f) {
    if (f >= a.nf) break;
    cpx<float>* o = out + f * a.fstride;
    for (int idx = tid; idx < RP * NH; idx += blockDim.x) {
      const int l2 = idx % RP, k = idx / RP;
      const int line = f * RP + l2;
      const int64_t ra = base + 2 * l2, rb = ra + 1;
      if (ra >= a.nrows) continue;
      const cpx<float> Z = res[sw<float, NP>(line, k)];
      const cpx<float> Zc = res[sw<float, NP>(line, k == 0 ? 0 : N - k)];
      const int64_t ia = (int64_t)k * a.nrows + ra;
      o[ia] = cpx<float>{(Z.x + Zc.x) * 0.5f, (Z.y - Zc.y) * 0.5f};
      if (rb < a.nrows) o[ia + 1] = cpx<float>{(Z.y + Zc.y) * 0.5f, (Zc.x - Z.x) * 0.5f};
    }
  }
}

// ---- rows inverse ----------------------------------------------------------------
struct CtRowsInv {
  const void* in;
  int64_t fstride;
  int nrows, nf;
  const void* tw;
  void* out;
  int64_t ostride;
  EvalDesc ev;
  Sc tf_v, tf_e, vw_y, two_alpha, inv_two_alpha, wt_beta;  // evaluation constants
  int b56;
  const void* rho;
  const void* vloc;
  void* pot;
  double* partials;
  int calc_e;
};

// irfftn line build (all fields) + inverse FFT; result line (f * RP + pair)
// holds row 2 pair in .x and row 2 pair + 1 in .y.
template <int N>
__device__ __forceinline__ cpx<float>* ct_rows_inv_lines(const CtRowsInv& a, int64_t base, cpx<float>* tw,
                                                         cpx<float>* A, cpx<float>* B) {
  constexpr int RP = kRowPairs, TPL = Tpl<N>::value, NP = Pad<float, N>::NP, NH = N / 2 + 1;
  const int tid = threadIdx.x, l = tid / TPL, lane = tid % TPL;
  const int nl = a.nf * RP;
  const cpx<float>* src0 = reinterpret_cast<const cpx<float>*>(a.in);
#pragma unroll
  for (int f = 0; f < GB_MAX_FIELDS; ++f) {
    if (f >= a.nf) break;
    const cpx<float>* src = src0 + f * a.fstride;
    for (int idx = tid; idx < RP * NH; idx += blockDim.x) {
      const int l2 = idx % RP, k = idx / RP;
      const int line = f * RP + l2;
      const int64_t ra = base + 2 * l2, rb = ra + 1;
      const int64_t ia = (int64_t)k * a.nrows + ra;
      cpx<float> va = {0.0f, 0.0f}, vb = {0.0f, 0.0f};
      if (ra < a.nrows) va = src[ia];
      if (rb < a.nrows) vb = src[ia + 1];
      if (k == 0 || 2 * k == N) { va.y = 0.0f; vb.y = 0.0f; }
      A[sw<float, NP>(line, k)] = cpx<float>{va.x - vb.y, va.y + vb.x};
      if (k > 0 && 2 * k < N) A[sw<float, NP>(line, N - k)] = cpx<float>{va.x + vb.y, vb.x - va.y};
    }
  }
  __syncthreads();
  return fft<1, float, N>(A, B, tw, l, lane, true);
}

template <int N>
__global__ void __launch_bounds__(rows_threads_max<N>()) k_ct_rows_inv_store(CtRowsInv a) {
  constexpr int RP = kRowPairs, NP = Pad<float, N>::NP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nl = a.nf * RP;
  cpx<float>* tw = reinterpret_cast<cpx<float>*>(smem_raw);
  cpx<float>* A = tw + N;
  cpx<float>* B = A + nl * NP;
  const int tid = threadIdx.x;
  const int64_t base = (int64_t)blockIdx.x * 2 * RP;
  const cpx<float>* twg = reinterpret_cast<const cpx<float>*>(a.tw);
  for (int i = tid; i < N; i += blockDim.x) tw[i] = twg[i];
  cpx<float>* res = ct_rows_inv_lines<N>(a, base, tw, A, B);
  float* out = reinterpret_cast<float*>(a.out);
  for (int idx = tid; idx < a.nf * 2 * RP * N; idx += blockDim.x) {
    const int f = idx / (2 * RP * N), r = idx % (2 * RP * N);
    const int rr = r / N, j = r % N;
    const int64_t row = base + rr;
    if (row >= a.nrows) continue;
    const cpx<float> z = res[sw<float, NP>(f * RP + (rr >> 1), j)];
    out[f * a.ostride + row * N + j] = (rr & 1) ? z.y : z.x;
  }
}

template <typename T>
__device__ __forceinline__ void pz_lda_ct(T rho, T& eps, T& pot, bool want_e) {
  const T a = (T)0.0311, b = (T)-0.048, c = (T)0.0020, d = (T)-0.0116;
  const T g = (T)-0.1423, b1 = (T)1.0529, b2 = (T)0.3334;
  const T cx = (T)0.98474502184269654115;                 // (3/pi)^(1/3)
  T rc, inv_rc;                                             // rho^(1/3), clamped at 1e-30
  if (rho > (T)kZero) {
    inv_rc = rcbrt_d(rho);
    rc = rho * inv_rc * inv_rc;
  } else {
    rc = cbrt(rho);
    if (rc < (T)kZero) rc = (T)kZero;
    inv_rc = (T)1 / rc;
  }
  const T rs = (T)0.62035049089940001667 * inv_rc;        // (3/(4 pi))^(1/3) / rho^(1/3)
  pot = -cx * rc;
  eps = (T)(-0.75) * cx * rc;
  if (rs < (T)1) {
    const T lr = log(rs);
    pot += lr * (a + (T)(2.0 / 3.0) * c * rs) + b - (T)(1.0 / 3.0) * a + (T)(1.0 / 3.0) * ((T)2 * d - c) * rs;
    if (want_e) eps += a * lr + b + c * rs * lr + d * rs;
  } else {
    const T sq = rs * rsqrt_d(rs);
    const T inv = (T)1 / ((T)1 + b1 * sq + b2 * rs);
    pot += (g + ((T)(7.0 / 6.0) * g * b1) * sq + ((T)(4.0 / 3.0) * g * b2 * rs)) * inv * inv;
    if (want_e) eps += g * inv;
  }
}

// WANT_E is a template parameter so the potential-only instantiation holds no
// FP64 accumulation at all (if-converted, never-taken FP64 code still
// occupies the FP64 pipe).
template <int N, bool WANT_E>
__global__ void __launch_bounds__(rows_threads_max<N>(), GB_CT_ROWS_MINB) k_ct_rows_inv_eval(CtRowsInv a) {
  constexpr int RP = kRowPairs, NP = Pad<float, N>::NP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nl = (a.nf > 0 ? a.nf : 1) * RP;
  cpx<float>* tw = reinterpret_cast<cpx<float>*>(smem_raw);
  cpx<float>* A = tw + N;
  cpx<float>* B = A + nl * NP;
  const int tid = threadIdx.x;
  const int64_t base = (int64_t)blockIdx.x * 2 * RP;
  const cpx<float>* twg = reinterpret_cast<const cpx<float>*>(a.tw);
  for (int i = tid; i < N; i += blockDim.x) tw[i] = twg[i];
  const EvalDesc& ev = a.ev;
  const float* rhop = reinterpret_cast<const float*>(a.rho);
  const float* vlocp = reinterpret_cast<const float*>(a.vloc);
  // the density and v_loc of this thread's first PF elements, loaded before
  // the transforms so their latency is hidden behind them
  constexpr int PF = GB_CT_PF_F32;
  float pre_rho[PF], pre_vl[PF];
#pragma unroll
  for (int m = 0; m < PF; ++m) {
    const int idx = tid + m * (int)blockDim.x;
    const int64_t row = base + idx / N;
    const bool ok = idx < 2 * RP * N && row < a.nrows;
    const int64_t gidx = row * N + idx % N;
    pre_rho[m] = ok ? __ldg(rhop + gidx) : 0.0f;
    pre_vl[m] = (ok && ev.pp) ? __ldg(vlocp + gidx) : 0.0f;
  }
  cpx<float>* res = A;
  if (a.nf > 0) res = ct_rows_inv_lines<N>(a, base, tw, A, B);
  float* potp = reinterpret_cast<float*>(a.pot);
  constexpr bool want_e = WANT_E;
  const float tf_v = sc<float>(a.tf_v);             // (5/3) C_TF x
  const float tf_e = sc<float>(a.tf_e);             // C_TF x
  const float vw_y = sc<float>(a.vw_y);
  const float two_alpha = sc<float>(a.two_alpha);
  const float inv_two_alpha = sc<float>(a.inv_two_alpha);
  const float wt_beta = sc<float>(a.wt_beta);
  const bool b56 = a.b56 != 0;
  // per-thread energy sums in the field precision (a handful of elements per
  // thread); combined in FP64 across threads and CTAs
  float es[6] = {0, 0, 0, 0, 0, 0};
  auto point = [&](int idx, float rho, float vl_pre) {
    const int rr = idx / N, j = idx % N;
    const int64_t row = base + rr;
    if (row >= a.nrows) return;
    const int64_t gidx = row * N + j;
    const int pr = rr >> 1;
    const bool odd = rr & 1;
    const bool pos = rho > (float)kZero;
    // rho^(-1/3) and rho^(-1/2) for positive densities (shared by TF, vW, WT)
    float z3 = 0.0f, z2 = 0.0f;
    if (pos) { z3 = rcbrt_d(rho); z2 = rsqrt_d(rho); }
    float pot = 0.0f;
    if (ev.tf) {
      float r23;                                              // cbrt(rho^2)
      if (pos) r23 = rho * z3;
      else r23 = cbrt(rho * rho);
      pot += tf_v * r23;
      if (want_e) {
        float r53;                                            // cbrt(rho^5)
        if (pos) r53 = rho * rho * z3;
        else { float r5 = rho * rho; r5 = r5 * rho; r5 = r5 * rho; r5 = r5 * rho; r53 = cbrt(r5); }
        es[0] += r53 * tf_e;
      }
    }
    if (ev.vw) {
      const cpx<float> zz = res[sw<float, NP>(ev.slot_vw * RP + pr, j)];
      const float w = odd ? zz.y : zz.x;
      // 1 / max(sqrt(rho_m), 1e-30), rho_m = rho if rho > 0 else 1e-30
      const float inv_sq = pos ? z2 : (rho > 0.0f ? 1.0f / fmax(sqrt(rho), (float)kZero) : 1e15f);
      const float v = 0.5f * w * inv_sq;
      pot += v * vw_y;
      if (want_e && rho > 0.0f) es[1] += rho * v * vw_y;
    }
    if (ev.wt) {
      const cpx<float> zz = res[sw<float, NP>(ev.slot_wt * RP + pr, j)];
      const float kc = odd ? zz.y : zz.x;
      float rb_over_rc;                                       // rc^(beta - 1), rc = max(rho, 1e-30)
      if (b56) {
        if (pos) rb_over_rc = rho * z3 * z3 * z2;          // rho^(1/3) rho^(-1/2)
        else { const float rc = (float)kZero; rb_over_rc = sqrt(rc) * cbrt(rc) / rc; }
      } else {
        const float rc = rho < (float)kZero ? (float)kZero : rho;
        rb_over_rc = pow(rc, wt_beta) / rc;
      }
      const float v = two_alpha * rb_over_rc * kc;
      pot += v;
      if (want_e) es[2] += v * rho * inv_two_alpha;
    }
    if (ev.xc) {
      float eps, vx;
      pz_lda_ct<float>(rho, eps, vx, want_e);
      pot += vx;
      if (want_e) es[3] += eps * rho;
    }
    if (ev.hartree) {
      const cpx<float> zz = res[sw<float, NP>(ev.slot_h * RP + pr, j)];
      const float vh = odd ? zz.y : zz.x;
      pot += vh;
      if (want_e) es[4] += 0.5f * vh * rho;
    }
    if (ev.pp) {
      const float vl = vl_pre;
      pot += vl;
      if (want_e) es[5] += vl * rho;
    }
    potp[gidx] = pot;
  };
  // one element per iteration (not unrolled: an unrolled epilogue doubles the
  // registers and halves the occupancy); the first PF come from the
  // prefetch registers
#pragma unroll 1
  for (int m = 0, idx = tid; idx < 2 * RP * N; ++m, idx += blockDim.x) {
    float rho, vl;
    if (m < PF) {
#pragma unroll
      for (int q = 0; q < PF; ++q)
        if (q == m) { rho = pre_rho[q]; vl = pre_vl[q]; }
    } else {
      const int64_t row = base + idx / N;
      if (row >= a.nrows) continue;
      const int64_t gidx = row * N + idx % N;
      rho = __ldg(rhop + gidx);
      vl = ev.pp ? __ldg(vlocp + gidx) : 0.0f;
    }
    point(idx, rho, vl);
  }
  if constexpr (!WANT_E) return;
  __shared__ double red[32][6];
  const int lane32 = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const double v = warp_sum((double)es[c]);
    if (lane32 == 0) red[warp][c] = v;
  }
  __syncthreads();
  if (tid < 6) {
    KSum s;
    s.init();
    const int nw = (blockDim.x + 31) >> 5;
    for (int w = 0; w < nw; ++w) s.add(red[w][tid]);
    a.partials[(int64_t)blockIdx.x * GB_NE + tid] = s.value();
  }
}

// reciprocal-space kernel value, out of line
template <typename T>
__device__ __noinline__ float kernel_value_slow(const GInfo& g, int type, const void* arr, int i0, int i1, int k2) {
  return gbk::kernel_value<T>(g, type, arr, i0, i1, k2);
}

// ---- launchers -------------------------------------------------------------------
inline int ct_rows_fwd(gbofdft_plan* p, const void* in, void* spec, int64_t fstride, int nf, const int* ops, double beta,
                       cudaStream_t st) {
  int rc = 1;
  ct_dispatch(p->n[2], [&](auto nc) {
    constexpr int N = decltype(nc)::value;
    constexpr int RP = kRowPairs, NP = Pad<float, N>::NP;
    CtRowsFwd a;
    a.in = in; a.out = spec; a.fstride = fstride;
    a.nrows = p->n[0] * p->n[1]; a.nf = nf;
    for (int f = 0; f < GB_MAX_FIELDS; ++f) a.op[f] = f < nf ? ops[f] : OP_RHO;
    a.b56 = fabs(beta - 5.0 / 6.0) < 1e-15;
    a.beta.set(beta);
    a.tw = p->tw[2];
    const size_t sm = sizeof(cpx<float>) * (N + 2 * (size_t)nf * RP * NP) + sizeof(float) * 2 * RP * N;
    if ((rc = ct_smem(k_ct_rows_fwd<N>, sm))) return;
    const int nblk = (a.nrows + 2 * RP - 1) / (2 * RP);
    k_ct_rows_fwd<N><<<nblk, Tpl<N>::value * RP * nf, sm, st>>>(a);
    gb_count_launch();
    cudaError_t e = cudaGetLastError();
    rc = e == cudaSuccess ? 0 : gb_set_error(GBOFDFT_ERR_CUDA, "ct_rows_fwd: %s", cudaGetErrorString(e));
  });
  return rc;
}

inline int ct_rows_inv(gbofdft_plan* p, const void* spec, int64_t fstride, int nf, void* out, int64_t ostride,
                       const EvalDesc* ev, const void* rho, const void* vloc, void* pot, int calc_e,
                       double* partials, int64_t* nblk_out, cudaStream_t st) {
  int rc = 1;
  ct_dispatch(p->n[2], [&](auto nc) {
    constexpr int N = decltype(nc)::value;
    constexpr int RP = kRowPairs, NP = Pad<float, N>::NP;
    CtRowsInv a;
    memset(&a, 0, sizeof(a));
    a.in = spec; a.fstride = fstride; a.nrows = p->n[0] * p->n[1]; a.nf = nf; a.tw = p->tw[2];
    a.out = out; a.ostride = ostride;
    const int nblk = (a.nrows + 2 * RP - 1) / (2 * RP);
    if (nblk_out) *nblk_out = nblk;
    if (ev) {
      a.ev = *ev; a.rho = rho; a.vloc = vloc; a.pot = pot; a.calc_e = calc_e; a.partials = partials;
      const double ctf = 2.87123400018819181594;    // (3/10)(3 pi^2)^(2/3)
      a.tf_v.set(5.0 / 3.0 * ctf * ev->tf_x);
      a.tf_e.set(ctf * ev->tf_x);
      a.vw_y.set(ev->vw_y);
      a.two_alpha.set(2.0 * ev->wt_alpha);
      a.inv_two_alpha.set(ev->wt_alpha != 0.0 ? 1.0 / (2.0 * ev->wt_alpha) : 0.0);
      a.wt_beta.set(ev->wt_beta);
      a.b56 = fabs(ev->wt_beta - 5.0 / 6.0) < 1e-15;
      const int nfl = nf > 0 ? nf : 1;
      const size_t sm = sizeof(cpx<float>) * (N + 2 * (size_t)nfl * RP * NP);
      if (calc_e) {
        if ((rc = ct_smem(k_ct_rows_inv_eval<N, true>, sm))) return;
        k_ct_rows_inv_eval<N, true><<<nblk, Tpl<N>::value * RP * nfl, sm, st>>>(a);
      } else {
        if ((rc = ct_smem(k_ct_rows_inv_eval<N, false>, sm))) return;
        k_ct_rows_inv_eval<N, false><<<nblk, Tpl<N>::value * RP * nfl, sm, st>>>(a);
      }
    } else {
      const size_t sm = sizeof(cpx<float>) * (N + 2 * (size_t)nf * RP * NP);
      if ((rc = ct_smem(k_ct_rows_inv_store<N>, sm))) return;
      k_ct_rows_inv_store<N><<<nblk, Tpl<N>::value * RP * nf, sm, st>>>(a);
    }
    gb_count_launch();
    cudaError_t e = cudaGetLastError();
    rc = e == cudaSuccess ? 0 : gb_set_error(GBOFDFT_ERR_CUDA, "ct_rows_inv: %s", cudaGetErrorString(e));
  });
  return rc;
}

}  // namespace gbct

#include "plane_ct.cuh"

namespace gbct {

// Plane convolution pass over plane-major spectra (FP32); returns 1 when the
// plane sizes have no specialisation or do not fit in shared memory.
inline int plane_conv_f32(gbofdft_plan* p, void* spec, int64_t fstride, int nf, const KerDesc& kd,
                          const float* const* pm_arr, double scale, cudaStream_t st) {
  int rc = 1;
  plane_dispatch(p->n[0], p->n[1], [&](auto a0, auto a1) {
    constexpr int N0 = decltype(a0)::value, N1 = decltype(a1)::value;
    PlaneArgs a;
    memset(&a, 0, sizeof(a));
    a.spec = reinterpret_cast<float2*>(spec);
    a.fstride = fstride;
    a.tw0 = p->tw[0];
    a.tw1 = p->tw[1];
    a.gi = p->gi;
    for (int i = 0; i < 9; ++i) a.bgf[i] = (float)p->bg[i];
    for (int f = 0; f < GB_MAX_FIELDS; ++f) {
      a.type[f] = f < nf ? kd.type[f] : KER_NONE;
      a.arr[f] = (f < nf && kd.type[f] == KER_ARRAY) ? pm_arr[f] : nullptr;
      a.coef[f] = (float)(kd.coef[f] * scale);
    }
    for (int f = 0; f < nf; ++f)
      if (a.type[f] == KER_ARRAY && !a.arr[f]) {
        rc = gb_set_error(GBOFDFT_ERR_ARG, "plane_conv: field %d has no plane-major kernel table", f);
        return;
      }
    const size_t sm = PlaneCfg<N0, N1>::kSmem;
    auto launch = [&](auto kern) {
      if ((rc = ct_smem(kern, sm))) return;
      kern<<<dim3(p->n2h, nf), PlaneCfg<N0, N1>::NT, sm, st>>>(a);
    };
    if constexpr (plane_variants<N0, N1>() > 1) {
      if (p->plane_variant == 1) launch(k_plane_conv<N0, N1, 1>);
      else launch(k_plane_conv<N0, N1, 0>);
    } else {
      launch(k_plane_conv<N0, N1, 0>);
    }
    if (rc) return;
    gb_count_launch();
    cudaError_t e = cudaGetLastError();
    rc = e == cudaSuccess ? 0 : gb_set_error(GBOFDFT_ERR_CUDA, "plane_conv: %s", cudaGetErrorString(e));
  });
  return rc;
}

}  // namespace gbct

// Plane-major evaluation pipeline (FP32 only).
#define GB_CT_DEFINE_PLANE()                                                                                   \
  int gb_ct_rows_fwd_pm_f32(gbofdft_plan* p, const void* in, void* spec, int64_t fstride, int nf,             \
                            const int* ops, double beta, cudaStream_t st) {                                   \
    return gbct::ct_rows_fwd(p, in, spec, fstride, nf, ops, beta, st);                   \
  }                                                                                                            \
  int gb_ct_rows_inv_eval_pm_f32(gbofdft_plan* p, const void* spec, int64_t fstride, int nf,                  \
                                 const EvalDesc* ev, const void* rho, const void* vloc, void* pot, int calc_e,  \
                                 double* partials, int64_t* nblk, cudaStream_t st) {                           \
    return gbct::ct_rows_inv(p, spec, fstride, nf, nullptr, 0, ev, rho, vloc, pot, calc_e, partials, nblk, st); \
  }                                                                                                            \
  int gb_plane_conv_f32(gbofdft_plan* p, void* spec, int64_t fstride, int nf, const KerDesc* kd,               \
                        const float* const* pm_arr, double scale, cudaStream_t st) {                          \
    return gbct::plane_conv_f32(p, spec, fstride, nf, *kd, pm_arr, scale, st);                                \
  }                                                                                                            \
  int gb_ct_rows_inv_store_pm_f32(gbofdft_plan* p, const void* spec, int64_t fstride, int nf, void* out,       \
                                  int64_t ostride, cudaStream_t st) {                                          \
    return gbct::ct_rows_inv(p, spec, fstride, nf, out, ostride, nullptr, nullptr, nullptr, nullptr, 0,        \
                             nullptr, nullptr, st);                                                            \
  }                                                                                                            \
  int gb_plane_supported_f32(int n0, int n1, int n2) {                                                         \
    bool rows = gbct::ct_dispatch(n2, [](auto) {});                                                            \
    bool plane = gbct::plane_dispatch(n0, n1, [](auto, auto) {});                                              \
    return rows && plane;                                                                                      \
  }                                                                                                            \
  int gb_plane_variants_f32(int n0, int n1) {                                                                  \
    int nv = 0;                                                                                                \
    gbct::plane_dispatch(n0, n1, [&](auto a0, auto a1) {                                                       \
      nv = gbct::plane_variants<decltype(a0)::value, decltype(a1)::value>();                                   \
    });                                                                                                        \
    return nv;                                                                                                 \
  }
