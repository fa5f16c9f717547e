// Host-side plan: grid geometry, FFT schedules, device tables and workspaces.
#pragma once
#include "common.cuh"
#include "rb_axis.h"

struct GInfo {           // reciprocal-space geometry passed to kernels by value
  double bg[9];          // reciprocal lattice vectors, rows (2 pi inv(L)^T)
  int n0, n1, n2, n2h, ld2;
  int full;              // 1: full-grid G convention (fftfreq on every axis)
};

struct gbofdft_plan {
  int n[3];
  int n2h;               // n2 / 2 + 1
  int ld2;               // row pitch of internal spectra (complex elements)
  int full;
  int prec;              // GBOFDFT_F32 / GBOFDFT_F64
  int device;
  double lattice[9];
  double bg[9];
  double volume, dV;
  int64_t N;             // n0 n1 n2
  int64_t NG;            // n0 n1 n2h (API spectrum size)
  int64_t NGld;          // n0 n1 ld2 (internal spectrum size)
  AxisPlan ax[3];
  gbrb::RbAxis rb[3], rbi[3];   // register-blocked passes: radices in stage order, and the other way round
  void* tw[3];           // device twiddle tables, complex<prec>[n_axis]
  void* spec;            // GB_MAX_FIELDS internal spectra
  double* partials;      // per-CTA energy partial sums
  int64_t max_partials;  // rows of GB_NE doubles
  double* scratch;       // small device scratch (reductions), 4096 doubles
  int tb[3];             // column tile width per axis
  int pairs;             // row pairs per CTA in the row passes
  GInfo gi;
  // FP32 plane-major evaluation pipeline (rows -> plane convolution -> rows)
  int plane;             // 1: the grid has the plane pipeline (and uses it)
  int plane_ok;          // 1: the grid has a plane specialisation
  int plane_variant;     // radix-schedule variant of the plane pass (autotuned)
  float* wt_pm;          // plane-major copy of the last WT kernel table built on this plan
  const void* wt_pm_src; // the table that copy belongs to
  // the buffers the last two TN preconditioners were built into and their
  // mean densities (a rebuild is skipped when both match): the FP32 stage
  // and the refinement's Hessian products keep one each on the same plan
  const void* precond_buf[2];
  double precond_rho0[2];
  int precond_next;         // slot the next build replaces
  float* precond_pm;        // FP32 plane-pipeline plans: plane-major copy of one preconditioner ...
  const void* precond_pm_src;  // ... the one built into this buffer
  int plane_precond;        // 1: preconditioner convolutions through the plane pipeline
};

size_t gb_elem(const gbofdft_plan* p);  // bytes per real scalar
// zero-initialised grid-reduction ticket in the plan's scratch (last double;
// scratch[0..4094] are free for per-CTA partial sums)
unsigned* gb_plan_counter(gbofdft_plan* p);

// ---- pass launchers (passes.cu) -------------------------------------------
// forward prologues; OP_WGC0..2: rho^e u^k (k = 0, 1, 2) of the WGC term,
// u = (rho - rho0) / rho0, exponent e in the beta argument
enum { OP_RHO = 0, OP_SQRT = 1, OP_POWB = 2, OP_WGC0 = 3, OP_WGC1 = 4, OP_WGC2 = 5 };
enum { KER_NONE = 0, KER_HARTREE = 1, KER_G2 = 2, KER_ARRAY = 3 };

struct EvalDesc {
  int tf, vw, wt, xc, hartree, pp;
  int slot_h, slot_vw, slot_wt;   // field slot of each convolution output
  double tf_x, vw_y, wt_alpha, wt_beta;
  double e_ion;
  // optional (FP64 register-blocked passes only): the convolution results
  // before the pointwise epilogue, field slot f at cout + f * cstride
  void* cout;
  int64_t cstride;
};

struct KerDesc {
  int type[GB_MAX_FIELDS];
  const void* arr[GB_MAX_FIELDS];
  double coef[GB_MAX_FIELDS];
};

int gb_rows_fwd(gbofdft_plan* p, const void* in, void* spec, int64_t fstride, int ld2, int nf,
                const int* ops, double beta, double scale, cudaStream_t st);
int gb_rows_inv_store(gbofdft_plan* p, const void* spec, int64_t fstride, int ld2, int nf,
                      void* out, int64_t ostride, double scale, cudaStream_t st);
int gb_rows_inv_eval(gbofdft_plan* p, const void* spec, int64_t fstride, int nf, const EvalDesc& ev,
                     const void* rho, const void* vloc, void* pot, int calc_e, double* energies,
                     cudaStream_t st);
int gb_cols(gbofdft_plan* p, void* spec, int64_t fstride, int ld2, int nf, int axis, int dir,
            double scale, cudaStream_t st);
int gb_cols_conv(gbofdft_plan* p, void* spec, int64_t fstride, int ld2, int nf, const KerDesc& kd,
                 double scale, cudaStream_t st);
// register-blocked passes (passes_rb_*.cu): return 1 when the axis length has a
// prime factor above 7 or its lines do not fit, 0 on success, an error code otherwise
#define GB_RB_FIELDS 10   // fused terms (GB_MAX_FIELDS - 1) and the six fields of the WGC term
#define GB_LWT_BATCH 4     // knots of one launch, at most
// The knot intervals of the knots k0 .. k0 + m - 1 of a LWT batch: interval e
// (lo, hi) lies left of knot k0 + e; lo = HUGE_VAL: none there.  below: k0 is the
// first knot, and its weight also holds (kf - kl) / kl at kf < kl_e.
struct LwtKnots {
  int m, below;
  double lo[GB_LWT_BATCH + 1], hi[GB_LWT_BATCH + 1], inv[GB_LWT_BATCH + 1];
  double kl, kl_e, inv_kl;
};
struct RbLwt {            // LWT columns along axis 0
  const void* in[GB_RB_FIELDS];   // inverse: in[0] = S for every field; accumulation: field f
  void* out[GB_RB_FIELDS];        // inverse: field f; accumulation: out[0] (+)= sum_f K_f in[f]
  const void* K[GB_RB_FIELDS];    // kernel fields [n0][n1][n2h]
  int nf, ld2, dir, first;
};
struct RbLwtRows {        // LWT rows of a batch of knots
  const LwtKnots* knots;
  const void* kf;         // k_F
  int ld2;
  // inverse: spectra p_i (0 .. m - 1) and, with out3, those of the derivative kernels (m .. 2 m - 1):
  // out1, out3 (+)= weights x fields
  const void* in[GB_RB_FIELDS];
  void *out1, *out3;
  int first;
  // forward: spectra of the weights times ra, scaled by scale
  const void* ra;
  void* out[GB_RB_FIELDS];
  double scale;
};
struct RbFwd {            // forward rows: fields derived from in[0] (OP_RHO alone: in[f]) to spectra out[f]
  const void* in[GB_RB_FIELDS];
  void* out[GB_RB_FIELDS];
  int nf, ld2;
  int op[GB_RB_FIELDS];
  double beta, scale, rho0;
  // OP_WGC0..2 on FP64 plans: store rho^beta (and rho^beta2), or take rho^beta from pw_in
  double beta2;
  void *pw_out, *pw2_out;
  const void* pw_in;
};
struct RbInv {            // inverse rows: store real fields (ev null) or the evaluation epilogue
  const void* in[GB_RB_FIELDS];
  int nf, ld2;
  void* out;
  int64_t ostride;
  double scale;
  const EvalDesc* ev;
  const void *rho, *vloc;
  void* pot;
  int calc_e, add;        // add: to pot
  double* partials;       // GB_NE doubles per CTA
  const gbofdft_wgc* wgc; // the WGC term from the fields wslot ...
  int wslot, two;
  const void *pa, *pb;    // FP64: rho^alpha and rho^beta
  void* wstore[6];        // with vstore: copies of its fields and potential
  void* vstore;
};
struct RbCols {           // columns of nf spectra: dir, the convolution (kd) or the WGC term (K)
  void* data[GB_RB_FIELDS];
  int nf, ld2, axis, dir;
  double scale;
  const KerDesc* kd;
  const void* K;
  const void* src;        // dir 1, nf = 1: the field is read from here (row pitch src_ld)
  int src_ld;
};
#define GB_RB_DECLARE(SUF)                                                                \
  int gb_rb_rows_fwd_##SUF(gbofdft_plan*, const RbFwd&, cudaStream_t);                    \
  int gb_rb_rows_inv_##SUF(gbofdft_plan*, const RbInv&, int64_t* nblk, cudaStream_t);     \
  int gb_rb_cols_##SUF(gbofdft_plan*, const RbCols&, cudaStream_t);                       \
  int gb_rb_wgc_##SUF(gbofdft_plan*, const RbCols&, cudaStream_t);                        \
  int gb_rb_lwt_##SUF(gbofdft_plan*, const RbLwt&, cudaStream_t);                         \
  int gb_rb_lwt_rows_##SUF(gbofdft_plan*, const RbLwtRows&, cudaStream_t);
GB_RB_DECLARE(f64_g0)
GB_RB_DECLARE(f32_g0)
GB_RB_DECLARE(f32_g1)
GB_RB_DECLARE(f32_g2)
GB_RB_DECLARE(f32_g3)
GB_RB_DECLARE(f32_g4)
#undef GB_RB_DECLARE
int gb_rb_rows_fwd(gbofdft_plan*, const RbFwd&, cudaStream_t);
int gb_rb_rows_inv(gbofdft_plan*, const RbInv&, int64_t* nblk, cudaStream_t);
int gb_rb_cols(gbofdft_plan*, const RbCols&, cudaStream_t);
int gb_rb_wgc(gbofdft_plan*, const RbCols&, cudaStream_t);
int gb_rb_lwt(gbofdft_plan*, const RbLwt&, cudaStream_t);
int gb_rb_lwt_rows(gbofdft_plan*, const RbLwtRows&, cudaStream_t);
// every axis has register-blocked passes, the WGC columns included
bool gb_rb_wgc_ok(const gbofdft_plan* p);
void gb_rb_plan(gbofdft_plan* p);   // the plan's rb / rbi from its lengths and precision
// plane-major FP32 pipeline (passes_ct_f32.cu): return 1 when the size has no
// specialisation, 0 on success, an error code otherwise
int gb_ct_rows_fwd_pm_f32(gbofdft_plan*, const void*, void*, int64_t, int, const int*, double, cudaStream_t);
int gb_ct_rows_inv_eval_pm_f32(gbofdft_plan*, const void*, int64_t, int, const EvalDesc*, const void*, const void*,
                               void*, int, double*, int64_t*, cudaStream_t);
int gb_plane_conv_f32(gbofdft_plan*, void*, int64_t, int, const KerDesc*, const float* const*, double, cudaStream_t);
int gb_plane_supported_f32(int n0, int n1, int n2);
int gb_ct_rows_inv_store_pm_f32(gbofdft_plan*, const void* spec, int64_t fstride, int nf, void* out, int64_t ostride,
                                cudaStream_t);
int gb_plane_variants_f32(int n0, int n1);
// the plane-major evaluation (returns 1 when the plan has no plane pipeline
// or a kernel table has no plane-major copy)
int gb_eval_plane(gbofdft_plan* p, const void* rho, int nf, const int* ops, double beta, const KerDesc& kd,
                  const EvalDesc& ev, const void* vloc, void* pot, int calc_e, double* energies, cudaStream_t st);
// delta evaluation (passes_delta.cu): FP32 transforms of the change of the
// derived fields against a reference density, FP64 pointwise work
int gb_delta_rows_fwd(gbofdft_plan* p32, const double* rho, const double* rho_ref, void* spec, int64_t fstride,
                      int nf, const int* ops, double beta, cudaStream_t st);
int gb_delta_rows_inv_eval(gbofdft_plan* p32, const void* spec, int64_t fstride, int nf, const EvalDesc* ev,
                           const double* rho, const double* rho_ref, const double* pot_ref, const double* vloc,
                           const double* cref, int64_t cstride, double* pot, int calc_e, double* partials,
                           int64_t* nblk, cudaStream_t st);
int gb_delta_supported(int n0, int n1, int n2);
// the whole delta evaluation of the fused terms (passes.cu): plane pipeline
// of p32 on the changes, FP64 epilogue into pot / energies (energies use p64's
// partials and dV)
int gb_eval_delta_core(gbofdft_plan* p64, gbofdft_plan* p32, const double* rho, const double* rho_ref,
                       const double* pot_ref, const double* eref, const double* cref, int nf, const int* ops,
                       double beta, const KerDesc& kd, const EvalDesc& ev, const double* vloc, double* pot,
                       int calc_e, double* energies, cudaStream_t st);
// the reference density of a delta-evaluation state (device, N doubles)
const double* gb_delta_ref(const gbofdft_delta* d);
void gb_count_launch();
int gb_smem_grant(const void* kern, int bytes);
int gb_use_ct();  // 0 forces the generic passes (GBOFDFT_GENERIC_FFT=1)

int gb_lwt_eval(gbofdft_plan* p, const void* rho, gbofdft_lwt* d, void* pot, double* energies, int calc_v,
                int calc_e, cudaStream_t st);
// the fused terms (ev, kd, nf fields of ops) and the WGC term in one pipeline;
// 1: an axis has no register-blocked passes
int gb_wgc_eval_fused(gbofdft_plan* p, const void* rho, int nf, const int* ops, double beta, const KerDesc& kd,
                      const EvalDesc& ev, const void* vloc, const gbofdft_wgc* d, void* pot, double* energies,
                      int calc_e, cudaStream_t st);
// the total of a row pass's energy partials (k_energy_final)
int gb_energy_final(gbofdft_plan* p, const double* partials, int64_t nblk, double e_ion, double* energies,
                    cudaStream_t st);
// store_ref (FP64 plans): keep this evaluation as the reference of gb_wgc_eval_delta
int gb_wgc_eval(gbofdft_plan* p, const void* rho, const gbofdft_wgc* d, void* pot, double* energies, int calc_v,
                int calc_e, int store_ref, cudaStream_t st);
// the WGC term at rho from the reference kept by the last store_ref
// evaluation with d64 (at rho_ref): FP32 transforms of the change with p32 /
// d32, the NL potential added to pot, the energy to energies (with calc_e)
int gb_wgc_eval_delta(gbofdft_plan* p64, gbofdft_plan* p32, const double* rho, const double* rho_ref,
                      const gbofdft_wgc* d64, const gbofdft_wgc* d32, double* pot, double* energies, int calc_e,
                      cudaStream_t st);

// phi-space TN preconditioner of the uniform gas rho0 on the half spectrum (real, NG values)
int gb_build_precond(gbofdft_plan* p, double rho0, void* out, cudaStream_t st);
int gb_build_wt_kernel(gbofdft_plan* p, double rho0, double x, double alpha, double beta, void* out,
                       cudaStream_t st);
