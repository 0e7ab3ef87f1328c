// Kernel declarations shared between the kernel translation units and the
// C-ABI translation unit.
#pragma once
#include <cuda.h>

#include "nrq_common.cuh"

namespace nrq {

// ---------------- gauge.cu
__global__ void k_links_f2soa(const double2 *__restrict__ f, double2 *__restrict__ U, int64_t V);
__global__ void k_links_soa2f(const double2 *__restrict__ U, double2 *__restrict__ f, int64_t V);
__global__ void k_efield_f2soa(const double *__restrict__ f, double *__restrict__ E, int64_t V);
__global__ void k_efield_soa2f(const double *__restrict__ E, double *__restrict__ f, int64_t V);
__global__ void k_cold(double2 *__restrict__ U, double *__restrict__ E, int64_t V);
void launch_update_links(Lat L, double2 *U, const double *E, double dt, cudaStream_t st);
void launch_update_efield(Lat L, const double2 *U, double *E, double dt, cudaStream_t st);
// precision form of the leapfrog: FP32 links, FP64 Ẽ (gauge.cu)
__global__ void k_update_links32(Lat L, float2 *__restrict__ U, const double *__restrict__ E, double dt);
__global__ void k_update_efield32(Lat L, const float2 *__restrict__ U, double *__restrict__ E, double dt);
__global__ void k_reunitarise(int64_t V, float2 *__restrict__ U32, double2 *__restrict__ U64);
__global__ void k_links_widen(int64_t n, const float2 *__restrict__ U32, double2 *__restrict__ U64);
__global__ void k_links_narrow(int64_t n, const double2 *__restrict__ U64, float2 *__restrict__ U32);
__global__ void k_unitarity(Lat L, const double2 *__restrict__ U, double *partials);
__global__ void k_energy(Lat L, const double2 *__restrict__ U, const double *__restrict__ E, double *partials);
__global__ void k_gauss(Lat L, const double2 *__restrict__ U, const double *__restrict__ E, double *partials);
__global__ void k_reduce_final(const double *__restrict__ partials, int64_t nblk, int nq, unsigned maxmask,
                               double *out);
void launch_reduce_final(const double *partials, int64_t nblk, int nq, unsigned maxmask, double *out, cudaStream_t st);
__global__ void k_ic_pspace(Lat L, const double2 *__restrict__ R, const double *__restrict__ mtab,
                            double fwd_scale, double Q, double n0, double g, double2 *__restrict__ A,
                            double2 *__restrict__ Ef);
__global__ void k_ic_write(Lat L, const double2 *__restrict__ A, const double2 *__restrict__ Ef,
                           double inv_volume, int identity_links, double2 *__restrict__ U,
                           double *__restrict__ E);

// ---------------- gauss_proj.cu
// device state of a Gauss projection: convergence flag, sweeps taken, last
// deviation, and the block ticket of the deviation reduction (zero between
// launches)
struct GaussProjState {
  int done;
  unsigned ticket;
  long long sweeps;
  double dev;
};
__global__ void k_gauss_g(Lat L, const double2 *__restrict__ U, const double *__restrict__ E,
                          double2 *__restrict__ G, double *__restrict__ partials, GaussProjState *st, double tol,
                          int count);
__global__ void k_gauss_sweep(Lat L, const double2 *__restrict__ U, const double2 *__restrict__ G,
                              double *__restrict__ E, const GaussProjState *st, double kdt);
// nsweeps sweeps in one launch, from Ein into Eout (may be the same), where
// gauss_run_applicable; devmax[n] = the deviation before sweep n = 0..nsweeps.
// messages: gauss_run_message_bytes, zero before a projection's first launch;
// te, ge: the numbers of the launch's first messages (nsweeps + 1 and nsweeps
// of them), from 1 on; dev: gauss_run_warps doubles per entry of devmax.
// stall: the last warp is left out, so that the waits for its messages run out
// (the host's test of the timeout path).
int gauss_run_warps(int64_t V);
bool gauss_run_applicable(int64_t V, int sm_count);
int64_t gauss_run_message_bytes(int64_t V);
cudaError_t launch_gauss_run(Lat L, const double2 *U, const double *Ein, double *Eout, void *messages, double *dev,
                             double *devmax, int nsweeps, uint32_t te, uint32_t ge, double kdt, int sm_count, int *err,
                             cudaStream_t st, long long wait_cycles, bool stall);

// ---------------- gluon.cu
__global__ void k_cg_divergence(Lat L, const double2 *__restrict__ U, double2 *__restrict__ D,
                                double *__restrict__ partials);
__global__ void k_cg_accelerate(Lat L, double2 *__restrict__ D, double pmax, double scale);
__global__ void k_cg_expah(int64_t V, double2 *__restrict__ D);
__global__ void k_cg_transform(Lat L, double2 *__restrict__ U, const double2 *__restrict__ G);
// gauge fixing on short extents (three launches an iteration)
constexpr int kCgMaxExtent = 32, kCgRowSites = 64;
bool cg_short_applicable(const Lat &L);
void launch_cg_tables(Lat L, double2 *tw, double *p2, cudaStream_t st);  // 3*kCgMaxExtent entries each
// U' = G U G^+ from Uin to Uout (G null: no transformation), then its
// deviation into dev[slot] (zero before) and the x transform of its
// divergence into F (5V; null: neither).  Nothing where dev[slot - 1] (slot >
// 0) has met tol.
void launch_cg_rows(Lat L, const double2 *Uin, const double2 *G, double2 *Uout, const double2 *tw, double2 *F,
                    double *dev, double tol, int slot, cudaStream_t st);
// G = ExpAH of the accelerated divergence; nothing where dev[slot] has met tol
void launch_cg_smooth(Lat L, const double2 *tw, const double *p2, double2 *F, double2 *G, double pmax, double scale,
                      const double *dev, double tol, int slot, cudaStream_t st);
__global__ void k_gluon_fields(Lat L, const double2 *__restrict__ U, const double *__restrict__ E,
                               double2 *__restrict__ F);
__global__ void k_transverse_corr(Lat L, const double2 *__restrict__ F, double fwd, double volume,
                                  double *__restrict__ out);

// ---------------- cn.cu
// Per-species, per-term complex coefficients of the assembled CN operator:
//   out = in + sum_t alpha_t G_t in      (t = kinetic, magnetic, Darwin, spin-orbit)
struct CnCoef {
  cplx kin[2], mag[2], dar[2], so[2];
  double dkin;       // sum_i 1/a_i^2
  double inva2[3];   // 1/a_i^2
};

// FMA stencil only, the plain solve with the merged update and the shadow
// residual rh kept in FP32 (sh32; any fixed shadow vector serves BiCGStab,
// and every product with it uses the same rounded values):
//   MV_RES2: MV_RES writing rh = f32(r) to sh32 and reducing rh^H r (rho_0);
//   MV_V2:   MV_V with rh^H v from sh32;
//   MV_T2:   MV_T on a materialised s that also reduces rh^H t from sh32,
//            from which the merged update takes beta
// Spin-structured stencil only, the Chebyshev semi-iteration of the plain
// solve (tab: its coefficients, ChebTab below):
//   MV_RESN: |b - y|^2 and |b|^2 alone;
//   MV_CH0:  x_1 = x_0 + r_0 / theta, with the sums of MV_RESN;
//   MV_CHK:  x_{k+1} = x_k + c1 (x_k - x_{k-1}) + c2 (b - y), x_{k-1} in out
//            and overwritten;
//   MV_CHH:  MV_CHK that also stores the step's history x - (2b - psi) in FP32
enum MvMode { MV_PLAIN = 0, MV_RHS = 1, MV_RES = 2, MV_V = 3, MV_T = 4, MV_RESC = 5, MV_T2 = 6, MV_RES2 = 7,
              MV_V2 = 8, MV_RESN = 9, MV_CH0 = 10, MV_CHK = 11, MV_CHH = 12 };

struct ChebTab;

struct MvArgs {
  const double2 *in;  // operand (PLAIN/RHS: psi, RES, CH*: x, V: p, T: r)
  const double2 *in2; // T: v ; CHH: psi ; RHS: (unused)
  double2 *out;       // PLAIN: A in ; RHS: b ; RES: r ; V: v ; T: t ; CH0: x_1 ; CHK, CHH: x_{k-1}, then x_{k+1}
  double2 *out2;      // RHS: x0 = 2b - psi ; RES: rh
  double2 *out3;      // RES: p
  const double2 *bvec;// RES, CH*: b
  const double *scal; // per-column scalars
  double *partials;   // per block, per column, NQ doubles
  // MV_RESC (residual for the FP32 Chebyshev inner solve): r32 = f32(b - A^H x),
  // d32 = f32((b - A^H x) / theta_species); CHH: r32 = the history slot
  float2 *r32;
  float2 *d32;
  cplx inv_theta[2];
  float2 *sh32;       // RES2: FP32 shadow residual written; V2, T2: read
  // spin-structured stencil: the Chebyshev table and step; RHS: the history
  // vectors added to x0 with their coefficients (null: none), r32 the FP32
  // copy of what they add (may be null, may be one of them)
  const ChebTab *cheb;
  int step;
  const float2 *hist[4];
  double hcoef[4];
};

// per-species coefficients of one Chebyshev step: d' = c1 d + c2 r
struct ChebCoef {
  cplx c1[2], c2[2];
};

// the Chebyshev coefficients of one operator by step (step[0]: c1 = 0, c2 =
// 1/theta) and the enclosure of its hermitian part they were made for
// (k_spin_bounds, cn_spin.cu)
constexpr int kChebTab = 40;
struct ChebTab {
  ChebCoef step[kChebTab];
  cplx inv_theta[2];
  double lo[2], hi[2];
};

// Chebyshev iteration on the segment of A^H = 1 + i tau H, spec(H) in [lo, hi]:
// theta its centre, delta its half length, sigma = theta / delta.  The ratios
// rho_k = T_k(sigma) / T_{k+1}(sigma), which the recurrence rho_0 = 1 / sigma,
// rho_{k+1} = 1 / (2 sigma - rho_k) makes one after another, come here from
// T_k = (w^k + w^-k) / 2, w = sigma + sqrt(sigma^2 - 1), |w| > 1, each by
// itself.  x_1 = x_0 + r_0 / theta, x_{k+1} = x_k + rho_k rho_{k-1} (x_k -
// x_{k-1}) + c2(rho_k) r_k.
struct ChebSegment {
  cplx theta, winv, u;  // u = w^-2
  double half;
  __device__ ChebSegment(double tau, double lo, double hi) {
    theta = {1.0, tau * 0.5 * (lo + hi)};
    half = fmax(fabs(tau) * 0.5 * (hi - lo), 1e-14);
    const cplx sigma = {theta.im / half, -theta.re / half};  // over i half
    const cplx z = sigma * sigma - cplx{1.0, 0.0};
    const double m = sqrt(0.5 * (hypot(z.re, z.im) + fabs(z.re)));
    cplx r = z.re >= 0.0 ? cplx{m, m > 0.0 ? 0.5 * z.im / m : 0.0} : cplx{0.5 * fabs(z.im) / m, copysign(m, z.im)};
    if (sigma.re * r.re + sigma.im * r.im < 0.0) r = -1.0 * r;
    winv = cdiv({1.0, 0.0}, sigma + r);
    u = winv * winv;
  }
  __device__ cplx pow_u(int k) const {
    cplx p = {1.0, 0.0}, b = u;
    for (; k > 0; k >>= 1) {
      if (k & 1) p = p * b;
      b = b * b;
    }
    return p;
  }
  __device__ cplx rho(int k) const {
    const cplx one = {1.0, 0.0}, p = pow_u(k);
    return cdiv(winv * (one + p), one + p * u);
  }
  // |T_m(sigma)|
  __device__ double gain(int m) const {
    double g = 0.5 * sqrt(norm2(cplx{1.0, 0.0} + pow_u(m))), b = 1.0 / sqrt(norm2(winv));
    for (; m > 0; m >>= 1) {
      if (m & 1) g *= b;
      b *= b;
    }
    return g;
  }
  __device__ cplx inv_theta() const { return cdiv({1.0, 0.0}, theta); }
  __device__ cplx c2(cplx rho) const { return {2.0 * rho.im / half, -2.0 * rho.re / half}; }
};

// The operator in its spin structure (cn_spin.cu), real Wilson coefficients:
// A^H psi(x) = (1 + i (S0 +- S1)) psi(x) + the six neighbours' blocks from
// three colour matrices a direction.  Planes of V: W 81 complex ((I*3 + m)*9
// + row*3 + column), S0 9 complex, S1 9 real, each per coefficient set.
struct SpinOp {
  double2 *W, *S0;
  double *S1;
};
// the same planes rounded to FP32
struct SpinOp32 {
  float2 *W, *S0;
  float *S1;
};
// Builds op and op32 (either left out where its W is null) for nm
// coefficient sets (device array Cm; null: the one set C), and seven real
// scratch planes a set for the spectral enclosure (null: none).  tau = dt a0 / 2.
void launch_spin_prepare(Lat L, const CnCoef &C, const CnCoef *Cm, int nm, double tau, const double2 *U,
                         const double *E, const SpinOp &op, const SpinOp32 &op32, double *scratch, cudaStream_t st);
// out[4*set] = {lo, hi} of the quark's and the antiquark's H, A^H = 1 + i tau
// H; partials: 4 doubles per 256 sites and set; ticket: one zero per set.  One
// set and tab: also the Chebyshev table of these bounds, and the bounds into
// the pinned host_bounds.
void launch_spin_bounds(Lat L, int nm, const double *scratch, double *partials, unsigned *ticket, double *out,
                        cudaStream_t st, double tau = 0.0, ChebTab *tab = nullptr, double *host_bounds = nullptr);
bool cn_spin_applicable(const Lat &L);
// the stencil over op (sign = -1: A = 2 - A^H, for MV_PLAIN and MV_RHS); one
// partial row per 32-site block.  early: the launch before this one on the
// stream did not write op.
void launch_cn_spin(int mode, Lat L, const SpinOp &op, double sign, const MvArgs &a, bool early, int *err,
                    cudaStream_t st, long long wait_cycles, int stall_load);

constexpr int CN_SITES_PER_BLOCK = 32;
constexpr int CN_COLS = 12;  // 2 species x 6 propagator columns
constexpr int SC_STRIDE = 16; // doubles per column in the scalar array
// scalar slots (per column)
enum {
  SC_RHO = 0,    // complex (2)
  SC_ALPHA = 2,  // complex
  SC_OMEGA = 4,  // complex
  SC_BETA = 6,   // complex
  SC_RR = 8,
  SC_BB = 9,
  SC_CONV = 10,  // 1.0 when converged
  SC_BREAK = 11, // 1.0 on breakdown (restart requested)
  SC_NONFIN = 12,
  SC_SS = 13,    // |s|^2 of the half step (when checked)
  SC_HALF = 14   // 1.0 when the half step s = r - alpha v met the tolerance
};

void launch_cn_prepare(Lat L, const double2 *U, const double *E, double2 *Dsum, double *Bsum, double2 *DE,
                       cudaStream_t st);
void launch_cn_mv(int mode, Lat L, const CnCoef &C, const double2 *U, const double2 *Dsum, const double *Bsum,
                  const double2 *DE, const MvArgs &a, cudaStream_t st);
void launch_vec_xr(Lat L, double2 *x, double2 *r, const double2 *p, const double2 *v, const double2 *t,
                   const double2 *rh, const double *scal, double *partials, cudaStream_t st);
void launch_vec_p(Lat L, double2 *p, const double2 *r, const double2 *v, const double *scal, cudaStream_t st);
void launch_vec_s(Lat L, double2 *s, const double2 *r, const double2 *v, const double *scal, cudaStream_t st,
                  double *partials = nullptr);
void launch_vec_xp(Lat L, double2 *x, const double2 *p, const double *scal, cudaStream_t st);
void launch_vec_xrp(Lat L, double2 *x, double2 *r, double2 *p, const double2 *s, const double2 *t,
                    const double2 *v, const double *scal, double *partials, cudaStream_t st);
void launch_vec_xr_s(Lat L, double2 *x, double2 *r, const double2 *p, const double2 *s, const double2 *t,
                     const double2 *rh, const double *scal, double *partials, cudaStream_t st);
// TMA-staged stencil (cn_mv3.cu); returns nonzero if the tensor maps cannot
// describe this lattice (then the caller uses launch_cn_mv).  For MV_T its
// input is the materialised s = r - alpha v.
int launch_cn_mv3(int mode, Lat L, const CnCoef &C, const double2 *U, const double2 *Dsum, const double *Bsum,
                  const double2 *DE, const MvArgs &a, int *err, int sm_count, cudaStream_t st);
// Tensor-core stencil (cn_mv4.cu): forward 6x6 blocks of every site,
// direction and species for coefficients C (216 complex per site), then the
// stencil over them; nb_sign = -1 applies the operator whose off-diagonal
// coefficients are those of C negated.  Needs imaginary off-diagonal
// coefficients.  Returns nonzero if the tensor maps cannot describe this
// lattice.  One partial row per CTA (cn_mv4_rows).
void launch_cn_blocks(Lat L, const CnCoef &C, const double2 *U, const double2 *DE, double2 *W, cudaStream_t st);
int64_t cn_mv4_units(int64_t V);
int64_t cn_mv4_rows(int64_t V, int sm_count);
int launch_cn_mv4(int mode, Lat L, const CnCoef &C, double nb_sign, const double2 *W, const double2 *Dsum,
                  const double *Bsum, const MvArgs &a, int *err, int sm_count, cudaStream_t st);
// finalize stages: 0 = after RES (rr, bb), 1 = alpha (rh.v), 2 = omega (t.s, t.t), 3 = beta (rh.r, r.r)
void launch_cn_finalize(int stage, int64_t nblocks, const double *partials, double *scal, double tol,
                        cudaStream_t st);
// one field of a batched Crank-Nicolson step (device table entry)
constexpr int BATCH_MAX_CHEB = 32;
struct BatchField {
  CnCoef CA, CH;                 // operator A and A^H coefficients at this field's mass
  double2 *psi, *b, *x;          // FP64 propagator, right-hand side, iterate (72 planes)
  float2 *r32, *dA, *dB, *e32;   // FP32 Chebyshev vectors (72 planes)
  double *partials;              // residual (r.r, b.b) partials of this field
  double *scal;                  // per-column scalars of this field (CN_COLS x SC_STRIDE)
  const double *bounds;          // spectral enclosure of this field's mass (lo0, hi0, lo1, hi1)
  double tau;                    // dt a0 / 2 (signed)
  double mass;                   // heavy mass of this field
  int wblk;                      // the field's coefficient set (its distinct mass)
  int hstart;                    // the field starts from the extrapolation of h1..h4
  // learned initial guess: the field's history (v1 newest, v2 older; null
  // when absent) and the slot the new history goes to (null: no learned guess)
  const float2 *h1, *h2;
  float2 *hnew;
  // history start without the learned guess: the field's third and fourth
  // newest history vectors (null when absent; h1, h2 the newest two)
  const float2 *h3, *h4;
  cplx inv_theta[2];             // 1/theta per species (written on the device)
  ChebCoef cheb[BATCH_MAX_CHEB]; // Chebyshev steps (written on the device)
  // guaranteed gain |T_m(sigma)| of m Chebyshev steps per species (written
  // on the device)
  double gain[2][BATCH_MAX_CHEB + 1];
};
// every column of the field converged at its last residual check
__device__ __forceinline__ bool batch_field_done(const BatchField &f) {
  bool d = true;
#pragma unroll
  for (int k = 0; k < CN_COLS; ++k) d = d && f.scal[k * SC_STRIDE + SC_CONV] != 0.0;
  return d;
}
// skip_done: residual launches after the first of a step leave converged
// fields alone (their iterate did not change since their last check)
void launch_batch_mv(int mode, int order, Lat L, const double2 *U, const double2 *Dsum, const double *Bsum,
                     const double2 *DE, const BatchField *tab, int nfields, int skip_done, cudaStream_t st);
// The same two modes (MV_RHS, MV_RESC) on the operator in its spin structure
// (cn_spin.cu), one coefficient set per distinct mass (the field's wblk).
// MV_RHS adds the fields' history to their start and fills hnew (hstart);
// MV_RESC writes d = r / theta only where want_d.  The residual's partials
// are one row per (field, 32-site unit), the rows of launch_batch_finalize.
void launch_batch_spin(int mode, int order, Lat L, const SpinOp &op, const BatchField *tab, int nfields, int skip_done,
                       bool want_d, int *err, cudaStream_t st, long long wait_cycles);
// Chebyshev kernel variants: 0 = one field per tile, 2 blocks/SM (168
// registers); 1 = one field per tile, 3 blocks/SM (113 registers); 2 = two
// fields of one mass per tile, 1 block/SM.  Returns nonzero for an
// unsupported variant (a two-field tile needs an even count per mass).
constexpr int BATCH_CHEB_VARIANTS = 4;
int launch_batch_cheb(int step, int variant, int order, Lat L, const float2 *U, const float2 *Dsum,
                      const float *Bsum, const float2 *DE, const BatchField *tab, int nfields, cudaStream_t st);
// Variant 3 of the batched Chebyshev step: launch_cheb_spin over every field
// (blocks over (field, unit), field fastest for order 0), e on the fields'
// dA and dB; the last launch of a pass updates x and hnew itself.  A pass of
// one step is launch_batch_cheb_one.
void launch_batch_cheb_spin(int step, bool last, int order, Lat L, const SpinOp32 &op, const BatchField *tab,
                            int nfields, int *err, cudaStream_t st, long long wait_cycles);
void launch_batch_cheb_one(int64_t n, const BatchField *tab, int nfields, cudaStream_t st);
void launch_batch_add_e(int64_t n, const BatchField *tab, int nfields, cudaStream_t st);
// Chebyshev coefficients of every field from its mass's bounds; sets
// flags[f] = 1 for non-finite bounds
void launch_batch_coef(BatchField *tab, int nfields, int *flags, cudaStream_t st);
// stage-0 reduction of every field's residual partials (nrows rows per field)
// skip_done: the residual launch skipped the fields whose every column had
// converged (their scalars stay as they are)
void launch_batch_finalize(const BatchField *tab, int nfields, int64_t nrows, double tol, int skip_done,
                           cudaStream_t st);
// The prediction of the scheduled step's last pass (m Chebyshev steps):
// every unconverged column's residual before the pass over the pass's
// guaranteed gain.  pstate = {ratio, steps}: the largest true-to-predicted
// ratio measured so far (-1: none) and the scheduled steps taken.  Where
// prediction is on (a ratio measured and steps not a multiple of 16) and
// twice the prediction, scaled by max(1, ratio), meets tol, the column is
// marked converged on it (SC_HALF = 1, SC_RR the scaled prediction);
// otherwise it waits for the residual check (SC_HALF = 2, SC_SS the
// prediction).  launch_batch_calibrate, after that check, takes the ratio
// of the measured columns into pstate and counts the step.
void launch_batch_predict(const BatchField *tab, int nfields, int m, double tol, const double *pstate,
                          cudaStream_t st);
void launch_batch_calibrate(const BatchField *tab, int nfields, double *pstate, cudaStream_t st);
// The history start of every field (no learned guess): with the field's
// history vectors h1.. (d of them, the first null ends the list) x +=
// sum_k c_k h_k, c of the degree d - 1 extrapolation, and hnew = the same
// sum in FP32 (0 without history), to which every correction is added.
void launch_batch_hist_start(int64_t V, const BatchField *tab, int nfields, cudaStream_t st);
void launch_cn_to_f32(int64_t V, const double2 *U, const double2 *DE, const double2 *D, const double *B, float2 *U32,
                      float2 *DE32, float2 *D32, float *B32, cudaStream_t st);
void launch_cheb32(bool first, Lat L, const CnCoef &C, const float2 *U, const float2 *Dsum, const float *Bsum,
                   const float2 *DE, const float2 *D, float2 *Dn, float2 *R, float2 *E, const ChebCoef &K,
                   cudaStream_t st);
// The inner solve A^H e = r on the operator in its spin structure, FP32
// (cn_spin32.cu): launch `step` = 0, 1, .. makes e_{step+2} with the step's
// coefficients K, into ea (even steps) or eb (odd ones); the last one adds it
// to x instead and, if not null, to hist, or with b and psi stores hist = x -
// (2b - psi).  m Chebyshev steps take m - 1
// launches, one step is launch_cheb_one over the n elements.
bool cheb_spin_applicable(const Lat &L);
void launch_cheb_spin(int step, bool last, Lat L, const SpinOp32 &op, const float2 *r, float2 *ea, float2 *eb,
                      double2 *x, float2 *hist, const double2 *b, const double2 *psi, const ChebCoef &K,
                      const cplx inv_theta[2], bool early, int *err, cudaStream_t st, long long wait_cycles);
void launch_cheb_one(int64_t n, const float2 *r, double2 *x, float2 *hist, const double2 *b, const double2 *psi,
                     const cplx inv_theta[2], cudaStream_t st);
void launch_add_e(int64_t n, double2 *X, const float2 *E, cudaStream_t st);
void launch_prop_f2soa(const double2 *f, double2 *P, int64_t V, cudaStream_t st);
void launch_prop_soa2f(const double2 *P, double2 *f, int64_t V, cudaStream_t st);
void launch_single_point(double2 *P, int64_t V, int64_t sq, int64_t sa, cudaStream_t st);
// |psi|^2 of species sp0 .. sp0 + nsp - 1 (nsp values per partial row)
void launch_norms(const double2 *P, int64_t V, int sp0, int nsp, double *partials, int64_t &nblk, cudaStream_t st);
// coefficient of the (k+1)-th newest of d history vectors (degree d - 1 extrapolation)
double hist_coef(int d, int k);
// x += sum_k c_k t_k over the d newest history vectors t[0..d-1] (d = 1..4),
// c the coefficients of the degree d - 1 extrapolation
void launch_hist_extrapolate(int64_t n, double2 *X, const float2 *const *t, int d, cudaStream_t st);
void launch_hist_store(int64_t n, const double2 *X, const double2 *B, const double2 *Psi, float2 *T, cudaStream_t st);
void launch_correlators(const double2 *P, int64_t V, double *partials, int64_t &nblk, cudaStream_t st,
                        bool gconjg = false);

}  // namespace nrq
