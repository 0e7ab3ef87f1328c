// FP64 stencil of the assembled Crank-Nicolson operator in its spin structure
// (src/nrqcd.f90:1175-1387 with PETSc's block transposition; the operator is
// described in cn.cu), for real Wilson coefficients.
//
// Operator.  With real coefficients the 6x6 block to the neighbour x + I is
// K 1 + s_a X + s_b Z in spin space, K the link, X and Z the two spin-orbit
// colour matrices, and the antiquark's is the quark's with K negated.  In the
// basis where the block is written down that leaves three colour matrices a
// direction for both species:
//   I = 0, 1:  quark [[m0, m2], [-+m2, m1]], antiquark [[-m1, m2], [-+m2, -m0]]
//   I = 2:     quark [[m0, m2], [m1, m0]],   antiquark [[-m0, m2], [m1, -m0]]
// (the lower sign for I = 1), 27 complex numbers in place of the 72 of two
// dense 6x6 blocks: 1296 B a site for all three directions (from 3456), and
// every matrix read serves both species.  The backward block is
// -W_I(x - I)^H.  The site term is 1 + i (S0 +- S1), S0 the Darwin matrix,
// S1 the magnetic one with the diagonal of the Laplacian (+ quark, -
// antiquark).  A = 2 - A^H, so one operator serves both.
//
// Products.  A block works on 32 consecutive sites, a warp on one propagator
// column of both species, a lane on one site: 12 complex accumulators.  The
// 18 steps (neighbour, input colour) each take nine matrix entries and four
// spinor entries, 96 FP64 FMAs on 13 16-byte loads; three further steps take
// the site term.  The matrices of a neighbour are staged in shared memory by
// all six warps (cp.async, one mbarrier per neighbour, two neighbours ahead:
// a warp that sees the matrices of neighbour n landed knows that every warp
// has left neighbour n - 3, so a fifth buffer is free), and the spinors go
// straight to registers three steps ahead.  Nothing depends on the lattice's
// shape: each lane reads its own neighbours' addresses, so one kernel serves
// rows of any length, and small lattices get one block per 32 sites.  In a
// batch the blocks run over (field, unit).  The device code is in
// cn_spin.cuh.
//
// Bound: 64^3, the solver's step (four vector streams, 6.1 KB a site): 0.25 ms
// at the copy rate, 0.21 ms at the FP64 rate that FMAs with distinct operands
// reach (49 of 64 a clock and SM).  It takes 0.37 ms (the TMA stencil on dense
// 6x6 blocks before it 0.47): 70 % of the copy rate, of the shared-memory
// path's wavefronts and half of the FP64 pipe at twelve warps an SM (166
// registers); the loads alone take 0.31 ms (the launch without its products).
// 24^3: 28 us, 12^3: 9 us.
//
// Every mbarrier wait is bounded (wait_cycles); on expiry the thread records
// NRQ_ERR_TIMEOUT in *err and its warp skips the remaining work.  stall_load
// >= 0 makes every block stop staging before that neighbour, so that the
// wait for it runs out: the host's test of the timeout path (nothing faults;
// the context stays usable).  A block waits for its own copies before it
// exits.
#include <algorithm>

#include "../../include/nrqcd_b200.h"
#include "cn_spin.cuh"
#include "nrq_eigen.cuh"

namespace nrq {

// ------------------------------------------------------------------ operator
namespace {
// symmetric real 3x3: 00 01 02 11 12 22
struct s3 {
  double e[6];
};
__device__ __forceinline__ constexpr int s3i(int r, int c) {
  return r <= c ? r * (5 - r) / 2 + c : c * (5 - c) / 2 + r;
}
// E_j(y) entering the operator: -Re(sum_a E~^a T^a)/a0/a_j
__device__ __forceinline__ s3 efield_s3(const Lat &L, const double *__restrict__ E, int64_t y, int j) {
  const int64_t V = L.V;
  const double h = 0.5, s8 = 0.5 / 1.7320508075688772, d8 = 1.0 / 1.7320508075688772;
  const double *e = E + (int64_t)(j * 8) * V + y;
  const double e1 = __ldg(e), e3 = __ldg(e + 2 * V), e4 = __ldg(e + 3 * V), e6 = __ldg(e + 5 * V),
               e8 = __ldg(e + 7 * V);
  const double f = -1.0 / L.a0 / L.a[j];
  return {{(h * e3 + s8 * e8) * f, (h * e1) * f, (h * e4) * f, (-h * e3 + s8 * e8) * f, (h * e6) * f, (-d8 * e8) * f}};
}
__device__ __forceinline__ m3 mul_us(const m3 &u, const s3 &e) {
  m3 r;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      cplx a = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        a.re = fma(u.e[i * 3 + k].re, e.e[s3i(k, j)], a.re);
        a.im = fma(u.e[i * 3 + k].im, e.e[s3i(k, j)], a.im);
      }
      r.e[i * 3 + j] = a;
    }
  return r;
}
__device__ __forceinline__ m3 mul_su(const s3 &e, const m3 &u) {
  m3 r;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      cplx a = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        a.re = fma(e.e[s3i(i, k)], u.e[k * 3 + j].re, a.re);
        a.im = fma(e.e[s3i(i, k)], u.e[k * 3 + j].im, a.im);
      }
      r.e[i * 3 + j] = a;
    }
  return r;
}
// Re(LogU(P)/i) of a plaquette (matrixoperations:510-531)
__device__ __noinline__ void log_jacobi(const m3 &P, m3 &H) {
  cplx ev[3];
  m3 S;
  eigenc3(P, ev, S);
  double th[3];
  for (int k = 0; k < 3; ++k) th[k] = atan2(ev[k].im, ev[k].re);
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) {
      double acc = 0.0;
      for (int k = 0; k < 3; ++k) {
        const cplx a = S.e[k * 3 + r], b = S.e[k * 3 + c];
        acc += th[k] * (a.re * b.re + a.im * b.im);
      }
      H.e[r * 3 + c] = {acc, 0.0};
    }
}
constexpr int kPrepSites = 32;
}  // namespace

// Builds the operator of the nm coefficient sets Cm (null: the one set C1),
// from the links and the electric field, in FP64 (op) and rounded to FP32
// (op32), either left out where its pointers are null: W (81 planes of V complex per set,
// (I*3 + m)*9 + row*3 + column), S0 (9 planes, row*3 + column), S1 (9 real
// planes) and, for the spectral enclosure, seven real planes per set: the
// norm bound of the block to x + I (I = 0..2), and centre and deviation of
// the site term of the hermitian H (A^H = 1 + i tau H) for quark and
// antiquark.  One thread per site and direction; the Darwin and magnetic
// matrices are sums over directions, exchanged through shared memory.  64^3:
// 217 us, with the FP32 copy 248, at 12 warps an SM (168 registers; without
// the test that the plaquettes are unitary 211 and 240; 255 registers, 8
// warps: 286 and 315; 136 registers, 15 warps: 280 with the copy), of which
// the traffic takes 90; 12^3: 14 us.
__global__ void __launch_bounds__(kPrepSites * 3, 4) k_spin_prepare(Lat L, CnCoef C1, const CnCoef *__restrict__ Cm,
                                                                int nm, double tau, const double2 *__restrict__ U,
                                                                const double *__restrict__ E, SpinOp op,
                                                                SpinOp32 op32, double *__restrict__ scratch) {
  __shared__ double sD[3][9][kPrepSites];  // Darwin: 0..2 the diagonal, then 01, 02, 12 as (re, im)
  __shared__ double sB[3][6][kPrepSites];
  const int l = threadIdx.x % kPrepSites, i = threadIdx.x / kPrepSites;
  const int64_t V = L.V;
  const int64_t x0 = (int64_t)blockIdx.x * kPrepSites + l;
  const bool act = x0 < V;
  const int64_t x = act ? x0 : V - 1;
  const int j = i == 2 ? 0 : i + 1, k = i == 0 ? 2 : i - 1;
  const int64_t xp = nb(L, x, i, +1), xm = nb(L, x, i, -1);
  const m3 u = load_link(U, V, x, i);
  {  // Darwin: (u E_i(x+i) u^+ - um^+ E_i(x-i) um) / 2a_i, hermitian
    const m3 um = load_link(U, V, xm, i);
    const m3 t1 = mul_nd(mul_us(u, efield_s3(L, E, xp, i)), u);
    const m3 t2 = mul_dn(um, mul_su(efield_s3(L, E, xm, i), um));
    const double s = 1.0 / (2.0 * L.a[i]);
#pragma unroll
    for (int r = 0; r < 3; ++r) sD[i][r][l] = s * (t1.e[4 * r].re - t2.e[4 * r].re);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const int p = e == 2 ? 5 : e + 1;  // 01, 02, 12
      sD[i][3 + 2 * e][l] = s * (t1.e[p].re - t2.e[p].re);
      sD[i][4 + 2 * e][l] = s * (t1.e[p].im - t2.e[p].im);
    }
  }
  {  // magnetic: F_jk, (i, j, k) cyclic
    const m3 P = mul_nd(mul_nd(mul(load_link(U, V, x, j), load_link(U, V, nb(L, x, j, +1), k)),
                               load_link(U, V, nb(L, x, k, +1), j)),
                        load_link(U, V, x, k));
    m3 H;
    if (!log_unitary(P, H, true)) log_jacobi(P, H);
    const double s = 1.0 / L.a[j] / L.a[k];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = r; c < 3; ++c) sB[i][s3i(r, c)][l] = s * H.e[r * 3 + c].re;
  }
  // spin-orbit: (E_j u + u E_j(x+i)) / 2a_i and the same for k
  m3 d0 = add(mul_su(efield_s3(L, E, x, j), u), mul_us(u, efield_s3(L, E, xp, j)));
  m3 d1 = add(mul_su(efield_s3(L, E, x, k), u), mul_us(u, efield_s3(L, E, xp, k)));
  const double so = 0.5 / L.a[i];
  double n0 = 0.0, n1 = 0.0;
#pragma unroll
  for (int e = 0; e < 9; ++e) {
    d0.e[e] = so * d0.e[e];
    d1.e[e] = so * d1.e[e];
    n0 += norm2(d0.e[e]);
    n1 += norm2(d1.e[e]);
  }
  const double nDE = sqrt(n0) + sqrt(n1);
  double nU;
  {  // |u|_2 <= sqrt(1 + |u^+ u - 1|_F)
    const m3 uu = mul_dn(u, u);
    double q = 0.0;
#pragma unroll
    for (int e = 0; e < 9; ++e) {
      const double re = uu.e[e].re - (e % 4 == 0 ? 1.0 : 0.0);
      q += re * re + uu.e[e].im * uu.e[e].im;
    }
    nU = sqrt(1.0 + sqrt(q));
  }
  __syncthreads();
  // row i of the site term
  double D[9], B[6];
#pragma unroll
  for (int e = 0; e < 9; ++e) D[e] = sD[0][e][l] + sD[1][e][l] + sD[2][e][l];
#pragma unroll
  for (int e = 0; e < 6; ++e) B[e] = sB[0][e][l] + sB[1][e][l] + sB[2][e][l];
  if (!act) return;
  for (int km = 0; km < nm; ++km) {
    const CnCoef &C = Cm ? Cm[km] : C1;
    const int64_t ow = (int64_t)km * 81 * V + (int64_t)(i * 27) * V + x;
    double2 *W = op.W + ow;
    float2 *Wf = op32.W + ow;
    const cplx ck = (-0.5 * C.inva2[i]) * C.kin[0];
    const cplx c0 = times_i(C.so[0]), c1 = -times_i(C.so[0]);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        // entry (r, c) of the transposed matrices (PETSc's block transposition)
        const cplx ku = ck * u.e[c * 3 + r], e0 = c0 * d0.e[c * 3 + r], e1 = c1 * d1.e[c * 3 + r];
        cplx a, b, o;
        if (i == 0) {  // s_3 e0 + s_2^T e1
          a = ku + e0;
          b = ku - e0;
          o = -times_i(e1);
        } else if (i == 1) {  // s_1 e0 + s_3 e1
          a = ku + e1;
          b = ku - e1;
          o = e0;
        } else {  // s_2^T e0 + s_1 e1
          a = ku;
          b = times_i(e0) + e1;
          o = e1 - times_i(e0);
        }
        if (op.W) {
          st(W + (int64_t)(r * 3 + c) * V, a);
          st(W + (int64_t)(9 + r * 3 + c) * V, b);
          st(W + (int64_t)(18 + r * 3 + c) * V, o);
        }
        if (op32.W) {
          Wf[(int64_t)(r * 3 + c) * V] = make_float2((float)a.re, (float)a.im);
          Wf[(int64_t)(9 + r * 3 + c) * V] = make_float2((float)b.re, (float)b.im);
          Wf[(int64_t)(18 + r * 3 + c) * V] = make_float2((float)o.re, (float)o.im);
        }
      }
    // S0 = Im(dar) D^T, S1 = Im(mag) B + Im(kin) sum 1/a^2
    const double dd = C.dar[0].im, mm = C.mag[0].im, kk = C.kin[0].im * C.dkin;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      // D^T[i][c] = conj(D[i][c])
      cplx v = {i == 0 ? D[0] : i == 1 ? D[1] : D[2], 0.0};
      if (i != c) {
        const int e = i + c - 1;  // 01, 02, 12
        v.re = e == 0 ? D[3] : e == 1 ? D[5] : D[7];
        v.im = e == 0 ? D[4] : e == 1 ? D[6] : D[8];
        if (i < c) v.im = -v.im;
      }
      const int q = s3i(i, c);
      double bv = B[0];
#pragma unroll
      for (int e = 1; e < 6; ++e) bv = q == e ? B[e] : bv;
      const int64_t os = (int64_t)km * 9 * V + (int64_t)(i * 3 + c) * V + x;
      const double b1 = mm * bv + (i == c ? kk : 0.0);
      if (op.W) {
        st(op.S0 + os, dd * v);
        op.S1[os] = b1;
      }
      if (op32.W) {
        op32.S0[os] = make_float2((float)(dd * v.re), (float)(dd * v.im));
        op32.S1[os] = (float)b1;
      }
    }
    if (scratch) {
      double *s = scratch + (int64_t)km * 7 * V + x;
      s[(int64_t)i * V] = (fabs(0.5 * C.inva2[i] * C.kin[0].im) * nU + fabs(C.so[0].im) * nDE) / fabs(tau);
      if (i < 2) {  // quark (i = 0), antiquark (i = 1): centre and deviation of the site term
        const double sg = i == 0 ? mm : -mm, kd = i == 0 ? kk : -kk, it = 1.0 / tau;
        double t[3], cen = 0.0, dev = 0.0;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          t[r] = (dd * D[r] + sg * B[s3i(r, r)] + kd) * it;
          cen += t[r] / 3.0;
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) dev += (t[r] - cen) * (t[r] - cen);
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const int p = e == 2 ? 4 : e + 1;  // B's 01, 02, 12
          const double re = (dd * D[3 + 2 * e] + sg * B[p]) * it, im = dd * D[4 + 2 * e] * it;
          dev += 2.0 * (re * re + im * im);
        }
        s[(int64_t)(3 + 2 * i) * V] = cen;
        s[(int64_t)(4 + 2 * i) * V] = sqrt(dev);
      }
    }
  }
}

// Enclosure of the spectrum of H by block Gershgorin discs from the planes
// of k_spin_prepare, per coefficient set (blockIdx.y): out[4*set] = {lo, hi}
// of the quark, then of the antiquark.  The last block of a set to finish
// reduces the partial rows (exact, order-independent); ticket[set] is zero
// between launches.  With tab (one set) it also makes the Chebyshev
// coefficients of the segments, a thread for each, and stores the bounds into
// the pinned host_bounds.  (40 steps of the recurrence by one thread took 18
// us, more than a stencil launch at 12^3.)
__global__ void __launch_bounds__(256) k_spin_bounds(Lat L, const double *__restrict__ scratch,
                                                     double *__restrict__ partials, unsigned *__restrict__ ticket,
                                                     double *__restrict__ out, double tau, ChebTab *__restrict__ tab,
                                                     double *__restrict__ host_bounds) {
  const int64_t V = L.V;
  const int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const double *s = scratch + (int64_t)blockIdx.y * 7 * V;
  double v[4] = {1e300, -1e300, 1e300, -1e300};
  bool bad = false;
  if (x < V) {
    double h = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) h += s[(int64_t)i * V + x] + s[(int64_t)i * V + nb(L, x, i, -1)];
#pragma unroll
    for (int sp = 0; sp < 2; ++sp) {
      const double cen = s[(int64_t)(3 + 2 * sp) * V + x], R = h + s[(int64_t)(4 + 2 * sp) * V + x];
      v[2 * sp] = cen - R;
      v[2 * sp + 1] = cen + R;
      bad = bad || !isfinite(cen) || !isfinite(R);
    }
  }
  __shared__ double sh[8][4];
  __shared__ int last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // a NaN would drop out of the minima and maxima: it becomes an infinite end
  if (bad) v[0] = v[2] = -INFINITY;
  double *row = partials + (int64_t)blockIdx.y * gridDim.x * 4;
  for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double w = __shfl_down_sync(0xffffffffu, v[q], o);
        v[q] = (q & 1) ? fmax(v[q], w) : fmin(v[q], w);
      }
    if (lane == 0)
#pragma unroll
      for (int q = 0; q < 4; ++q) sh[warp][q] = v[q];
    __syncthreads();
    if (threadIdx.x < 4) {
      const int q = threadIdx.x;
      double a = sh[0][q];
      for (int w = 1; w < 8; ++w) a = (q & 1) ? fmax(a, sh[w][q]) : fmin(a, sh[w][q]);
      if (pass == 0)
        row[(int64_t)blockIdx.x * 4 + q] = a;
      else
        out[4 * blockIdx.y + q] = sh[0][q] = a;
    }
    if (pass == 1) break;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      last = atomicAdd(ticket + blockIdx.y, 1u) == gridDim.x - 1;
      if (last) ticket[blockIdx.y] = 0u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    v[0] = v[2] = 1e300;
    v[1] = v[3] = -1e300;
    for (int64_t b = threadIdx.x; b < gridDim.x; b += blockDim.x)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double w = ((volatile double *)row)[b * 4 + q];
        v[q] = (q & 1) ? fmax(v[q], w) : fmin(v[q], w);
      }
  }
  if (!tab) return;
  __syncthreads();
  const int sp = threadIdx.x / kChebTab, k = threadIdx.x - sp * kChebTab;
  if (sp >= 2) return;
  const double lo = sh[0][2 * sp], hi = sh[0][2 * sp + 1];
  const ChebSegment g(tau, lo, hi);
  const cplx rho = g.rho(k);
  tab->step[k].c1[sp] = k == 0 ? cplx{0.0, 0.0} : rho * g.rho(k - 1);
  tab->step[k].c2[sp] = k == 0 ? g.inv_theta() : g.c2(rho);
  if (k != 0) return;
  tab->inv_theta[sp] = g.inv_theta();
  tab->lo[sp] = lo;
  tab->hi[sp] = hi;
  host_bounds[2 * sp] = lo;
  host_bounds[2 * sp + 1] = hi;
}

// ------------------------------------------------------------------ stencil
// One application of the operator (sign = +1: A^H, -1: A = 2 - A^H) to the 12
// columns, with the mode's vector work at the own site (MvMode); partial sums
// in one row per block: partials[(block*12 + column)*NQ + q].
//
// BATCH (MV_RHS, MV_RESC): the fields of the device table, each on its own
// coefficient set, blocks over (field, unit); MV_RHS adds the field's history
// to its start and keeps the added part in hnew, MV_RESC skips fields that
// have converged (skip_done).
struct SpinBatch {
  const BatchField *tab;
  int nf, nunits, order, skip_done, want_d;
};
template <int MODE, bool BATCH>
__global__ void __launch_bounds__(spin::kUnit *spin::kWarps, 2)
    k_cn_spin(Lat L, SpinOp op, double sign, MvArgs A, SpinBatch Bt, int *err, long long wait_cycles, int stall_load,
              bool early) {
  using namespace spin;
  constexpr int kAhead = Num<double>::kAhead;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem<double> &sm = *reinterpret_cast<Smem<double> *>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int V = (int)L.V;
  int u = (int)blockIdx.x;
  const BatchField *F = nullptr;
  if (BATCH) {
    int f;
    batch_item(Bt.nf, Bt.nunits, Bt.order, f, u);
    F = Bt.tab + f;
    if (MODE == MV_RESC && Bt.skip_done && batch_field_done(*F)) return;
    op.W += (int64_t)F->wblk * 81 * V;
    op.S0 += (int64_t)F->wblk * 9 * V;
    op.S1 += (int64_t)F->wblk * 9 * V;
    if (MODE == MV_RHS) {
      A.in = F->psi;
      A.out = F->b;
      A.out2 = F->x;
      A.hist[0] = A.hist[1] = A.hist[2] = A.hist[3] = nullptr;
      A.r32 = nullptr;
      if (F->hstart) {
        A.hist[0] = F->h1;
        A.hist[1] = F->h2;
        A.hist[2] = F->h3;
        A.hist[3] = F->h4;
        A.r32 = F->hnew;
        // the degree d - 1 extrapolation of d vectors
        const int d = F->h4 ? 4 : F->h3 ? 3 : F->h2 ? 2 : 1;
        A.hcoef[0] = d;
        A.hcoef[1] = d == 4 ? -6.0 : d == 3 ? -3.0 : -1.0;
        A.hcoef[2] = d == 4 ? 4.0 : 1.0;
        A.hcoef[3] = -1.0;
      }
    } else {
      A.in = F->x;
      A.bvec = F->b;
      A.r32 = F->r32;
      A.d32 = Bt.want_d ? F->dA : nullptr;
      A.inv_theta[0] = F->inv_theta[0];
      A.inv_theta[1] = F->inv_theta[1];
      A.partials = F->partials;
    }
  }
  init_barriers(sm);
  const int s = unit_start(L, u) + lane;
  const bool act = s < V;
  const int x = act ? s : V - 1;  // a valid site for the addresses of idle lanes
  cx<double> acc[4][3];
  double2 own[kAhead][4];
  const bool ok = apply<double>(L, op.W, op.S0, op.S1, A.in, x, warp, sm, err, wait_cycles, stall_load,
                                early, acc, own);
  cp_async_wait_all();
  constexpr int NQ = MODE == MV_T2 ? 5 : MODE == MV_RES2 ? 4 : MODE == MV_T ? 3
                   : (MODE == MV_RES || MODE == MV_V || MODE == MV_V2 || MODE == MV_RESC || MODE == MV_CH0 ||
                      MODE == MV_RESN)
                       ? 2
                       : 0;
  double qs[2][5];
#pragma unroll
  for (int sp = 0; sp < 2; ++sp)
#pragma unroll
    for (int k = 0; k < 5; ++k) qs[sp][k] = 0.0;
  if (ok && act) {
    constexpr bool kB = MODE == MV_RES || MODE == MV_RES2 || MODE == MV_RESC || MODE == MV_RESN || MODE == MV_CH0 ||
                        MODE == MV_CHK || MODE == MV_CHH;
    constexpr bool kCheb = MODE == MV_CHK || MODE == MV_CHH;
    constexpr bool kShadow = MODE == MV_V2 || MODE == MV_T2;
    cplx c1[2], c2[2];
#pragma unroll
    for (int sp = 0; sp < 2; ++sp) {
      if (kCheb) c1[sp] = A.cheb->step[A.step].c1[sp];
      if (kCheb) c2[sp] = A.cheb->step[A.step].c2[sp];
      if (MODE == MV_CH0) c2[sp] = A.cheb->inv_theta[sp];
    }
    // batches of three rows, the operands of the next batch loaded before
    // this one's results are stored
    cplx e1[2][3], e2[2][3], e3[2][3];
    float2 f[2][3][4];
    auto fetch = [&](int h) {
      const int64_t off = (int64_t)((h >> 1) * 36 + warp * 6 + 3 * (h & 1)) * V + x;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const int64_t o = off + (int64_t)r * V;
        if (kB) e1[h & 1][r] = ld_c(A.bvec + o);
        if (MODE == MV_V) e1[h & 1][r] = ld_c(A.in2 + o);
        if (kCheb) e2[h & 1][r] = ld(A.out + o);
        if (MODE == MV_CHH) e3[h & 1][r] = ld_c(A.in2 + o);
        if (kShadow) f[h & 1][r][0] = __ldca(A.sh32 + o);
        if (MODE == MV_RHS)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (A.hist[k]) f[h & 1][r][k] = A.hist[k][o];  // one of them may be r32
      }
    };
    fetch(0);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int sp = h >> 1, r0 = 3 * (h & 1);
      const int64_t off = (int64_t)(sp * 36 + warp * 6 + r0) * V + x;
      if (h < 3) fetch(h + 1);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const int64_t o = off + (int64_t)r * V;
        const int sr = (r0 + r) & 1, i = (r0 + r) >> 1;
        const double2 ow = own[(18 + i) % kAhead][2 * sp + sr];
        const cplx in = {ow.x, ow.y};
        const cplx ev = e1[h & 1][r];
        const float2 fv = f[h & 1][r][0];
        // (A^H - 1) in; the residuals subtract the input first, which leaves
        // the smaller numbers' rounding
        const cplx nv = {acc[2 * sp + sr][i].re, acc[2 * sp + sr][i].im};
        cplx y = in + nv;
        if (MODE == MV_PLAIN || MODE == MV_RHS)
          if (BATCH || sign < 0.0) y = in - nv;
        if (MODE == MV_PLAIN) {
          st(A.out + o, y);
        } else if (MODE == MV_RHS) {
          st(A.out + o, y);
          cplx dx = {0.0, 0.0};
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (A.hist[k]) {
              dx.re = fma(A.hcoef[k], (double)f[h & 1][r][k].x, dx.re);
              dx.im = fma(A.hcoef[k], (double)f[h & 1][r][k].y, dx.im);
            }
          st(A.out2 + o, 2.0 * y - in + dx);
          if (A.r32) A.r32[o] = make_float2((float)dx.re, (float)dx.im);
        } else if (MODE == MV_V || MODE == MV_V2) {
          st(A.out + o, y);
          const cplx rh = MODE == MV_V ? ev : cplx{(double)fv.x, (double)fv.y};
          cplx d = {0.0, 0.0};
          cmac_cj(d, rh, y);
          qs[sp][0] += d.re;
          qs[sp][1] += d.im;
        } else if (MODE == MV_T || MODE == MV_T2) {
          st(A.out + o, y);
          cplx d = {0.0, 0.0};
          cmac_cj(d, y, in);
          qs[sp][0] += d.re;
          qs[sp][1] += d.im;
          qs[sp][2] += norm2(y);
          if (MODE == MV_T2) {
            cplx t = {0.0, 0.0};
            cmac_cj(t, cplx{(double)fv.x, (double)fv.y}, y);
            qs[sp][3] += t.re;
            qs[sp][4] += t.im;
          }
        } else {
          const cplx rv = (ev - in) - nv;
          if (MODE == MV_RES) {
            st(A.out + o, rv);
            st(A.out2 + o, rv);
            st(A.out3 + o, rv);
          } else if (MODE == MV_RES2) {
            const float2 g = make_float2((float)rv.re, (float)rv.im);
            st(A.out + o, rv);
            A.sh32[o] = g;
            st(A.out3 + o, rv);
            cplx d = {0.0, 0.0};
            cmac_cj(d, cplx{(double)g.x, (double)g.y}, rv);
            qs[sp][2] += d.re;
            qs[sp][3] += d.im;
          } else if (MODE == MV_RESC) {
            A.r32[o] = make_float2((float)rv.re, (float)rv.im);
            if (A.d32) {
              const cplx dv = rv * A.inv_theta[sp];
              A.d32[o] = make_float2((float)dv.re, (float)dv.im);
            }
          } else if (MODE == MV_CH0) {
            st(A.out + o, in + c2[sp] * rv);
          } else if (kCheb) {
            const cplx xn = in + c1[sp] * (in - e2[h & 1][r]) + c2[sp] * rv;
            st(A.out + o, xn);
            if (MODE == MV_CHH) {
              const cplx t = xn - (2.0 * ev - e3[h & 1][r]);
              A.r32[o] = make_float2((float)t.re, (float)t.im);
            }
          }
          if (!kCheb) {
            qs[sp][0] += norm2(rv);
            qs[sp][1] += norm2(ev);
          }
        }
      }
    }
  }
  if constexpr (NQ > 0) {
#pragma unroll
    for (int sp = 0; sp < 2; ++sp)
#pragma unroll
      for (int k = 0; k < NQ; ++k) {
        double v = qs[sp][k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) A.partials[((int64_t)u * CN_COLS + sp * 6 + warp) * NQ + k] = v;
      }
  }
}

// ------------------------------------------------------------------ host
void launch_spin_prepare(Lat L, const CnCoef &C, const CnCoef *Cm, int nm, double tau, const double2 *U,
                         const double *E, const SpinOp &op, const SpinOp32 &op32, double *scratch, cudaStream_t st) {
  const unsigned grid = (unsigned)((L.V + kPrepSites - 1) / kPrepSites);
  k_spin_prepare<<<grid, kPrepSites * 3, 0, st>>>(L, C, Cm, nm, tau, U, E, op, op32, scratch);
}

void launch_spin_bounds(Lat L, int nm, const double *scratch, double *partials, unsigned *ticket, double *out,
                        cudaStream_t st, double tau, ChebTab *tab, double *host_bounds) {
  k_spin_bounds<<<dim3((unsigned)((L.V + 255) / 256), (unsigned)nm), 256, 0, st>>>(L, scratch, partials, ticket, out,
                                                                                  tau, tab, host_bounds);
}

bool cn_spin_applicable(const Lat &L) { return L.V <= 0x7fffffffLL; }

void launch_cn_spin(int mode, Lat L, const SpinOp &op, double sign, const MvArgs &a, bool early, int *err,
                    cudaStream_t st, long long wait_cycles, int stall_load) {
  using namespace spin;
  const unsigned grid = (unsigned)((L.V + kUnit - 1) / kUnit);
  auto go = [&](auto kern) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem<double>));
    launch_pdl(kern, grid, kUnit * kWarps, sizeof(Smem<double>), st, L, op, sign, a, SpinBatch{}, err, wait_cycles,
               stall_load, early);
  };
  switch (mode) {
    case MV_PLAIN: go(k_cn_spin<MV_PLAIN, false>); break;
    case MV_RHS: go(k_cn_spin<MV_RHS, false>); break;
    case MV_RES: go(k_cn_spin<MV_RES, false>); break;
    case MV_V: go(k_cn_spin<MV_V, false>); break;
    case MV_T: go(k_cn_spin<MV_T, false>); break;
    case MV_RESC: go(k_cn_spin<MV_RESC, false>); break;
    case MV_T2: go(k_cn_spin<MV_T2, false>); break;
    case MV_RES2: go(k_cn_spin<MV_RES2, false>); break;
    case MV_V2: go(k_cn_spin<MV_V2, false>); break;
    case MV_RESN: go(k_cn_spin<MV_RESN, false>); break;
    case MV_CH0: go(k_cn_spin<MV_CH0, false>); break;
    case MV_CHK: go(k_cn_spin<MV_CHK, false>); break;
    default: go(k_cn_spin<MV_CHH, false>); break;
  }
}

void launch_batch_spin(int mode, int order, Lat L, const SpinOp &op, const BatchField *tab, int nfields, int skip_done,
                       bool want_d, int *err, cudaStream_t st, long long wait_cycles) {
  using namespace spin;
  const int nunits = (int)((L.V + kUnit - 1) / kUnit);
  const SpinBatch bt{tab, nfields, nunits, order, skip_done, want_d ? 1 : 0};
  auto go = [&](auto kern) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem<double>));
    kern<<<(unsigned)nunits * (unsigned)nfields, kUnit * kWarps, sizeof(Smem<double>), st>>>(
        L, op, 1.0, MvArgs{}, bt, err, wait_cycles, -1, false);
  };
  if (mode == MV_RHS)
    go(k_cn_spin<MV_RHS, true>);
  else
    go(k_cn_spin<MV_RESC, true>);
}

}  // namespace nrq
