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
// all six warps (cp.async, three buffers, one mbarrier per neighbour: a warp
// that sees the matrices of neighbour n landed knows that every warp has
// left neighbour n - 2, so the third buffer is free), and the spinors go
// straight to registers two steps ahead.  Nothing depends on the lattice's
// shape: each lane reads its own neighbours' addresses, so one kernel serves
// rows of any length, and small lattices get one block per 32 sites.
//
// Bound: 64^3, the solver's step (four vector streams, 6.1 KB a site): 0.25 ms
// at the copy rate, 0.21 ms at the FP64 rate that FMAs with distinct operands
// reach (49 of 64 a clock and SM).  It takes 0.41 ms: twelve warps an SM (166
// registers) hide the loads only in part, a block spends a fifth of its time
// before its first product and in its epilogue, and the loads alone take 0.31
// ms (the launch without its products).  24^3: 28 us, 12^3: 12 us.
//
// Every mbarrier wait is bounded (wait_cycles); on expiry the thread records
// NRQ_ERR_TIMEOUT in *err and its warp skips the remaining work.  stall_load
// >= 0 makes every block stop staging before that neighbour, so that the
// wait for it runs out: the host's test of the timeout path (nothing faults;
// the context stays usable).  A block waits for its own copies before it
// exits.
#include <algorithm>

#include "../../include/nrqcd_b200.h"
#include "nrq_eigen.cuh"
#include "nrq_kernels.cuh"
#include "stage.cuh"

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
// from the links and the electric field: W (81 planes of V complex per set,
// (I*3 + m)*9 + row*3 + column), S0 (9 planes, row*3 + column), S1 (9 real
// planes) and, for the spectral enclosure, seven real planes per set: the
// norm bound of the block to x + I (I = 0..2), and centre and deviation of
// the site term of the hermitian H (A^H = 1 + i tau H) for quark and
// antiquark.  One thread per site and direction; the Darwin and magnetic
// matrices are sums over directions, exchanged through shared memory.  64^3:
// 280 us (254 registers, 8 warps an SM; the FP64 pipe 28 % active), 12^3: 10 us.
__global__ void __launch_bounds__(kPrepSites * 3) k_spin_prepare(Lat L, CnCoef C1, const CnCoef *__restrict__ Cm,
                                                                int nm, double tau, const double2 *__restrict__ U,
                                                                const double *__restrict__ E, SpinOp op,
                                                                double *__restrict__ scratch) {
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
    if (!log_unitary(P, H)) log_jacobi(P, H);
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
    double2 *W = op.W + (int64_t)km * 81 * V + (int64_t)(i * 27) * V + x;
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
        st(W + (int64_t)(r * 3 + c) * V, a);
        st(W + (int64_t)(9 + r * 3 + c) * V, b);
        st(W + (int64_t)(18 + r * 3 + c) * V, o);
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
      st(op.S0 + (int64_t)km * 9 * V + (int64_t)(i * 3 + c) * V + x, dd * v);
      op.S1[(int64_t)km * 9 * V + (int64_t)(i * 3 + c) * V + x] = mm * bv + (i == c ? kk : 0.0);
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
// between launches.
__global__ void __launch_bounds__(256) k_spin_bounds(Lat L, const double *__restrict__ scratch,
                                                     double *__restrict__ partials, unsigned *__restrict__ ticket,
                                                     double *__restrict__ out) {
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
        out[4 * blockIdx.y + q] = a;
    }
    if (pass == 1) return;
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
}

// ------------------------------------------------------------------ stencil
namespace {
constexpr int kUnit = 32;   // sites of a block, one per lane
constexpr int kWarps = 6;   // one propagator column of both species each
// Spinor operands in registers: this step's and the next three's; matrices
// staged two neighbours ahead.  (64^3, a coupled step: 4.16 ms with the next
// two and one neighbour, 4.09 with the next three, 3.98 with both.  Prefetches
// to L2, of the epilogue's operands or of later units', cost 2-20 %; a
// persistent form with the next unit's first loads issued early 10 %.)
constexpr int kAhead = 4;
constexpr int kWBufs = 5;

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
// arrives on bar once this thread's copies so far have landed
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// acc += +-(w or conj(w)) p in halves: the products with Re w, then those
// with Im w, so that consecutive FMAs share an operand register (an FP64 FMA
// with three fresh operands issues every 2.7 cycles, with one reused 2.3)
template <int S>
__device__ __forceinline__ void smac_re(cplx &acc, const double2 w, const double2 p) {
  const double wr = S > 0 ? w.x : -w.x;
  acc.re = fma(wr, p.x, acc.re);
  acc.im = fma(wr, p.y, acc.im);
}
template <int S, bool CJ>
__device__ __forceinline__ void smac_im(cplx &acc, const double2 w, const double2 p) {
  const double wi = (S > 0) == !CJ ? w.y : -w.y;
  acc.re = fma(-wi, p.y, acc.re);
  acc.im = fma(wi, p.x, acc.im);
}
template <int SA, int SB, bool CJ>
__device__ __forceinline__ void smac2(const double2 w, cplx &a, const double2 p, cplx &b, const double2 q) {
  smac_re<SA>(a, w, p);
  smac_re<SB>(b, w, q);
  smac_im<SA, CJ>(a, w, p);
  smac_im<SB, CJ>(b, w, q);
}
template <int SA, int SB, bool CJ>
__device__ __forceinline__ void smac4(const double2 w, cplx &a, const double2 p, cplx &b, const double2 q, cplx &c,
                                      const double2 r, cplx &d, const double2 s) {
  smac_re<SA>(a, w, p);
  smac_re<SA>(b, w, q);
  smac_re<SB>(c, w, r);
  smac_re<SB>(d, w, s);
  smac_im<SA, CJ>(a, w, p);
  smac_im<SA, CJ>(b, w, q);
  smac_im<SB, CJ>(c, w, r);
  smac_im<SB, CJ>(d, w, s);
}

// One step: direction I, forward (B = false) or backward, one input colour.
// m[t][i]: entry (i, j) of matrix t, backward entry (j, i) of the
// neighbour's; q = the input entries (quark spin 0, 1, antiquark spin 0, 1);
// a[species*2 + spin][i] the output colours.
template <int I, bool B>
__device__ __forceinline__ void spin_products(cplx (&a)[4][3], const double2 (&m)[3][3], const double2 (&q)[4]) {
  constexpr int S = B ? -1 : 1;
  // signs of the off-diagonal blocks (upper right, lower left), I < 2
  constexpr int S01 = I == 0 ? 1 : S, S10 = I == 0 ? -1 : S;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (I < 2) smac2<S, -S, B>(m[0][i], a[0][i], q[0], a[3][i], q[3]);
    if (I < 2) smac2<S, -S, B>(m[1][i], a[1][i], q[1], a[2][i], q[2]);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (I < 2) {
      smac4<S01, S10, B>(m[2][i], a[0][i], q[1], a[2][i], q[3], a[1][i], q[0], a[3][i], q[2]);
    } else {
      smac4<S, -S, B>(m[0][i], a[0][i], q[0], a[1][i], q[1], a[2][i], q[2], a[3][i], q[3]);
      smac2<S, S, B>(m[B ? 1 : 2][i], a[0][i], q[1], a[2][i], q[3]);
      smac2<S, S, B>(m[B ? 2 : 1][i], a[1][i], q[0], a[3][i], q[2]);
    }
  }
}

// First site of work unit u.  Where every row holds whole units (nx a
// multiple of 32) and ny, nz are multiples of 8, the units are taken in
// blocks of 8 x 8 rows (x fastest, then y and z within the block), so that
// the +-y and +-z neighbours of a unit are read within a few hundred units
// of it, while L2 still holds them (in site order the +-z neighbours are a
// plane apart: 100 MB of loads at 128^3); otherwise in site order.
__device__ __forceinline__ int unit_start(const Lat &L, int u) {
  const int nx = (int)L.nx, ny = (int)L.ny, nz = (int)L.nz;
  if ((nx & 31) || (ny & 7) || (nz & 7)) return u * kUnit;
  const int nxu = nx >> 5;
  int t = u / nxu;
  const int cx = (u - t * nxu) << 5;
  const int yi = t & 7, zi = (t >> 3) & 7;
  t >>= 6;
  const int nby = ny >> 3;
  const int bz = t / nby, by = t - bz * nby;
  return cx + nx * ((by << 3) + yi + ny * ((bz << 3) + zi));
}

// the six periodic neighbours (+x,-x,+y,-y,+z,-z) of site x (V < 2^31)
__device__ __forceinline__ void neighbours(const Lat &L, int x, int (&nbr)[6]) {
  const int nx = (int)L.nx, ny = (int)L.ny, nz = (int)L.nz, nxy = nx * ny, V = (int)L.V;
  const int t = x / nx, px = x - t * nx, pz = t / ny, py = t - pz * ny;
  nbr[0] = px + 1 < nx ? x + 1 : x + 1 - nx;
  nbr[1] = px > 0 ? x - 1 : x - 1 + nx;
  nbr[2] = py + 1 < ny ? x + nx : x + nx - nxy;
  nbr[3] = py > 0 ? x - nx : x - nx + nxy;
  nbr[4] = pz + 1 < nz ? x + nxy : x + nxy - V;
  nbr[5] = pz > 0 ? x - nxy : x - nxy + V;
}

struct SpinSmem {
  double2 w[kWBufs][27][kUnit];
  double2 s0[9][kUnit];
  double s1[9][kUnit];
  uint64_t full[6];  // the matrices of neighbour n (and, n = 0, the site term) landed
};

// y = A^H in of the warp's column c at the lane's site x: acc[species*2 +
// spin][colour]; own[colour] = the input at x itself.  Returns false where a
// wait ran out.
__device__ __forceinline__ bool spin_apply(const Lat &L, const double2 *__restrict__ W, const double2 *__restrict__ S0,
                                           const double *__restrict__ S1, const double2 *__restrict__ in, int x, int c,
                                           SpinSmem &sm, int *err, long long wait_cycles, int stall_load,
                                           cplx (&acc)[4][3], double2 (&own)[kAhead][4]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t V = L.V;
  int nbr[6];
  neighbours(L, x, nbr);
  auto stage = [&](int n) {
    if (stall_load >= 0 && n >= stall_load) return;
    const double2 *w = W + (int64_t)((n >> 1) * 27) * V + ((n & 1) ? nbr[n] : x);
    for (int p = warp; p < 27; p += kWarps) cp_async16(smem_u32(&sm.w[n % kWBufs][p][lane]), w + (int64_t)p * V);
    if (n == 0)
      for (int p = warp; p < 9; p += kWarps) {
        cp_async16(smem_u32(&sm.s0[p][lane]), S0 + (int64_t)p * V + x);
        cp_async8(smem_u32(&sm.s1[p][lane]), S1 + (int64_t)p * V + x);
      }
    cp_async_arrive(&sm.full[n]);
  };
  // operand of step t: neighbour t / 3 (18 and on: the site itself), input
  // colour t % 3
  const double2 *pq = in + (int64_t)(6 * c) * V, *pa = in + (int64_t)(36 + 6 * c) * V;
  auto load = [&](int t, double2 (&q)[4]) {
    const int y = t < 18 ? nbr[t / 3] : x;
    const int64_t o = (int64_t)(2 * (t % 3)) * V + y;
    q[0] = __ldg(pq + o);
    q[1] = __ldg(pq + o + V);
    q[2] = __ldg(pa + o);
    q[3] = __ldg(pa + o + V);
  };
  stage(0);
#pragma unroll
  for (int t = 0; t < kAhead - 1; ++t) load(t, own[t]);
  stage(1);
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int i = 0; i < 3; ++i) acc[s][i] = {0.0, 0.0};
  bool ok = true;
#pragma unroll
  for (int n = 0; n < 6; ++n) {
    if (ok && !mbar_try_wait(&sm.full[n], 0)) {
      const long long t0 = clock64();
      while (ok && !mbar_try_wait(&sm.full[n], 0)) ok = clock64() - t0 <= wait_cycles;
      if (!ok) record_timeout(err, 5, 0, n);
    }
    if (!__all_sync(0xffffffffu, ok)) return false;
    // every warp issued its copies of n when it entered neighbour n - 2, so
    // all have left n - 3, whose buffer n + 2 takes
    if (n + 2 < 6) stage(n + 2);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int t = 3 * n + j;
      if (t + kAhead - 1 < 21) load(t + kAhead - 1, own[(t + kAhead - 1) % kAhead]);
      double2 m[3][3];
#pragma unroll
      for (int t3 = 0; t3 < 3; ++t3)
#pragma unroll
        for (int i = 0; i < 3; ++i) m[t3][i] = sm.w[n % kWBufs][t3 * 9 + ((n & 1) ? 3 * j + i : 3 * i + j)][lane];
      const double2 (&q)[4] = own[t % kAhead];
      if (n == 0) spin_products<0, false>(acc, m, q);
      if (n == 1) spin_products<0, true>(acc, m, q);
      if (n == 2) spin_products<1, false>(acc, m, q);
      if (n == 3) spin_products<1, true>(acc, m, q);
      if (n == 4) spin_products<2, false>(acc, m, q);
      if (n == 5) spin_products<2, true>(acc, m, q);
    }
  }
  // the site term
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double2 (&q)[4] = own[(18 + j) % kAhead];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      acc[s][j].re += q[s].x;
      acc[s][j].im += q[s].y;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double2 d = sm.s0[i * 3 + j][lane];
      const double b = sm.s1[i * 3 + j][lane];
      const double gq = d.x + b, ga = d.x - b;
#pragma unroll
      for (int s = 0; s < 4; ++s) {  // += i (g + i d.y) q
        const double g = s < 2 ? gq : ga;
        acc[s][i].re = fma(-g, q[s].y, fma(-d.y, q[s].x, acc[s][i].re));
        acc[s][i].im = fma(g, q[s].x, fma(-d.y, q[s].y, acc[s][i].im));
      }
    }
  }
  return true;
}
}  // namespace

// One application of the operator (sign = +1: A^H, -1: A = 2 - A^H) to the 12
// columns, with the mode's vector work at the own site (MvMode); partial sums
// in one row per block: partials[(block*12 + column)*NQ + q].
template <int MODE>
__global__ void __launch_bounds__(kUnit *kWarps, 2)
    k_cn_spin(Lat L, SpinOp op, double sign, MvArgs A, int *err, long long wait_cycles, int stall_load) {
  extern __shared__ __align__(16) unsigned char raw_[];
  SpinSmem &sm = *reinterpret_cast<SpinSmem *>(raw_);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < 6) mbar_init(&sm.full[threadIdx.x], kUnit * kWarps);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  const int V = (int)L.V;
  const int s = unit_start(L, (int)blockIdx.x) + lane;
  const bool act = s < V;
  const int x = act ? s : V - 1;  // a valid site for the addresses of idle lanes
  cplx acc[4][3];
  double2 own[kAhead][4];
  const bool ok = spin_apply(L, op.W, op.S0, op.S1, A.in, x, warp, sm, err, wait_cycles, stall_load, acc, own);
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
        if (kB) e1[h & 1][r] = ldg(A.bvec + o);
        if (MODE == MV_V) e1[h & 1][r] = ldg(A.in2 + o);
        if (kCheb) e2[h & 1][r] = ld(A.out + o);
        if (MODE == MV_CHH) e3[h & 1][r] = ldg(A.in2 + o);
        if (kShadow) f[h & 1][r][0] = __ldg(A.sh32 + o);
        if (MODE == MV_RHS)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (A.hist[k]) f[h & 1][r][k] = __ldg(A.hist[k] + o);
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
        cplx y = acc[2 * sp + sr][i];
        if (MODE == MV_PLAIN || MODE == MV_RHS)
          if (sign < 0.0) y = 2.0 * in - y;
        if (MODE == MV_PLAIN) {
          st(A.out + o, y);
        } else if (MODE == MV_RHS) {
          st(A.out + o, y);
          cplx x0 = 2.0 * y - in;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (A.hist[k]) {
              x0.re = fma(A.hcoef[k], (double)f[h & 1][r][k].x, x0.re);
              x0.im = fma(A.hcoef[k], (double)f[h & 1][r][k].y, x0.im);
            }
          st(A.out2 + o, x0);
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
          const cplx rv = ev - y;
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
        if (lane == 0) A.partials[((int64_t)blockIdx.x * CN_COLS + sp * 6 + warp) * NQ + k] = v;
      }
  }
}

// The Chebyshev coefficients of the segments the bounds give (lo, hi of
// quark and antiquark), A^H = 1 + i tau H: theta its centre, delta its half
// length, sigma = theta / delta, rho_0 = 1 / sigma, rho_{k+1} = 1 / (2 sigma
// - rho_k); x_1 = x_0 + r_0 / theta, then x_{k+1} = x_k + c1 (x_k - x_{k-1})
// + c2 r_k with c1 = rho_k rho_{k-1}, c2 = 2 rho_k / delta.  One thread per
// species; the bounds also go to the pinned host_bounds.
__global__ void k_cheb_tab(const double *__restrict__ bounds, double tau, ChebTab *__restrict__ tab,
                           double *__restrict__ host_bounds) {
  const int sp = threadIdx.x;
  if (sp >= 2) return;
  const double lo = bounds[2 * sp], hi = bounds[2 * sp + 1];
  tab->lo[sp] = lo;
  tab->hi[sp] = hi;
  host_bounds[2 * sp] = lo;
  host_bounds[2 * sp + 1] = hi;
  const cplx one = {1.0, 0.0};
  const cplx theta = {1.0, tau * 0.5 * (lo + hi)};
  const cplx delta = {0.0, fmax(fabs(tau) * 0.5 * (hi - lo), 1e-14)};
  const cplx sigma = cdiv(theta, delta);
  tab->inv_theta[sp] = cdiv(one, theta);
  cplx rho = cdiv(one, sigma);
  tab->step[0].c1[sp] = {0.0, 0.0};
  tab->step[0].c2[sp] = tab->inv_theta[sp];
  for (int k = 1; k < kChebTab; ++k) {
    const cplx rn = cdiv(one, 2.0 * sigma - rho);
    tab->step[k].c1[sp] = rn * rho;
    tab->step[k].c2[sp] = cdiv(2.0 * rn, delta);
    rho = rn;
  }
}

// ------------------------------------------------------------------ host
void launch_spin_prepare(Lat L, const CnCoef &C, const CnCoef *Cm, int nm, double tau, const double2 *U,
                         const double *E, const SpinOp &op, double *scratch, cudaStream_t st) {
  const unsigned grid = (unsigned)((L.V + kPrepSites - 1) / kPrepSites);
  k_spin_prepare<<<grid, kPrepSites * 3, 0, st>>>(L, C, Cm, nm, tau, U, E, op, scratch);
}

void launch_spin_bounds(Lat L, int nm, const double *scratch, double *partials, unsigned *ticket, double *out,
                        cudaStream_t st) {
  k_spin_bounds<<<dim3((unsigned)((L.V + 255) / 256), (unsigned)nm), 256, 0, st>>>(L, scratch, partials, ticket, out);
}

void launch_cheb_tab(const double *bounds, double tau, ChebTab *tab, double *host_bounds, cudaStream_t st) {
  k_cheb_tab<<<1, 32, 0, st>>>(bounds, tau, tab, host_bounds);
}

bool cn_spin_applicable(const Lat &L) { return L.V <= 0x7fffffffLL; }

void launch_cn_spin(int mode, Lat L, const SpinOp &op, double sign, const MvArgs &a, int *err, cudaStream_t st,
                    long long wait_cycles, int stall_load) {
  const unsigned grid = (unsigned)((L.V + kUnit - 1) / kUnit);
  auto go = [&](auto kern) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SpinSmem));
    kern<<<grid, kUnit * kWarps, sizeof(SpinSmem), st>>>(L, op, sign, a, err, wait_cycles, stall_load);
  };
  switch (mode) {
    case MV_PLAIN: go(k_cn_spin<MV_PLAIN>); break;
    case MV_RHS: go(k_cn_spin<MV_RHS>); break;
    case MV_RES: go(k_cn_spin<MV_RES>); break;
    case MV_V: go(k_cn_spin<MV_V>); break;
    case MV_T: go(k_cn_spin<MV_T>); break;
    case MV_RESC: go(k_cn_spin<MV_RESC>); break;
    case MV_T2: go(k_cn_spin<MV_T2>); break;
    case MV_RES2: go(k_cn_spin<MV_RES2>); break;
    case MV_V2: go(k_cn_spin<MV_V2>); break;
    case MV_RESN: go(k_cn_spin<MV_RESN>); break;
    case MV_CH0: go(k_cn_spin<MV_CH0>); break;
    case MV_CHK: go(k_cn_spin<MV_CHK>); break;
    default: go(k_cn_spin<MV_CHH>); break;
  }
}

}  // namespace nrq
