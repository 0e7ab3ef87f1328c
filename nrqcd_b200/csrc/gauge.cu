// Gauge-field kernels of the hot path (FP64):
//   - leapfrog link update  U <- exp(i dt E^a T^a) U   (gauge:2118-2140)
//   - leapfrog E update from the U/D staples           (gauge:2147-2259)
//   - energy (gauge:1769-1817) and both Gauss-law measures (gauge:1480-1531,
//     :724-768) as deterministic two-stage FP64 reductions
//   - layout transposes between the reference's Fortran arrays and the
//     structure-of-arrays planes held in HBM
//   - the device part of the transverse-polarised initial condition
//     (gauge:1263-1446): momentum-space construction between two FFTs.
// Paths are those of the reference project (src/gaugeconfiguration_su3.f90
// abbreviated "gauge").
#include "nrq_kernels.cuh"
#include "pdl.cuh"

namespace nrq {

// ------------------------------------------------------------ layout moves
// Fortran links(3,3,3,V): element (row, col, dir, site) at ((site*3+dir)*3+col)*3+row
__global__ void k_links_f2soa(const double2 *__restrict__ f, double2 *__restrict__ U, int64_t V) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= V) return;
  const double2 *src = f + s * 27;
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = 0; r < 3; ++r) U[(int64_t)(d * 9 + r * 3 + c) * V + s] = src[(d * 3 + c) * 3 + r];
}
__global__ void k_links_soa2f(const double2 *__restrict__ U, double2 *__restrict__ f, int64_t V) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= V) return;
  double2 *dst = f + s * 27;
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = 0; r < 3; ++r) dst[(d * 3 + c) * 3 + r] = U[(int64_t)(d * 9 + r * 3 + c) * V + s];
}
// Fortran efield(8,3,V): (site*3+dir)*8 + a
__global__ void k_efield_f2soa(const double *__restrict__ f, double *__restrict__ E, int64_t V) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= V) return;
#pragma unroll
  for (int k = 0; k < 24; ++k) E[(int64_t)k * V + s] = f[s * 24 + k];
}
__global__ void k_efield_soa2f(const double *__restrict__ E, double *__restrict__ f, int64_t V) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= V) return;
#pragma unroll
  for (int k = 0; k < 24; ++k) f[s * 24 + k] = E[(int64_t)k * V + s];
}

__global__ void k_cold(double2 *__restrict__ U, double *__restrict__ E, int64_t V) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= V) return;
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int k = 0; k < 9; ++k)
      U[(int64_t)(d * 9 + k) * V + s] = make_double2((k % 4 == 0) ? 1.0 : 0.0, 0.0);
#pragma unroll
  for (int k = 0; k < 24; ++k) E[(int64_t)k * V + s] = 0.0;
}

// ------------------------------------------------------------ leapfrog
constexpr int kLinkSites = 32, kForceSites = 16;  // consecutive sites of a block
// One thread per link.  64^3: 62 us, of which the traffic takes 43; the
// exponential's chain of FMAs at 12 warps an SM (154 registers) the rest (128
// registers with a little spilled: 3 % faster there, 6 % slower at 30x21x14).
__global__ void __launch_bounds__(3 * kLinkSites) k_update_links(Lat L, double2 *__restrict__ U,
                                                                const double *__restrict__ E, double dt) {
  const int d = (int)threadIdx.x / kLinkSites;
  const int64_t s = (int64_t)blockIdx.x * kLinkSites + threadIdx.x % kLinkSites;
  pdl_wait();
  pdl_trigger();
  if (s >= L.V) return;
  const int64_t V = L.V;
  double al[8];
#pragma unroll
  for (int a = 0; a < 8; ++a) al[a] = __ldca(E + (int64_t)(d * 8 + a) * V + s) * dt;
  const m3 u = load_link_c(U, V, s, d);
  const m3 G = expi_herm(algebra_matrix(al));
  store_link(U, V, s, d, mul(G, u));
}

// The force on link (x, i) from its four staples, one thread for each of the
// two directions k != i: two staples, U_i(x) times their sum, and the traces,
// which the lane pair adds.  The three directions of a block's sites run side
// by side and read the links they share through the SM's L1.
// Bound: latency of the loads (12 matrices a thread, FP64 pipe a third
// active).  64^3: 142 us at 15 warps an SM (one thread per link, three
// matrices live, 12 warps: 147; one thread per row of a link, 24 warps, three
// times the load instructions: 230); a step at 30x21x14 10.1 -> 7 us, with
// the launch of the second kernel hidden.
__global__ void __launch_bounds__(6 * kForceSites, 5) k_update_efield(Lat L, const double2 *U, double *E, double dt) {
  pdl_wait();
  pdl_trigger();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, kk = lane >> 4;
  const int i = w % 3;
  const int64_t V = L.V, x0 = (int64_t)blockIdx.x * kForceSites + (w / 3) * 16 + (lane & 15);
  const bool act = x0 < V;
  const int64_t s = act ? x0 : V - 1;
  const int k = kk + (kk >= i ? 1 : 0);
  const double r = L.a0 / L.a[k];
  const double coef = dt * (r * r);
  const int64_t xpi = nb(L, s, i, +1), xpk = nb(L, s, k, +1), xmk = nb(L, s, k, -1), xpimk = nb(L, xmk, i, +1);
  // U staple  U_k(x+i) U_i(x+k)^+ U_k(x)^+
  m3 t = mul_nd(mul_nd(load_link_c(U, V, xpi, k), load_link_c(U, V, xpk, i)), load_link_c(U, V, s, k));
  {  // D staple  U_k(x+i-k)^+ U_i(x-k)^+ U_k(x-k)
    const m3 d = mul_dn(mul(load_link_c(U, V, xmk, i), load_link_c(U, V, xpimk, k)), load_link_c(U, V, xmk, k));
#pragma unroll
    for (int m = 0; m < 9; ++m) t.e[m] = t.e[m] + d.e[m];
  }
  t = mul(load_link_c(U, V, s, i), t);
  cplx tr[8];
  traces_with_generators(t, tr);
  double f[8];
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    f[a] = coef * tr[a].im;
    f[a] += __shfl_xor_sync(0xffffffffu, f[a], 16);
  }
  if (!act) return;
  double *e = E + (int64_t)(i * 8 + 4 * kk) * V + s;  // four coordinates a lane
#pragma unroll
  for (int a = 0; a < 4; ++a) e[(int64_t)a * V] -= 2.0 * (kk ? f[4 + a] : f[a]);
}

// the two kernels of a leapfrog step, in either order
void launch_update_links(Lat L, double2 *U, const double *E, double dt, cudaStream_t st) {
  launch_pdl(k_update_links, (unsigned)((L.V + kLinkSites - 1) / kLinkSites), 3 * kLinkSites, 0, st, L, U, E, dt);
}
void launch_update_efield(Lat L, const double2 *U, double *E, double dt, cudaStream_t st) {
  launch_pdl(k_update_efield, (unsigned)((L.V + kForceSites - 1) / kForceSites), 6 * kForceSites, 0, st, L, U, E, dt);
}

// ------------------------------------------------------------ FP32 links
// Precision form of the leapfrog: links stored in FP32 (27 float2 planes,
// the same plane order), Ẽ kept in FP64.  Staple products run in FP32; their
// sum over k, the force projection and Ẽ accumulate in FP64; the group
// exponential is FP64 and the product exp(iẼdt)·U FP32.  FP64
// reunitarisation (k_reunitarise) restores det U = 1 and U U^+ = 1.
struct m3f {
  float2 e[9];
};
__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ void cmacf_(float2 &acc, float2 a, float2 b) {
  acc.x = fmaf(a.x, b.x, fmaf(-a.y, b.y, acc.x));
  acc.y = fmaf(a.x, b.y, fmaf(a.y, b.x, acc.y));
}
// acc += a * conj(b)
__device__ __forceinline__ void cmacf_nc(float2 &acc, float2 a, float2 b) {
  acc.x = fmaf(a.x, b.x, fmaf(a.y, b.y, acc.x));
  acc.y = fmaf(a.y, b.x, fmaf(-a.x, b.y, acc.y));
}
__device__ __forceinline__ m3f load_link32(const float2 *__restrict__ U, int64_t V, int64_t s, int d) {
  m3f m;
  const float2 *p = U + (int64_t)d * 9 * V + s;
#pragma unroll
  for (int k = 0; k < 9; ++k) m.e[k] = __ldg(p + k * V);
  return m;
}
__device__ __forceinline__ m3f mulf(const m3f &a, const m3f &b) {
  m3f r;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      float2 acc = cmulf(a.e[i * 3], b.e[j]);
      cmacf_(acc, a.e[i * 3 + 1], b.e[3 + j]);
      cmacf_(acc, a.e[i * 3 + 2], b.e[6 + j]);
      r.e[i * 3 + j] = acc;
    }
  return r;
}
// a * b^+
__device__ __forceinline__ m3f mulf_nd(const m3f &a, const m3f &b) {
  m3f r;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      float2 acc = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < 3; ++k) cmacf_nc(acc, a.e[i * 3 + k], b.e[j * 3 + k]);
      r.e[i * 3 + j] = acc;
    }
  return r;
}
// a^+ * b
__device__ __forceinline__ m3f mulf_dn(const m3f &a, const m3f &b) {
  m3f r;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      float2 acc = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        // conj(a[k][i]) * b[k][j]
        const float2 x = a.e[k * 3 + i], y = b.e[k * 3 + j];
        acc.x = fmaf(x.x, y.x, fmaf(x.y, y.y, acc.x));
        acc.y = fmaf(x.x, y.y, fmaf(-x.y, y.x, acc.y));
      }
      r.e[i * 3 + j] = acc;
    }
  return r;
}

__global__ void __launch_bounds__(128) k_update_links32(Lat L, float2 *__restrict__ U, const double *__restrict__ E,
                                                        double dt) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= L.V) return;
  const int64_t V = L.V;
#pragma unroll 1
  for (int d = 0; d < 3; ++d) {
    double al[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) al[a] = __ldg(E + (int64_t)(d * 8 + a) * V + s) * dt;
    const m3 G = expi_herm(algebra_matrix(al));
    m3f g;
#pragma unroll
    for (int k = 0; k < 9; ++k) g.e[k] = make_float2((float)G.e[k].re, (float)G.e[k].im);
    const m3f r = mulf(g, load_link32(U, V, s, d));
    float2 *p = U + (int64_t)d * 9 * V + s;
#pragma unroll
    for (int k = 0; k < 9; ++k) p[k * V] = r.e[k];
  }
}

__global__ void __launch_bounds__(128) k_update_efield32(Lat L, const float2 *__restrict__ U,
                                                         double *__restrict__ E, double dt) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= L.V) return;
  const int64_t V = L.V;
#pragma unroll 1
  for (int i = 0; i < 3; ++i) {
    m3 sum = m3_zero();
    const int64_t xpi = nb(L, s, i, +1);
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
      if (k == i) continue;
      const double r = L.a0 / L.a[k];
      const double coef = dt * (r * r);
      const int64_t xpk = nb(L, s, k, +1), xmk = nb(L, s, k, -1);
      const int64_t xpimk = nb(L, xmk, i, +1);
      // U staple  U_k(x+i) U_i(x+k)^+ U_k(x)^+ ; D staple  U_k(x+i-k)^+ U_i(x-k)^+ U_k(x-k)
      const m3f su = mulf_nd(mulf_nd(load_link32(U, V, xpi, k), load_link32(U, V, xpk, i)), load_link32(U, V, s, k));
      const m3f sd = mulf_dn(mulf(load_link32(U, V, xmk, i), load_link32(U, V, xpimk, k)), load_link32(U, V, xmk, k));
#pragma unroll
      for (int m = 0; m < 9; ++m) {
        sum.e[m].re += coef * ((double)su.e[m].x + (double)sd.e[m].x);
        sum.e[m].im += coef * ((double)su.e[m].y + (double)sd.e[m].y);
      }
    }
    const m3f ui = load_link32(U, V, s, i);
    m3 u;
#pragma unroll
    for (int k = 0; k < 9; ++k) u.e[k] = {(double)ui.e[k].x, (double)ui.e[k].y};
    const m3 ls = mul(u, sum);
    cplx tr[8];
    traces_with_generators(ls, tr);
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      double *e = E + (int64_t)(i * 8 + a) * V + s;
      *e = *e - 2.0 * tr[a].im;
    }
  }
}

// FP64 projection of every link onto SU(3): rows 0 and 1 orthonormalised
// (Gram-Schmidt), row 2 = conj(row0 x row1).  Reads the FP32 links, writes
// the FP64 links and their FP32 rounding.
__global__ void k_reunitarise(int64_t V, float2 *__restrict__ U32, double2 *__restrict__ U64) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= V) return;
#pragma unroll 1
  for (int d = 0; d < 3; ++d) {
    cplx m[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const float2 v = U32[(int64_t)(d * 9 + k) * V + s];
      m[k] = {(double)v.x, (double)v.y};
    }
    double n0 = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) n0 += norm2(m[c]);
    n0 = 1.0 / sqrt(n0);
#pragma unroll
    for (int c = 0; c < 3; ++c) m[c] = n0 * m[c];
    cplx p = {0.0, 0.0};  // <row0, row1>
#pragma unroll
    for (int c = 0; c < 3; ++c) cmac_cj(p, m[c], m[3 + c]);
#pragma unroll
    for (int c = 0; c < 3; ++c) m[3 + c] = m[3 + c] - p * m[c];
    double n1 = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) n1 += norm2(m[3 + c]);
    n1 = 1.0 / sqrt(n1);
#pragma unroll
    for (int c = 0; c < 3; ++c) m[3 + c] = n1 * m[3 + c];
    // row2 = conj(row0 x row1)
    m[6] = conj(m[1] * m[5] - m[2] * m[4]);
    m[7] = conj(m[2] * m[3] - m[0] * m[5]);
    m[8] = conj(m[0] * m[4] - m[1] * m[3]);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int64_t o = (int64_t)(d * 9 + k) * V + s;
      U64[o] = make_double2(m[k].re, m[k].im);
      U32[o] = make_float2((float)m[k].re, (float)m[k].im);
    }
  }
}

__global__ void k_links_widen(int64_t n, const float2 *__restrict__ U32, double2 *__restrict__ U64) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float2 v = U32[i];
  U64[i] = make_double2((double)v.x, (double)v.y);
}
__global__ void k_links_narrow(int64_t n, const double2 *__restrict__ U64, float2 *__restrict__ U32) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double2 v = U64[i];
  U32[i] = make_float2((float)v.x, (float)v.y);
}

// ------------------------------------------------------------ reductions
// Block-level sum of nq values per thread into partials[block*nq + q].
template <int NQ>
__device__ __forceinline__ void block_sum_store(double v[NQ], double *partials) {
  __shared__ double sh[32][NQ];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
  }
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; ++q) sh[warp][q] = v[q];
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double t = (lane < nw) ? sh[lane][q] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
      if (lane == 0) partials[blockIdx.x * NQ + q] = t;
    }
  }
}

__global__ void __launch_bounds__(256) k_energy(Lat L, const double2 *__restrict__ U,
                                                const double *__restrict__ E, double *partials) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  double v[1] = {0.0};
  if (s < L.V) {
    const int64_t V = L.V;
    double loc = 0.0;
    for (int i = 0; i < 3; ++i) {
      double sq = 0.0;
      for (int a = 0; a < 8; ++a) {
        double ea = E[(int64_t)(i * 8 + a) * V + s] / L.a[i] / L.a0;
        sq += ea * ea;
      }
      loc += sq / 2.0;
      for (int j = i + 1; j < 3; ++j) {
        // Re Tr( U_i(x) U_j(x+i) U_i(x+j)^+ U_j(x)^+ ) = Re sum (M1 .* conj(M2)), M2 = U_j(x) U_i(x+j)
        m3 m1 = mul(load_link(U, V, s, i), load_link(U, V, nb(L, s, i, +1), j));
        m3 m2 = mul(load_link(U, V, s, j), load_link(U, V, nb(L, s, j, +1), i));
        double tr = 0.0;
#pragma unroll
        for (int k = 0; k < 9; ++k) tr += m1.e[k].re * m2.e[k].re + m1.e[k].im * m2.e[k].im;
        loc += 2.0 * 3.0 * ((1.0 - tr / 3.0) / L.a[i] / L.a[j]);
      }
    }
    v[0] = loc;
  }
  block_sum_store<1>(v, partials);
}

// G-like covariant backward divergence pieces for the two Gauss measures.
__global__ void __launch_bounds__(256) k_gauss(Lat L, const double2 *__restrict__ U,
                                               const double *__restrict__ E, double *partials) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  double v[2] = {0.0, 0.0};  // [0] reference sum measure, [1] max-norm
  if (s < L.V) {
    const int64_t V = L.V;
    m3 G = m3_zero();
    double refsum = 0.0;
    for (int i = 0; i < 3; ++i) {
      const int64_t xm = nb(L, s, i, -1);
      double al[8], aln[8];
      for (int a = 0; a < 8; ++a) {
        al[a] = E[(int64_t)(i * 8 + a) * V + s];
        aln[a] = E[(int64_t)(i * 8 + a) * V + xm];
      }
      m3 Em = algebra_matrix(al), En = algebra_matrix(aln);
      m3 un = load_link(U, V, xm, i);
      m3 T = mul(mul_dn(un, En), un);
      m3 Dd = sub(Em, T);
      // reference measure: sum_a 2|Im Tr(T^a D)|, D = (E - U^+ E' U)/a_i^2/a0
      m3 D = scale(Dd, 1.0 / (L.a[i] * L.a[i]) / L.a0);
      cplx tr[8];
      traces_with_generators(D, tr);
      for (int a = 0; a < 8; ++a) refsum += 2.0 * fabs(tr[a].im);
      G = add(G, scale(Dd, 1.0 / L.a[i]));
    }
    G = scale(G, 1.0 / L.a0);
    cplx tr[8];
    traces_with_generators(G, tr);
    double mx = 0.0;
    for (int a = 0; a < 8; ++a) mx = fmax(mx, 2.0 * hypot(tr[a].re, tr[a].im));
    v[0] = refsum;
    v[1] = mx;
  }
  // sum for [0], max for [1]
  __shared__ double sh[32][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v[0] += __shfl_down_sync(0xffffffffu, v[0], o);
    v[1] = fmax(v[1], __shfl_down_sync(0xffffffffu, v[1], o));
  }
  if (lane == 0) {
    sh[warp][0] = v[0];
    sh[warp][1] = v[1];
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    double t0 = (lane < nw) ? sh[lane][0] : 0.0, t1 = (lane < nw) ? sh[lane][1] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      t0 += __shfl_down_sync(0xffffffffu, t0, o);
      t1 = fmax(t1, __shfl_down_sync(0xffffffffu, t1, o));
    }
    if (lane == 0) {
      partials[blockIdx.x * 2] = t0;
      partials[blockIdx.x * 2 + 1] = t1;
    }
  }
}

// Final deterministic reduction: out[q] = op over nblk partials[b*nq+q]
// (op: 0 sum, 1 max selected by mask bit q); the blocks of the grid share
// the values q.
__global__ void k_reduce_final(const double *__restrict__ partials, int64_t nblk, int nq,
                               unsigned maxmask, double *out) {
  __shared__ double sh[256];
  pdl_wait();
  for (int q = blockIdx.x; q < nq; q += gridDim.x) {
    const bool isMax = (maxmask >> q) & 1u;
    double acc = 0.0;
    for (int64_t b = threadIdx.x; b < nblk; b += blockDim.x) {
      double v = __ldcg(partials + b * nq + q);
      acc = isMax ? fmax(acc, v) : acc + v;
    }
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
      if (threadIdx.x < w) sh[threadIdx.x] = isMax ? fmax(sh[threadIdx.x], sh[threadIdx.x + w])
                                                    : sh[threadIdx.x] + sh[threadIdx.x + w];
      __syncthreads();
    }
    if (threadIdx.x == 0) out[q] = sh[0];
    __syncthreads();
  }
}

void launch_reduce_final(const double *partials, int64_t nblk, int nq, unsigned maxmask, double *out,
                         cudaStream_t st) {
  launch_pdl(k_reduce_final, (unsigned)nq, 256, 0, st, partials, nblk, nq, maxmask, out);
}

// ------------------------------------------------------------ initial condition
// p-space construction of TransversePolarisedOccupiedInit (gauge:1349-1381)
// R: 16 complex planes (pol*8 + a) holding x2p of the real normals (unscaled
// FFT); writes A, Ef: 24 complex planes (i*8 + a) in p-space.
// mtab: per direction i and coordinate n (offsets 0, nx, nx + ny) the
// backward-derivative momentum component (re, im) and its modulus, computed
// on the host with the reference's expression (lattice:963-979), so that the
// box edge |p| < Q is decided as on the host also where |p| equals Q up to
// rounding; |p| sums the squared moduli without fused multiply-adds.
__global__ void k_ic_pspace(Lat L, const double2 *__restrict__ R, const double *__restrict__ mtab,
                            double fwd_scale, double Q, double n0, double g, double2 *__restrict__ A,
                            double2 *__restrict__ Ef) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= L.V) return;
  const int64_t V = L.V;
  uint32_t pos[3];
  coords(L, s, pos[0], pos[1], pos[2]);
  const int64_t off[3] = {0, L.nx, L.nx + L.ny};
  cplx p[3];
  double pn2 = 0.0;
  for (int i = 0; i < 3; ++i) {
    const double *m = mtab + 3 * (off[i] + pos[i]);
    p[i] = {m[0], m[1]};
    pn2 = __dadd_rn(pn2, __dmul_rn(m[2], m[2]));
  }
  double pn = sqrt(pn2);
  cplx eps1[3], eps2[3];
  bool zero = !(pn > 1e-12);
  if (!zero) {
    const double tol = 1e-12;
    if (hypot(p[0].re, p[0].im) > tol) {
      double a0 = hypot(p[0].re, p[0].im), a1 = hypot(p[1].re, p[1].im);
      double n12 = sqrt(a0 * a0 + a1 * a1);
      eps1[0] = (-1.0 / n12) * p[1];
      eps1[1] = (1.0 / n12) * p[0];
      eps1[2] = {0.0, 0.0};
      double den = pn * n12;
      eps2[0] = (1.0 / den) * (conj(p[0]) * p[2]);
      eps2[1] = (1.0 / den) * (conj(p[1]) * p[2]);
      eps2[2] = {-n12 / pn, 0.0};
    } else {
      double a1 = hypot(p[1].re, p[1].im), a2 = hypot(p[2].re, p[2].im);
      double n23 = sqrt(a1 * a1 + a2 * a2);
      eps1[0] = {0.0, 0.0};
      eps1[1] = (1.0 / n23) * p[2];
      eps1[2] = (-1.0 / n23) * p[1];
      eps2[0] = {1.0, 0.0};
      eps2[1] = {0.0, 0.0};
      eps2[2] = {0.0, 0.0};
    }
  }
  double occ = (pn < Q) ? n0 : g * g / 2.0;
  double pa = zero ? 0.0 : sqrt(occ / pn * 2.0);
  double pe = zero ? 0.0 : sqrt(occ * pn * 2.0);
  for (int a = 0; a < 8; ++a) {
    cplx r1 = fwd_scale * ldg(R + (int64_t)a * V + s);
    cplx r2 = fwd_scale * ldg(R + (int64_t)(8 + a) * V + s);
    for (int i = 0; i < 3; ++i) {
      cplx m = zero ? cplx{0.0, 0.0} : r1 * eps1[i] + r2 * eps2[i];
      st(A + (int64_t)(i * 8 + a) * V + s, pa * m);
      st(Ef + (int64_t)(i * 8 + a) * V + s, times_i(pe * m));
    }
  }
}

// links = exp(i Re(A) a_i) (or 1), E = Re(Ef) a0 a_i after the backward FFT
// (scale 1/Volume folded in here), gauge:1431-1443.
__global__ void k_ic_write(Lat L, const double2 *__restrict__ A, const double2 *__restrict__ Ef,
                           double inv_volume, int identity_links, double2 *__restrict__ U,
                           double *__restrict__ E) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= L.V) return;
  const int64_t V = L.V;
  for (int i = 0; i < 3; ++i) {
    double as[8];
    for (int a = 0; a < 8; ++a) {
      as[a] = __ldg(&A[(int64_t)(i * 8 + a) * V + s].x) * inv_volume * L.a[i];
      E[(int64_t)(i * 8 + a) * V + s] = __ldg(&Ef[(int64_t)(i * 8 + a) * V + s].x) * inv_volume * L.a0 * L.a[i];
    }
    m3 G = identity_links ? m3_id() : expi_herm(algebra_matrix(as));
    store_link(U, V, s, i, G);
  }
}

// max over sites and directions of max_ij |(U U^+ - 1)_ij| and of |det U - 1|
// (partials[block*2 + q], both maxima)
__global__ void __launch_bounds__(256) k_unitarity(Lat L, const double2 *__restrict__ U, double *partials) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  double v[2] = {0.0, 0.0};
  if (s < L.V) {
    for (int d = 0; d < 3; ++d) {
      const m3 u = load_link(U, L.V, s, d);
      const m3 p = mul_nd(u, u);
      for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
          const cplx e = p.e[i * 3 + j] - cplx{i == j ? 1.0 : 0.0, 0.0};
          v[0] = fmax(v[0], hypot(e.re, e.im));
        }
      const cplx det = u.e[0] * (u.e[4] * u.e[8] - u.e[5] * u.e[7]) - u.e[1] * (u.e[3] * u.e[8] - u.e[5] * u.e[6]) +
                       u.e[2] * (u.e[3] * u.e[7] - u.e[4] * u.e[6]);
      v[1] = fmax(v[1], hypot(det.re - 1.0, det.im));
    }
  }
  __shared__ double sh[32][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v[0] = fmax(v[0], __shfl_down_sync(0xffffffffu, v[0], o));
    v[1] = fmax(v[1], __shfl_down_sync(0xffffffffu, v[1], o));
  }
  if (lane == 0) {
    sh[warp][0] = v[0];
    sh[warp][1] = v[1];
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    double t0 = (lane < nw) ? sh[lane][0] : 0.0, t1 = (lane < nw) ? sh[lane][1] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      t0 = fmax(t0, __shfl_down_sync(0xffffffffu, t0, o));
      t1 = fmax(t1, __shfl_down_sync(0xffffffffu, t1, o));
    }
    if (lane == 0) {
      partials[blockIdx.x * 2] = t0;
      partials[blockIdx.x * 2 + 1] = t1;
    }
  }
}

}  // namespace nrq
