// Gluon-distribution observables on the device (src/gaugeconfiguration_su3.f90,
// abbreviated "gauge"; src/lattice.f90 "lattice"):
//   - Coulomb gauge fixing of the links, CoulombGaugefixing_Links
//     (gauge:2297-2456): the divergence D(x) = sum_i AH(U_i(x-i) - U_i(x))
//     (gauge:2460-2478), Fourier acceleration by (pmax/|p|)^2, the gauge
//     transformation G = ExpAH(alpha D) and U_i(x) <- G(x) U_i(x) G(x+i)^+;
//     the electric field is not transformed, as in the reference
//   - the transverse AA and EE correlators (gauge:1825-1972): algebra
//     coordinates of ArgLogU(U_i)/a_i and of E/(a_i a0), their x2p transforms
//     and f_i P_ij conj(f_j) / Volume with the real part of the transverse
//     projector (lattice:1184-1198) at the backward-derivative momentum
//     (lattice:963-979), averaged over the eight generators.
// The FFTs are cuFFT Z2Z transforms over all components at once; the x2p
// (a1 a2 a3) and p2x (1/Volume) scales of the reference are applied in the
// kernels around them.
#include "nrq_eigen.cuh"
#include "nrq_kernels.cuh"
#include "pdl.cuh"

namespace nrq {

namespace {
// backward-derivative lattice momentum (lattice:963-979) of site s; returns |p|
__device__ __forceinline__ double lattice_momentum(const Lat &L, int64_t s, cplx p[3]) {
  uint32_t pos[3];
  coords(L, s, pos[0], pos[1], pos[2]);
  const int64_t ext[3] = {L.nx, L.ny, L.nz};
  double n2 = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double sn, cs;
    sincospi((double)pos[i] / (double)ext[i], &sn, &cs);
    const double m = 2.0 * sn / L.a[i];
    p[i] = {m * cs, -m * sn};
    n2 += m * m;
  }
  return sqrt(n2);
}
}  // namespace

// exp(i H) of a hermitian H: exp(i tr(H)/3) exp(i (H - tr(H)/3))
__device__ __forceinline__ m3 exp_herm(m3 h) {
  const double tr = (h.e[0].re + h.e[4].re + h.e[8].re) / 3.0;
  h.e[0].re -= tr;
  h.e[4].re -= tr;
  h.e[8].re -= tr;
  m3 g = expi_herm(h);
  double sn, cs;
  sincos(tr, &sn, &cs);
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const cplx v = g.e[k];
    g.e[k] = {cs * v.re - sn * v.im, cs * v.im + sn * v.re};
  }
  return g;
}

// D(x) = sum_i AH(U_i(x-i) - U_i(x)), AH(M) = (M - M^+)/2, as 9 complex
// planes (r*3 + c); partials[block] = max over the block of |D(x)|_F / 9
__global__ void __launch_bounds__(128) k_cg_divergence(Lat L, const double2 *__restrict__ U,
                                                       double2 *__restrict__ D, double *__restrict__ partials) {
  const int64_t V = L.V;
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  double f = 0.0;
  if (s < V) {
    m3 d = m3_zero();
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const m3 u = load_link(U, V, s, i), um = load_link(U, V, nb(L, s, i, -1), i);
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const cplx a = um.e[r * 3 + c] - u.e[r * 3 + c];
          const cplx b = um.e[c * 3 + r] - u.e[c * 3 + r];
          d.e[r * 3 + c].re += 0.5 * (a.re - b.re);
          d.e[r * 3 + c].im += 0.5 * (a.im + b.im);
        }
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      D[(int64_t)k * V + s] = make_double2(d.e[k].re, d.e[k].im);
      f += norm2(d.e[k]);
    }
    f = sqrt(f) / 9.0;
  }
  __shared__ double sh[4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) f = fmax(f, __shfl_down_sync(0xffffffffu, f, o));
  if (lane == 0) sh[warp] = f;
  __syncthreads();
  if (threadIdx.x == 0) partials[blockIdx.x] = fmax(fmax(sh[0], sh[1]), fmax(sh[2], sh[3]));
}

// p-space step of the Fourier acceleration: D(p) *= scale (pmax/|p|)^2 for
// |p| above the reference's zero tolerance, D(p) *= scale otherwise (scale
// carries alpha and the x2p/p2x normalisation)
__global__ void k_cg_accelerate(Lat L, double2 *__restrict__ D, double pmax, double scale) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= L.V) return;
  cplx p[3];
  const double pn = lattice_momentum(L, s, p);
  const double f = pn > 1e-12 ? scale * (pmax / pn) * (pmax / pn) : scale;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    double2 v = D[(int64_t)k * L.V + s];
    v.x *= f;
    v.y *= f;
    D[(int64_t)k * L.V + s] = v;
  }
}

// G = ExpAH(A) = exp(i H), H = -i A (hermitian; A anti-hermitian, not
// traceless), in place: exp(i H) = exp(i tr(H)/3) exp(i (H - tr(H)/3))
__global__ void __launch_bounds__(128) k_cg_expah(int64_t V, double2 *__restrict__ D) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= V) return;
  m3 a;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = D[(int64_t)k * V + s];
    a.e[k] = {v.x, v.y};
  }
  // H = -i A, made exactly hermitian
  m3 h;
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      // (H + H^+)/2 with H = -i A: -i x = (x.im, -x.re), conj(-i y) = (y.im, y.re)
      const cplx x = a.e[r * 3 + c], y = a.e[c * 3 + r];
      h.e[r * 3 + c] = {0.5 * (x.im + y.im), 0.5 * (y.re - x.re)};
    }
  store_link(D, V, s, 0, exp_herm(h));
}

// U_i(x) <- G(x) U_i(x) G(x+i)^+ (in place: a thread reads and writes only
// its own site's links)
__global__ void __launch_bounds__(128) k_cg_transform(Lat L, double2 *__restrict__ U, const double2 *__restrict__ G) {
  const int64_t V = L.V;
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= V) return;
  m3 g;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = G[(int64_t)k * V + s];
    g.e[k] = {v.x, v.y};
  }
#pragma unroll 1
  for (int i = 0; i < 3; ++i) {
    const int64_t xp = nb(L, s, i, +1);
    m3 gp;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const double2 v = G[(int64_t)k * V + xp];
      gp.e[k] = {v.x, v.y};
    }
    store_link(U, V, s, i, mul_nd(mul(g, load_link(U, V, s, i)), gp));
  }
}

// F plane (field*24 + i*8 + a): field 0 the gauge field 2 Re Tr(T^a ArgLogU(U_i))/a_i
// (gauge:1992-2000, su3:318-334), field 1 the electric field E^a_i/(a_i a0)
// (gauge:2032-2049); complex with zero imaginary part, for the FFT
__global__ void __launch_bounds__(128) k_gluon_fields(Lat L, const double2 *__restrict__ U,
                                                      const double *__restrict__ E, double2 *__restrict__ F) {
  const int64_t V = L.V;
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= V) return;
  const int i = blockIdx.y;
  {
    const m3 u = load_link(U, V, s, i);
    m3 h;
    if (!log_unitary(u, h, false)) {
      cplx ev[3];
      m3 S;
      eigenc3(u, ev, S);
      double th[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) th[k] = atan2(ev[k].im, ev[k].re);
      // ArgLogU = S^+ diag(theta) S
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          cplx acc = {0.0, 0.0};
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const cplx a = conj(S.e[k * 3 + r]), b = S.e[k * 3 + c];
            acc = acc + th[k] * (a * b);
          }
          h.e[r * 3 + c] = acc;
        }
    }
    cplx tr[8];
    traces_with_generators(h, tr);
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      F[(int64_t)(i * 8 + a) * V + s] = make_double2(2.0 * tr[a].re / L.a[i], 0.0);
      F[(int64_t)(24 + i * 8 + a) * V + s] = make_double2(E[(int64_t)(i * 8 + a) * V + s] / L.a[i] / L.a0, 0.0);
    }
  }
}

// per momentum site and field (blockIdx.y): out[0][s] = AA, out[1][s] = EE, out[2][s] = |p|
// (F holds the unscaled forward transforms; fwd = a1 a2 a3)
__global__ void __launch_bounds__(64) k_transverse_corr(Lat L, const double2 *__restrict__ F, double fwd,
                                                         double volume, double *__restrict__ out) {
  const int64_t V = L.V;
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= V) return;
  cplx p[3];
  const double pn = lattice_momentum(L, s, p);
  // the reference's projector is real: Re[(delta_ij - conj(p_i) p_j / |p|^2) / 2]
  double P[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double re = p[i].re * p[j].re + p[i].im * p[j].im;  // Re(conj(p_i) p_j)
      P[i][j] = pn < 1e-12 ? 0.0 : ((i == j ? 1.0 : 0.0) - re / (pn * pn)) / 2.0;
    }
  const int field = blockIdx.y;
  double acc = 0.0;
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    cplx f[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double2 v = F[(int64_t)(field * 24 + i * 8 + a) * V + s];
      f[i] = {v.x * fwd, v.y * fwd};
    }
    double res = 0.0;  // Re sum_ij f_i P_ij conj(f_j)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) res += P[i][j] * (f[i].re * f[j].re + f[i].im * f[j].im);
    acc += (res / volume) / 8.0;
  }
  out[(int64_t)field * V + s] = acc;
  if (field == 0) out[2 * V + s] = pn;
}

// ------------------------------------------------------------ short extents
// Gauge fixing on lattices whose extents are at most kCgMaxExtent: three
// launches an iteration and no host synchronisation within a batch of them.
//
// D is anti-hermitian and the filter (pmax/|p|)^2 real and even, so its nine
// real numbers a site (the imaginary diagonal, three complex entries) go
// through five complex transforms, two reals in one, in place of nine.  A
// transform along one direction is the direct sum over N terms: with N <= 32
// its arithmetic is small beside the latency of a library transform's three
// launches (the outputs k and N - k come from the same four sums, and for even
// N the terms j and j + N/2 are added first), and each of the three
// directions joins the kernel that has its data:
//   k_cg_rows   (x rows)    U' = G U G^+ of the iteration before, D, its
//                           maximum, transform along x
//   k_cg_planes (yz planes) transforms along y and z, filter, back along z, y
//   k_cg_exp    (x rows)    back along x, G = ExpAH
// A thread of k_cg_rows makes U'_i(x) and again U'_i(x-i), so links go from
// one buffer to another.  Whether the deviation has met the tolerance is
// decided on the device: each launch looks at the last deviation at entry and
// returns where that met it, which leaves the following slots zero.
// Bound: latency, at a few thousand threads a launch.  An iteration at 16^3
// takes 21 us (library transforms of nine planes, five kernels of its own and
// a synchronisation: 69), at 32^3 45 us (75); above 32 the direct sums would
// lose to the library.
namespace {
// outputs k, n - k (p, q) and k + 2, n - k - 2 of a transform of z_j =
// in[j*stride]: p_k = sum_j z_j w^(jk), q_k = sum_j z_j w^(-jk), tw[m] = w^m
struct Dft {
  double2 p[2], q[2];
};
__device__ __forceinline__ Dft dft(const double2 *in, int stride, int n, int k, const double2 *tw) {
  const bool even = (n & 1) == 0;
  const int h = even ? n >> 1 : n, off = h * stride;
  const double sgn = (k & 1) ? -1.0 : 1.0;
  const int k1 = k + 2 < n ? k + 2 : 0;
  double a[2] = {0.0, 0.0}, b[2] = {0.0, 0.0}, c[2] = {0.0, 0.0}, d[2] = {0.0, 0.0};
  int m0 = 0, m1 = 0;
#pragma unroll 4
  for (int j = 0; j < h; ++j) {
    double2 z = in[j * stride];
    if (even) {
      const double2 y = in[j * stride + off];
      z.x = fma(sgn, y.x, z.x);
      z.y = fma(sgn, y.y, z.y);
    }
    const double2 w0 = tw[m0], w1 = tw[m1];
    a[0] = fma(z.x, w0.x, a[0]);
    b[0] = fma(z.y, w0.y, b[0]);
    c[0] = fma(z.x, w0.y, c[0]);
    d[0] = fma(z.y, w0.x, d[0]);
    a[1] = fma(z.x, w1.x, a[1]);
    b[1] = fma(z.y, w1.y, b[1]);
    c[1] = fma(z.x, w1.y, c[1]);
    d[1] = fma(z.y, w1.x, d[1]);
    m0 += k;
    if (m0 >= n) m0 -= n;
    m1 += k1;
    if (m1 >= n) m1 -= n;
  }
  Dft r;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    r.p[e] = make_double2(a[e] - b[e], c[e] + d[e]);
    r.q[e] = make_double2(a[e] + b[e], d[e] - c[e]);
  }
  return r;
}
// The work items of a transform are groups of outputs {k, k + 2} and their
// mirror images: k = 0, 1, 4, 5, 8, ...
__host__ __device__ __forceinline__ int dft_groups(int n) {
  const int h = n >> 1;  // the largest k
  return 2 * (h >> 2) + ((h & 3) ? 2 : 1);
}
__device__ __forceinline__ int dft_k(int g) { return 4 * (g >> 1) + (g & 1); }
// stores a group's outputs: put(k, value); inverse: the conjugate transform
template <bool INV, typename Put>
__device__ __forceinline__ void dft_put(const Dft &r, int n, int k, Put put) {
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int kk = k + 2 * e;
    if (2 * kk > n) break;
    put(kk, INV ? r.q[e] : r.p[e]);
    if (kk > 0 && 2 * kk != n) put(n - kk, INV ? r.p[e] : r.q[e]);
  }
}
__device__ __forceinline__ void load_table(double2 *tw, const double2 *__restrict__ tab, int n) {
  for (int m = threadIdx.x; m < n; m += blockDim.x) tw[m] = __ldg(tab + m);
}
// slot < 0: no deviation yet
__device__ __forceinline__ bool cg_done(const double *dev, int slot, double tol) {
  return slot >= 0 && !(*(const volatile double *)(dev + slot) > tol);
}
constexpr int kCgRow = kCgRowSites + 5;  // a component's sites in shared memory, rows padded to odd lengths
}  // namespace

// tw[d*kCgMaxExtent + m] = exp(-2 pi i m / N_d), p2[d*kCgMaxExtent + m] = (2 sin(pi m / N_d) / a_d)^2
__global__ void k_cg_tables(Lat L, double2 *__restrict__ tw, double *__restrict__ p2) {
  const int d = blockIdx.x, n = (int)(d == 0 ? L.nx : d == 1 ? L.ny : L.nz);
  for (int m = threadIdx.x; m < n; m += blockDim.x) {
    double sn, cs;
    sincospi(-2.0 * (double)m / (double)n, &sn, &cs);
    tw[d * kCgMaxExtent + m] = make_double2(cs, sn);
    const double h = 2.0 * sinpi((double)m / (double)n) / L.a[d];
    p2[d * kCgMaxExtent + m] = h * h;
  }
}

// S = rows * nx sites a block, thread = (direction, site).  G null: no
// transformation (the first iteration).  F null: the transformation alone.
// dev[slot]: this iteration's deviation, zero before.
__global__ void __launch_bounds__(3 * kCgRowSites)
    k_cg_rows(Lat L, int rows, const double2 *__restrict__ Uin, const double2 *__restrict__ G,
              double2 *__restrict__ Uout, const double2 *__restrict__ tw, double2 *__restrict__ F, double *dev,
              double tol, int slot) {
  pdl_wait();
  pdl_trigger();
  if (cg_done(dev, slot - 1, tol)) return;
  __shared__ double sd[3][9][kCgRowSites];
  __shared__ double2 z[5][kCgRow], w[kCgMaxExtent];
  const int V = (int)L.V, nx = (int)L.nx, nrows = (int)(L.ny * L.nz), S = rows * nx, ld = nx | 1;
  const int i = threadIdx.x / S, l = threadIdx.x - i * S;
  const int x0 = blockIdx.x * S + l;
  if (i < 3) {
    const int x = x0 < V ? x0 : V - 1;
    const int xm = (int)nb(L, x, i, -1);
    m3 u = load_link_c(Uin, V, x, i), um = load_link_c(Uin, V, xm, i);
    if (G) {
      const m3 g = load_link_c(G, V, x, 0);
      u = mul_nd(mul(g, u), load_link_c(G, V, (int)nb(L, x, i, +1), 0));
      if (x0 < V) store_link(Uout, V, x, i, u);
      um = mul_nd(mul(load_link_c(G, V, xm, 0), um), g);
    }
    // AH(um - u): diagonal (imaginary), entries 01, 02, 12
#pragma unroll
    for (int r = 0; r < 3; ++r) sd[i][r][l] = um.e[4 * r].im - u.e[4 * r].im;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const int r = e == 2 ? 1 : 0, c = e == 0 ? 1 : 2;
      const cplx a = um.e[r * 3 + c] - u.e[r * 3 + c], b = um.e[c * 3 + r] - u.e[c * 3 + r];
      sd[i][3 + 2 * e][l] = 0.5 * (a.re - b.re);
      sd[i][4 + 2 * e][l] = 0.5 * (a.im + b.im);
    }
  }
  if (!F) return;
  load_table(w, tw, nx);
  __syncthreads();
  double f = 0.0;
  if (i == 0) {
    double d[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) d[q] = sd[0][q][l] + sd[1][q][l] + sd[2][q][l];
    const int r = l / nx, o = r * ld + l - r * nx;
    z[0][o] = make_double2(d[0], d[1]);
    z[1][o] = make_double2(d[2], 0.0);
#pragma unroll
    for (int e = 0; e < 3; ++e) z[2 + e][o] = make_double2(d[3 + 2 * e], d[4 + 2 * e]);
    double diag = 0.0, off = 0.0;
#pragma unroll
    for (int q = 0; q < 3; ++q) diag = fma(d[q], d[q], diag);
#pragma unroll
    for (int q = 3; q < 9; ++q) off = fma(d[q], d[q], off);
    f = sqrt(fma(2.0, off, diag)) / 9.0;
  }
  // the maximum of the non-negative numbers is that of their bits
  if (threadIdx.x < ((S + 31) & ~31)) {
    f = fmax(f, 0.0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) f = fmax(f, __shfl_down_sync(0xffffffffu, f, o));
    if ((threadIdx.x & 31) == 0) atomicMax((unsigned long long *)(dev + slot), (unsigned long long)__double_as_longlong(f));
  }
  __syncthreads();
  // along x, into F[(c*nx + k)*nrows + row]
  const int lines = 5 * rows, items = lines * dft_groups(nx);
  for (int o = threadIdx.x; o < items; o += blockDim.x) {
    const int g = o / lines, cr = o - g * lines, c = cr / rows, r = cr - c * rows, row = blockIdx.x * rows + r;
    if (row >= nrows) continue;
    const int k = dft_k(g);
    const Dft t = dft(&z[c][r * ld], 1, nx, k, w);
    dft_put<false>(t, nx, k, [&](int kk, double2 v) { F[((int64_t)c * nx + kk) * nrows + row] = v; });
  }
}

// one block per (component, k_x): the yz plane in shared memory, y rows
// padded to an odd length
__global__ void __launch_bounds__(320)
    k_cg_planes(Lat L, const double2 *__restrict__ tw, const double *__restrict__ p2, double2 *__restrict__ F,
                double pmax, double scale, const double *dev, double tol, int slot) {
  pdl_wait();
  pdl_trigger();
  if (cg_done(dev, slot, tol)) return;
  extern __shared__ double2 sm[];
  const int ny = (int)L.ny, nz = (int)L.nz, n = ny * nz, ld = ny | 1, kx = blockIdx.x % (int)L.nx;
  double2 *A = sm, *B = sm + ld * nz, *wy = sm + 2 * ld * nz, *wz = wy + ny;
  double2 *plane = F + (int64_t)blockIdx.x * n;
  load_table(wy, tw + kCgMaxExtent, ny);
  load_table(wz, tw + 2 * kCgMaxExtent, nz);
  for (int o = threadIdx.x; o < n; o += blockDim.x) A[(o / ny) * ld + o % ny] = __ldca(plane + o);
  const int iy = dft_groups(ny) * nz, iz = dft_groups(nz) * ny;
  const double px2 = __ldg(p2 + kx), top = scale * pmax * pmax;
  __syncthreads();
  for (int o = threadIdx.x; o < iy; o += blockDim.x) {
    const int z = o % nz, k = dft_k(o / nz);
    const Dft t = dft(A + z * ld, 1, ny, k, wy);
    dft_put<false>(t, ny, k, [&](int kk, double2 v) { B[z * ld + kk] = v; });
  }
  __syncthreads();
  for (int o = threadIdx.x; o < iz; o += blockDim.x) {
    const int y = o % ny, k = dft_k(o / ny);
    const Dft t = dft(B + y, ld, nz, k, wz);
    const double pxy = px2 + __ldg(p2 + kCgMaxExtent + y);
    dft_put<false>(t, nz, k, [&](int kk, double2 v) {
      const double q = pxy + __ldg(p2 + 2 * kCgMaxExtent + kk), f = q > 1e-24 ? top / q : scale;
      A[kk * ld + y] = make_double2(f * v.x, f * v.y);
    });
  }
  __syncthreads();
  for (int o = threadIdx.x; o < iz; o += blockDim.x) {
    const int y = o % ny, k = dft_k(o / ny);
    const Dft t = dft(A + y, ld, nz, k, wz);
    dft_put<true>(t, nz, k, [&](int kk, double2 v) { B[kk * ld + y] = v; });
  }
  __syncthreads();
  for (int o = threadIdx.x; o < iy; o += blockDim.x) {
    const int z = o % nz, k = dft_k(o / nz);
    const Dft t = dft(B + z * ld, 1, ny, k, wy);
    dft_put<true>(t, ny, k, [&](int kk, double2 v) { plane[z * ny + kk] = v; });
  }
}

// rows * nx sites a block, 3 threads a site for the transform, one for the exponential
__global__ void __launch_bounds__(3 * kCgRowSites)
    k_cg_exp(Lat L, int rows, const double2 *__restrict__ tw, const double2 *__restrict__ F, double2 *__restrict__ G,
             const double *dev, double tol, int slot) {
  pdl_wait();
  pdl_trigger();
  if (cg_done(dev, slot, tol)) return;
  __shared__ double2 f[5][kCgRow], z[5][kCgRowSites], w[kCgMaxExtent];
  const int nx = (int)L.nx, nrows = (int)(L.ny * L.nz), S = rows * nx, ld = nx | 1;
  load_table(w, tw, nx);
  for (int o = threadIdx.x; o < 5 * S; o += blockDim.x) {  // f[c][r*ld + k]
    const int r = o % rows, ck = o / rows, k = ck % nx, c = ck / nx, row = blockIdx.x * rows + r;
    f[c][r * ld + k] = row < nrows ? __ldca(F + ((int64_t)c * nx + k) * nrows + row) : make_double2(0.0, 0.0);
  }
  __syncthreads();
  const int lines = 5 * rows, items = lines * dft_groups(nx);
  for (int o = threadIdx.x; o < items; o += blockDim.x) {
    const int g = o / lines, cr = o - g * lines, c = cr / rows, r = cr - c * rows, k = dft_k(g);
    const Dft t = dft(&f[c][r * ld], 1, nx, k, w);
    dft_put<true>(t, nx, k, [&](int kk, double2 v) { z[c][r * nx + kk] = v; });
  }
  __syncthreads();
  const int l = threadIdx.x;
  const int64_t x = (int64_t)blockIdx.x * S + l;
  if (l >= S || x >= L.V) return;
  // H = -i A, hermitian: diagonal Im A, off-diagonal (Im A, -Re A)
  m3 h;
  h.e[0] = {z[0][l].x, 0.0};
  h.e[4] = {z[0][l].y, 0.0};
  h.e[8] = {z[1][l].x, 0.0};
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const int r = e == 2 ? 1 : 0, c = e == 0 ? 1 : 2;
    h.e[r * 3 + c] = {z[2 + e][l].y, -z[2 + e][l].x};
    h.e[c * 3 + r] = {z[2 + e][l].y, z[2 + e][l].x};
  }
  store_link(G, L.V, x, 0, exp_herm(h));
}

bool cg_short_applicable(const Lat &L) {
  return L.nx <= kCgMaxExtent && L.ny <= kCgMaxExtent && L.nz <= kCgMaxExtent;
}
namespace {
int cg_rows(const Lat &L) {  // x rows of a block
  const int r = (kCgRowSites / 2) / (int)L.nx;
  return r < 1 ? 1 : r > 4 ? 4 : r;
}
unsigned cg_threads(const Lat &L, int rows) { return (unsigned)((3 * rows * (int)L.nx + 31) / 32 * 32); }
unsigned cg_row_blocks(const Lat &L, int rows) { return (unsigned)((L.ny * L.nz + rows - 1) / rows); }
}  // namespace
void launch_cg_tables(Lat L, double2 *tw, double *p2, cudaStream_t st) {
  k_cg_tables<<<3, kCgMaxExtent, 0, st>>>(L, tw, p2);
}
void launch_cg_rows(Lat L, const double2 *Uin, const double2 *G, double2 *Uout, const double2 *tw, double2 *F,
                    double *dev, double tol, int slot, cudaStream_t st) {
  const int rows = cg_rows(L);
  launch_pdl(k_cg_rows, cg_row_blocks(L, rows), cg_threads(L, rows), 0, st, L, rows, Uin, G, Uout, tw, F, dev, tol, slot);
}
void launch_cg_smooth(Lat L, const double2 *tw, const double *p2, double2 *F, double2 *G, double pmax, double scale,
                      const double *dev, double tol, int slot, cudaStream_t st) {
  const int rows = cg_rows(L), ny = (int)L.ny, nz = (int)L.nz;
  const size_t bytes = sizeof(double2) * (2 * (ny | 1) * nz + ny + nz);
  const int items = dft_groups(ny) * nz > dft_groups(nz) * ny ? dft_groups(ny) * nz : dft_groups(nz) * ny;
  const unsigned threads = items > 320 ? 320u : (unsigned)((items + 31) / 32 * 32);
  launch_pdl(k_cg_planes, (unsigned)(5 * L.nx), threads, bytes, st, L, tw, p2, F, pmax, scale, dev, tol, slot);
  launch_pdl(k_cg_exp, cg_row_blocks(L, rows), cg_threads(L, rows), 0, st, L, rows, tw, F, G, dev, tol, slot);
}

}  // namespace nrq
