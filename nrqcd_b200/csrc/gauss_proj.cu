// Gauss-law projection of the thermal initial condition (EquilibriumInit,
// src/gaugeconfiguration_su3.f90:455-500, abbreviated "gauge"): Jacobi
// sweeps
//   E_k(x) <- coords( kdt (U_k(x) G(x) U_k(x)^+ G(x+k) - G(x)) + E_k(x) ),
//   kdt = 0.01 a0,
// with G(x) = sum_i (E_i(x) - U_i(x-i)^+ E_i(x-i) U_i(x-i)) / a_i / a0
// (GetG, gauge:786-812) taken from the field before the sweep, until the
// max-norm deviation max_{x,a} 2|Tr(T^a G(x))| (GetGdeviation,
// gauge:724-768) is at most the tolerance.
//
// Lattices that fit the GPU at one thread per link run many sweeps a launch
// (k_gauss_run, below).  On the others one sweep is two launches (V < 2^31
// sites): k_gauss_g writes G of every site (9 complex
// planes) and the deviation (the last block to finish reduces the per-block
// maxima and decides convergence), then k_gauss_sweep updates E in place
// (each thread reads and writes only its own site's E).  Convergence is
// decided on the device: once the deviation is at most the tolerance both
// kernels return at entry, so the host can queue many sweeps between reads
// and the sweep count is the reference's exactly.
#include "../../include/nrqcd_b200.h"
#include "nrq_kernels.cuh"

namespace nrq {

namespace {
// site coordinates with 32-bit arithmetic (V < 2^31, checked by the host),
// computed once per thread; neighbours by periodic offsets
struct Pos32 {
  uint32_t s, x, y, z, nx, nxy;
};
__device__ __forceinline__ Pos32 pos32(const Lat &L, uint32_t s) {
  Pos32 p;
  p.s = s;
  p.nx = (uint32_t)L.nx;
  p.nxy = p.nx * (uint32_t)L.ny;
  const uint32_t t = s / p.nx;
  p.x = s - t * p.nx;
  p.z = t / (uint32_t)L.ny;
  p.y = t - p.z * (uint32_t)L.ny;
  return p;
}
__device__ __forceinline__ uint32_t fwd32(const Lat &L, const Pos32 &p, int d) {
  if (d == 0) return p.x + 1 == p.nx ? p.s + 1 - p.nx : p.s + 1;
  if (d == 1) return p.y + 1 == (uint32_t)L.ny ? p.s + p.nx - p.nxy : p.s + p.nx;
  return p.z + 1 == (uint32_t)L.nz ? p.s + p.nxy - (uint32_t)L.V : p.s + p.nxy;
}
__device__ __forceinline__ uint32_t bwd32(const Lat &L, const Pos32 &p, int d) {
  if (d == 0) return p.x == 0 ? p.s + p.nx - 1 : p.s - 1;
  if (d == 1) return p.y == 0 ? p.s + p.nxy - p.nx : p.s - p.nx;
  return p.z == 0 ? p.s + (uint32_t)L.V - p.nxy : p.s - p.nxy;
}
}  // namespace

__global__ void __launch_bounds__(128, 3) k_gauss_g(Lat L, const double2 *__restrict__ U,
                                                 const double *__restrict__ E, double2 *__restrict__ G,
                                                 double *__restrict__ partials, GaussProjState *st, double tol,
                                                 int count) {
  if (*(volatile int *)&st->done) return;
  const int64_t V = L.V;
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  double mx = 0.0;
  if (s < V) {
    const Pos32 p = pos32(L, (uint32_t)s);
    m3 g = m3_zero();
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int64_t xm = bwd32(L, p, i);
      double al[8], aln[8];
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        al[a] = E[(int64_t)(i * 8 + a) * V + s];
        aln[a] = E[(int64_t)(i * 8 + a) * V + xm];
      }
      const m3 un = load_link(U, V, xm, i);
      const m3 t = mul(mul_dn(un, algebra_matrix(aln)), un);
      const m3 d = sub(algebra_matrix(al), t);
      const double c = 1.0 / (L.a[i] * L.a0);  // one division per direction, not per entry
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        g.e[k].re = fma(d.e[k].re, c, g.e[k].re);
        g.e[k].im = fma(d.e[k].im, c, g.e[k].im);
      }
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) G[(int64_t)k * V + s] = make_double2(g.e[k].re, g.e[k].im);
    cplx tr[8];
    traces_with_generators(g, tr);
    // max |Tr(T^a G)|^2 here; the deviation 2|Tr| is taken once, by the last block
#pragma unroll
    for (int a = 0; a < 8; ++a) mx = fmax(mx, tr[a].re * tr[a].re + tr[a].im * tr[a].im);
  }
  // block maximum
  __shared__ double sh[4];  // one per warp of the 128-thread block
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
  if (lane == 0) sh[warp] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, sh[w]);
    partials[blockIdx.x] = m;
    __threadfence();
    last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  // last block: maximum over all blocks (order-independent, exact)
  __threadfence();
  double m = 0.0;
  for (int64_t b = threadIdx.x; b < gridDim.x; b += blockDim.x) m = fmax(m, ((volatile double *)partials)[b]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  if (lane == 0) sh[warp] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m2 = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m2 = fmax(m2, sh[w]);
    const double dev = 2.0 * sqrt(m2);
    st->dev = dev;
    if (count) st->sweeps += 1;
    if (!(dev > tol)) st->done = 1;
    st->ticket = 0u;
    __threadfence();
  }
}

__global__ void __launch_bounds__(128) k_gauss_sweep(Lat L, const double2 *__restrict__ U,
                                                     const double2 *__restrict__ G, double *__restrict__ E,
                                                     const GaussProjState *st, double kdt) {
  if (*(const volatile int *)&st->done) return;
  const int64_t V = L.V;
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= V) return;
  const Pos32 p = pos32(L, (uint32_t)s);
  m3 g;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = G[(int64_t)k * V + s];
    g.e[k] = {v.x, v.y};
  }
#pragma unroll 1
  for (int k = 0; k < 3; ++k) {
    const int64_t xp = fwd32(L, p, k);
    m3 gn;
#pragma unroll
    for (int m = 0; m < 9; ++m) {
      const double2 v = G[(int64_t)m * V + xp];
      gn.e[m] = {v.x, v.y};
    }
    double al[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) al[a] = E[(int64_t)(k * 8 + a) * V + s];
    const m3 u = load_link(U, V, s, k);
    const m3 t = mul(mul_nd(mul(u, g), u), gn);  // U G U^+ G(x+k)
    const m3 e = algebra_matrix(al);
    m3 term;
#pragma unroll
    for (int m = 0; m < 9; ++m) {
      term.e[m].re = kdt * (t.e[m].re - g.e[m].re) + e.e[m].re;
      term.e[m].im = kdt * (t.e[m].im - g.e[m].im) + e.e[m].im;
    }
    cplx tr[8];
    traces_with_generators(term, tr);
#pragma unroll
    for (int a = 0; a < 8; ++a) E[(int64_t)(k * 8 + a) * V + s] = 2.0 * tr[a].re;
  }
}

// One launch of many sweeps where the lattice fits the GPU at one thread per
// site and direction (kRunSites sites an SM): the thread of (x, k) keeps
// E_k(x) and the 8 x 8 adjoint matrix of its link, R_ab = 2 Tr(T^a U T^b U^+),
// in registers for the whole launch, and a sweep exchanges only
//   T_k(x) = U^+ E U = R^T E     with the thread of (x + k, k), and
//   G(x)                          with the threads of (x - k, k),
// eight numbers each.  In coordinates (M = m_a T^a, [m]_a = 2 Tr(T^a M))
//   G(x)_a = sum_k (E_k(x) - T_k(x-k))_a / a_k / a0,   deviation max |G_a|,
//   E_k <- E_k + kdt (1/2 d_abc (R G(x))_b G(x+k)_c - G(x)_a),
// with SU(3)'s symmetric d_abc: 190 FMAs in place of the 540 of five 3x3
// products.
//
// The threads wait for each other's numbers, not for a grid barrier: a
// message is ten 8-byte words that each carry seven bytes of it and a one-byte
// tag, the number of the message in its slot, so that a reader that sees its
// tag in all ten words (8-byte accesses do not tear) has the message.  A slot
// is free again when its next message is written: the writer of T_k(x) has
// read the G(x+k) to which this T went, and the writer of G(x) the T_k(x-k) of
// every reader, each after the reader had read it.  All blocks are resident
// (cooperative launch) and every wait is bounded: one that runs out records
// NRQ_ERR_TIMEOUT in *err, and each warp that finds it there returns.
//
// Bound: the latency of two exchanges through L2 a sweep, about 1.1 us each.
// 24^3: 3.3 us a sweep (two launches a sweep: 17), 8^3 2.6.  The lanes of a
// warp are ten sites x three directions, so that G(x) is a sum of three lanes'
// numbers.  Two rows of R lie in shared memory: with all of it in registers
// (168 a thread at ten warps) a sweep takes 3.5 us, with three rows the same
// 3.3.
namespace {
constexpr int kRunSitesWarp = 10;  // sites of a warp
constexpr int kRunWarps = 10;      // warps of a block, one block an SM
constexpr int kRegRows = 6;        // rows of R in registers, the others in shared memory

// 2 Tr(T^8 T^8) - 1 of the generators' double entries: the factor by which a
// sweep on 3x3 matrices moves E_8 each time it takes its coordinates, 3e-13
// after a thousand sweeps and kept here
constexpr double kT8 = 0x1.35cf5e19f6cf7p-52;

struct Msg {
  ulonglong2 q[5];
};
__device__ __forceinline__ unsigned long long word(uint32_t lo, uint32_t hi) {
  return (unsigned long long)hi << 32 | lo;
}
__device__ __forceinline__ Msg pack(const double (&v)[8], uint32_t tag) {
  uint32_t lo[8], hi[8];
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    lo[a] = (uint32_t)__double2loint(v[a]);
    hi[a] = (uint32_t)__double2hiint(v[a]);
  }
  // the low bytes: bytes 1-7 of the ninth word, byte 1 of the tenth
  const uint32_t w8l = tag | (lo[0] & 0xff) << 8 | (lo[1] & 0xff) << 16 | lo[2] << 24;
  const uint32_t w8h = (lo[3] & 0xff) | (lo[4] & 0xff) << 8 | (lo[5] & 0xff) << 16 | lo[6] << 24;
  const uint32_t w9l = tag | (lo[7] & 0xff) << 8;
  Msg m;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    m.q[j] = make_ulonglong2(word((lo[2 * j] & ~0xffu) | tag, hi[2 * j]),
                             word((lo[2 * j + 1] & ~0xffu) | tag, hi[2 * j + 1]));
  m.q[4] = make_ulonglong2(word(w8l, w8h), word(w9l, 0u));
  return m;
}
__device__ __forceinline__ void unpack(const Msg &m, double (&v)[8]) {
  const uint32_t w8l = (uint32_t)m.q[4].x, w8h = (uint32_t)(m.q[4].x >> 32), w9l = (uint32_t)m.q[4].y;
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const unsigned long long w = (a & 1) ? m.q[a >> 1].y : m.q[a >> 1].x;
    const uint32_t b = a < 3 ? w8l >> (8 * (a + 1)) : a < 7 ? w8h >> (8 * (a - 3)) : w9l >> 8;
    v[a] = __hiloint2double((int)(w >> 32), (int)(((uint32_t)w & ~0xffu) | (b & 0xffu)));
  }
}
// (vector accesses are as many accesses of their element's type: 8-byte
// elements, so that a word is never seen in part)
__device__ __forceinline__ void send(ulonglong2 *p, const ulonglong2 &q) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(q.x), "l"(q.y) : "memory");
}
// the warp's lanes wait for the message `tag` in their slots p[j*stride]
__device__ __forceinline__ bool receive(const ulonglong2 *p, int64_t stride, uint32_t tag, Msg &m, int *err,
                                        long long wait_cycles) {
  long long t0 = 0;
  for (int spins = 0;; ++spins) {
#pragma unroll
    for (int j = 0; j < 5; ++j)
      asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];"
                   : "=l"(m.q[j].x), "=l"(m.q[j].y)
                   : "l"(p + j * stride)
                   : "memory");
    uint32_t off = 0;
#pragma unroll
    for (int j = 0; j < 5; ++j) off |= ((uint32_t)m.q[j].x ^ tag) | ((uint32_t)m.q[j].y ^ tag);
    if (__all_sync(0xffffffffu, (off & 0xffu) == 0)) return true;
    if ((spins & 63) == 63) {
      if (t0 == 0) t0 = clock64();
      const bool late = clock64() - t0 > wait_cycles;
      if (late) atomicExch(err, NRQ_ERR_TIMEOUT);
      if (__any_sync(0xffffffffu, late || *(volatile int *)err != 0)) return false;
    }
  }
}
// 2 Re Tr(T^a A B) of A = x_a T^a, B = y_a T^a: 1/2 d_abc x_b y_c
__device__ __forceinline__ void half_d(const double (&x)[8], const double (&y)[8], double (&v)[8]) {
  const double r = 0.5 / 1.7320508075688772, h = 0.25;
  auto s = [&](int i, int j) { return fma(x[i], y[j], x[j] * y[i]); };
  v[0] = r * s(0, 7) + h * (s(3, 5) + s(4, 6));
  v[1] = r * s(1, 7) + h * (s(4, 5) - s(3, 6));
  v[2] = r * s(2, 7) + h * (fma(x[3], y[3], x[4] * y[4]) - fma(x[5], y[5], x[6] * y[6]));
  v[3] = h * (s(0, 5) - s(1, 6) + s(2, 3)) - 0.5 * r * s(3, 7);
  v[4] = h * (s(0, 6) + s(1, 5) + s(2, 4)) - 0.5 * r * s(4, 7);
  v[5] = h * (s(0, 3) + s(1, 4) - s(2, 5)) - 0.5 * r * s(5, 7);
  v[6] = h * (s(0, 4) - s(1, 3) - s(2, 6)) - 0.5 * r * s(6, 7);
  v[7] = r * (fma(x[0], y[0], fma(x[1], y[1], x[2] * y[2])) - x[7] * y[7]) -
         0.5 * r * (fma(x[3], y[3], x[4] * y[4]) + fma(x[5], y[5], x[6] * y[6]));
}
}  // namespace

// dev[n*nwarps + w]: the deviation before sweep n = 0..nsweeps over warp w's
// sites; Eout may be Ein.  Messages are numbered from te (T) and ge (G).
__global__ void __launch_bounds__(32 * kRunWarps, 1)
    k_gauss_run(Lat L, const double2 *__restrict__ U, const double *Ein, double *Eout, ulonglong2 *T, ulonglong2 *G,
                double *__restrict__ dev, int nwarps, int nsweeps, uint32_t te, uint32_t ge, double kdt, int *err,
                long long wait_cycles) {
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= nwarps) return;
  const int V = (int)L.V, lane = threadIdx.x & 31;
  const int l = lane < 30 ? lane : 29, k = l / kRunSitesWarp, i = l - k * kRunSitesWarp;
  const int site = w * kRunSitesWarp + i;
  const bool act = lane < 30 && site < V;
  const int x = site < V ? site : V - 1;  // lanes without a site follow the last one's
  const Pos32 p = pos32(L, (uint32_t)x);
  const int xm = (int)bwd32(L, p, k), xp = (int)fwd32(L, p, k);
  __shared__ double Rs[8 - kRegRows][8][32 * kRunWarps];
  double Rr[kRegRows][8], e[8];
  auto R = [&](int a, int b) {  // (volatile: kept where it is)
    return a < kRegRows ? Rr[a < kRegRows ? a : 0][b]
                        : *(volatile double *)&Rs[a < kRegRows ? 0 : a - kRegRows][b][threadIdx.x];
  };
  {
    const m3 u = load_link(U, V, x, k);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      double unit[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      unit[b] = 1.0;
      cplx tr[8];
      traces_with_generators(mul_nd(mul(u, algebra_matrix(unit)), u), tr);
#pragma unroll
      for (int a = 0; a < 8; ++a)
        if (a < kRegRows)
          Rr[a < kRegRows ? a : 0][b] = 2.0 * tr[a].re;
        else
          Rs[a < kRegRows ? 0 : a - kRegRows][b][threadIdx.x] = 2.0 * tr[a].re;
    }
#pragma unroll
    for (int a = 0; a < 8; ++a) e[a] = Ein[(int64_t)(k * 8 + a) * V + x];
  }
  const double c = 1.0 / (L.a[k] * L.a0);
  ulonglong2 *const Tw = T + (int64_t)k * V + x, *const Gw = G + x;
  const ulonglong2 *const Tr = T + (int64_t)k * V + xm, *const Gr = G + xp;
  for (int n = 0;; ++n) {
    Msg m;
    double v[8], g[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      double t = R(0, a) * e[0];
#pragma unroll
      for (int b = 1; b < 8; ++b) t = fma(R(b, a), e[b], t);
      v[a] = t;
    }
    m = pack(v, (te + n) & 0xffu);
    if (act)
#pragma unroll
      for (int j = 0; j < 5; ++j) send(Tw + (int64_t)(3 * j) * V, m.q[j]);
    if (!receive(Tr, 3 * (int64_t)V, (te + n) & 0xffu, m, err, wait_cycles)) return;
    unpack(m, v);
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const double q = c * (e[a] - v[a]);
      g[a] = __shfl_sync(0xffffffffu, q, i) + __shfl_sync(0xffffffffu, q, i + kRunSitesWarp) +
             __shfl_sync(0xffffffffu, q, i + 2 * kRunSitesWarp);
    }
    if (n < nsweeps) {
      m = pack(g, (ge + n) & 0xffu);
      if (act)
#pragma unroll
        for (int j = 0; j < 5; ++j)
          if (j % 3 == k) send(Gw + (int64_t)j * V, m.q[j]);
    }
    double mx = 0.0;
#pragma unroll
    for (int a = 0; a < 8; ++a) mx = fmax(mx, fabs(g[a]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) dev[(int64_t)n * nwarps + w] = mx;
    if (n >= nsweeps) break;
    double r[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      double t = R(a, 0) * g[0];
#pragma unroll
      for (int b = 1; b < 8; ++b) t = fma(R(a, b), g[b], t);
      r[a] = t;
    }
    if (!receive(Gr, V, (ge + n) & 0xffu, m, err, wait_cycles)) return;
    double gn[8];
    unpack(m, gn);
    half_d(r, gn, v);
#pragma unroll
    for (int a = 0; a < 8; ++a) e[a] += fma(kdt, v[a] - g[a], a == 7 ? kT8 * e[7] : 0.0);
  }
  if (act)
#pragma unroll
    for (int a = 0; a < 8; ++a) Eout[(int64_t)(k * 8 + a) * V + x] = e[a];
}

// out[n] = the deviation before sweep n, over all warps (one block per n)
__global__ void __launch_bounds__(256) k_gauss_dev(const double *__restrict__ dev, int nwarps,
                                                   double *__restrict__ out) {
  __shared__ double sh[8];
  const double *d = dev + (int64_t)blockIdx.x * nwarps;
  double mx = 0.0;
  for (int w = threadIdx.x; w < nwarps; w += blockDim.x) mx = fmax(mx, d[w]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int j = 1; j < 8; ++j) mx = fmax(mx, sh[j]);
    out[blockIdx.x] = mx;
  }
}

int gauss_run_warps(int64_t V) { return (int)((V + kRunSitesWarp - 1) / kRunSitesWarp); }
bool gauss_run_applicable(int64_t V, int sm_count) {
  return V <= (int64_t)kRunSitesWarp * kRunWarps * sm_count;
}
int64_t gauss_run_message_bytes(int64_t V) { return 80 * 4 * V; }

cudaError_t launch_gauss_run(Lat L, const double2 *U, const double *Ein, double *Eout, void *messages, double *dev,
                             double *devmax, int nsweeps, uint32_t te, uint32_t ge, double kdt, int sm_count, int *err,
                             cudaStream_t st, long long wait_cycles, bool stall) {
  int nwarps = gauss_run_warps(L.V);
  if (stall && nwarps > 1) --nwarps;
  const int per = (nwarps + sm_count - 1) / sm_count;  // warps a block: spread over the SMs
  const unsigned grid = (unsigned)((nwarps + per - 1) / per);
  ulonglong2 *T = (ulonglong2 *)messages, *G = T + 15 * L.V;
  void *args[] = {&L, &U, &Ein, &Eout, &T, &G, &dev, &nwarps, &nsweeps, &te, &ge, &kdt, &err, &wait_cycles};
  const cudaError_t e = cudaLaunchCooperativeKernel((const void *)k_gauss_run, dim3(grid), dim3(32 * per), args, 0, st);
  if (e != cudaSuccess) return e;
  k_gauss_dev<<<(unsigned)nsweeps + 1, 256, 0, st>>>(dev, nwarps, devmax);
  return cudaGetLastError();
}

}  // namespace nrq
