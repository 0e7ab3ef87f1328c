// Device code shared by the spin-structured stencils (cn_spin.cu in FP64,
// cn_spin32.cu the FP32 Chebyshev step): one application of A^H - 1 to a
// unit of 32 sites, one propagator column of both species a warp.  The
// operator, the split of the work and the pipeline are described in
// cn_spin.cu.
#pragma once
#include "nrq_kernels.cuh"
#include "pdl.cuh"
#include "stage.cuh"

namespace nrq {
namespace spin {

constexpr int kUnit = 32;   // sites of a block, one per lane
constexpr int kWarps = 6;   // one propagator column of both species each

template <typename T>
struct Num;
template <>
struct Num<double> {
  using v2 = double2;
  // Spinor operands in registers: this step's and the next three's; matrices
  // staged two neighbours ahead.  (64^3, a coupled step: 4.24 ms with the
  // next two and one neighbour, 4.09 with the next three, 4.02 with both.
  // Prefetches to L2, of the epilogue's operands or of later units', cost
  // 2-20 %; a persistent form with the next unit's first loads issued early
  // 10 %.)
  static constexpr int kAhead = 4, kDist = 2;  // kAhead >= 3: the input at the site itself stays
};
template <>
struct Num<float> {
  using v2 = float2;
  static constexpr int kAhead = 3, kDist = 1;
};
template <typename T>
struct cx {
  T re, im;
};
__device__ __forceinline__ double fma_(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fma_(float a, float b, float c) { return fmaf(a, b, c); }

__device__ __forceinline__ void cp_async(uint32_t dst, const double2 *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async(uint32_t dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async(uint32_t dst, const float2 *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async(uint32_t dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
// arrives on bar once this thread's copies so far have landed
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// acc += +-(w or conj(w)) p: the products with Re w, then those with Im w
template <int S, typename T, typename V>
__device__ __forceinline__ void smac_re(cx<T> &acc, const V w, const V p) {
  const T wr = S > 0 ? w.x : -w.x;
  acc.re = fma_(wr, p.x, acc.re);
  acc.im = fma_(wr, p.y, acc.im);
}
template <int S, bool CJ, typename T, typename V>
__device__ __forceinline__ void smac_im(cx<T> &acc, const V w, const V p) {
  const T wi = (S > 0) == !CJ ? w.y : -w.y;
  acc.re = fma_(-wi, p.y, acc.re);
  acc.im = fma_(wi, p.x, acc.im);
}
template <int SA, int SB, bool CJ, typename T, typename V>
__device__ __forceinline__ void smac2(const V w, cx<T> &a, const V p, cx<T> &b, const V q) {
  smac_re<SA>(a, w, p);
  smac_re<SB>(b, w, q);
  smac_im<SA, CJ>(a, w, p);
  smac_im<SB, CJ>(b, w, q);
}
template <int SA, int SB, bool CJ, typename T, typename V>
__device__ __forceinline__ void smac4(const V w, cx<T> &a, const V p, cx<T> &b, const V q, cx<T> &c, const V r,
                                      cx<T> &d, const V s) {
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
template <int I, bool B, typename T, typename V>
__device__ __forceinline__ void products(cx<T> (&a)[4][3], const V (&m)[3][3], const V (&q)[4]) {
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

template <typename T>
struct Smem {
  using V2 = typename Num<T>::v2;
  // staging kDist neighbours ahead needs 2 kDist + 1 buffers (see apply)
  static constexpr int kBufs = 2 * Num<T>::kDist + 1;
  V2 w[kBufs][27][kUnit];
  V2 s0[9][kUnit];
  T s1[9][kUnit];
  uint64_t full[6];  // the matrices of neighbour n (and, n = 0, the site term) landed
};

// barriers of a block; every thread arrives on each once
template <typename T>
__device__ __forceinline__ void init_barriers(Smem<T> &sm) {
  if (threadIdx.x < 6) mbar_init(&sm.full[threadIdx.x], kUnit * kWarps);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
}

// acc = (A^H - 1) in of column c (the warp's) at the lane's site x:
// acc[species*2 + spin][colour]; the input at x itself is left in
// own[(18 + colour) % kAhead].  W, S0, S1: the operator's planes.  The kernel
// before this one on the stream may still run (pdl.cuh) until the input is
// read; early: the operator is none of its results, so that the first matrices
// are staged before that.  Returns false where a wait ran out.
template <typename T>
__device__ __forceinline__ bool apply(const Lat &L, const typename Num<T>::v2 *__restrict__ W,
                                      const typename Num<T>::v2 *__restrict__ S0, const T *__restrict__ S1,
                                      const typename Num<T>::v2 *__restrict__ in, int x, int c, Smem<T> &sm, int *err,
                                      long long wait_cycles, int stall_load, bool early, cx<T> (&acc)[4][3],
                                      typename Num<T>::v2 (&own)[Num<T>::kAhead][4]) {
  using V2 = typename Num<T>::v2;
  constexpr int kAhead = Num<T>::kAhead, kDist = Num<T>::kDist, kBufs = Smem<T>::kBufs;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t V = L.V;
  int nbr[6];
  neighbours(L, x, nbr);
  auto stage = [&](int n) {
    if (stall_load >= 0 && n >= stall_load) return;
    const V2 *w = W + (int64_t)((n >> 1) * 27) * V + ((n & 1) ? nbr[n] : x);
    for (int p = warp; p < 27; p += kWarps) cp_async(smem_u32(&sm.w[n % kBufs][p][lane]), w + (int64_t)p * V);
    if (n == 0)
      for (int p = warp; p < 9; p += kWarps) {
        cp_async(smem_u32(&sm.s0[p][lane]), S0 + (int64_t)p * V + x);
        cp_async(smem_u32(&sm.s1[p][lane]), S1 + (int64_t)p * V + x);
      }
    cp_async_arrive(&sm.full[n]);
  };
  // operand of step t: neighbour t / 3 (18 and on: the site itself), input
  // colour t % 3
  const V2 *pq = in + (int64_t)(6 * c) * V, *pa = in + (int64_t)(36 + 6 * c) * V;
  auto load = [&](int t, V2(&q)[4]) {
    const int y = t < 18 ? nbr[t / 3] : x;
    const int64_t o = (int64_t)(2 * (t % 3)) * V + y;
    q[0] = __ldca(pq + o);
    q[1] = __ldca(pq + o + V);
    q[2] = __ldca(pa + o);
    q[3] = __ldca(pa + o + V);
  };
  if (!early) pdl_wait();
  stage(0);
  if (early) pdl_wait();
  pdl_trigger();
#pragma unroll
  for (int t = 0; t < kAhead - 1; ++t) load(t, own[t]);
#pragma unroll
  for (int n = 1; n < kDist; ++n) stage(n);
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int i = 0; i < 3; ++i) acc[s][i] = {T(0), T(0)};
  bool ok = true;
#pragma unroll
  for (int n = 0; n < 6; ++n) {
    if (ok && !mbar_try_wait(&sm.full[n], 0)) {
      const long long t0 = clock64();
      while (ok && !mbar_try_wait(&sm.full[n], 0)) ok = clock64() - t0 <= wait_cycles;
      if (!ok) record_timeout(err, sizeof(T) == 8 ? 5 : 6, 0, n);
    }
    if (!__all_sync(0xffffffffu, ok)) return false;
    // every warp issued its copies of n when it entered neighbour n - kDist,
    // so all have left n - kDist - 1, whose buffer n + kDist takes
    if (n + kDist < 6) stage(n + kDist);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int t = 3 * n + j;
      if (t + kAhead - 1 < 21) load(t + kAhead - 1, own[(t + kAhead - 1) % kAhead]);
      V2 m[3][3];
#pragma unroll
      for (int t3 = 0; t3 < 3; ++t3)
#pragma unroll
        for (int i = 0; i < 3; ++i) m[t3][i] = sm.w[n % kBufs][t3 * 9 + ((n & 1) ? 3 * j + i : 3 * i + j)][lane];
      const V2(&q)[4] = own[t % kAhead];
      if (n == 0) products<0, false>(acc, m, q);
      if (n == 1) products<0, true>(acc, m, q);
      if (n == 2) products<1, false>(acc, m, q);
      if (n == 3) products<1, true>(acc, m, q);
      if (n == 4) products<2, false>(acc, m, q);
      if (n == 5) products<2, true>(acc, m, q);
    }
  }
  // the site term, i (S0 +- S1)
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    if (18 + j + kAhead - 1 < 21) load(18 + j + kAhead - 1, own[(18 + j + kAhead - 1) % kAhead]);
    const V2(&q)[4] = own[(18 + j) % kAhead];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const V2 d = sm.s0[i * 3 + j][lane];
      const T b = sm.s1[i * 3 + j][lane];
      const T gq = d.x + b, ga = d.x - b;
#pragma unroll
      for (int s = 0; s < 4; ++s) {  // += i (g + i d.y) q
        const T g = s < 2 ? gq : ga;
        acc[s][i].re = fma_(-g, q[s].y, fma_(-d.y, q[s].x, acc[s][i].re));
        acc[s][i].im = fma_(g, q[s].x, fma_(-d.y, q[s].y, acc[s][i].im));
      }
    }
  }
  return true;
}

// a batch's work item: blocks run over (field, unit), field fastest (order
// 0) or unit fastest (order 1)
__device__ __forceinline__ void batch_item(int nf, int nunits, int order, int &f, int &u) {
  const int w = (int)blockIdx.x;
  if (order == 0) {
    f = w % nf;
    u = w / nf;
  } else {
    f = w / nunits;
    u = w - f * nunits;
  }
}

}  // namespace spin
}  // namespace nrq
