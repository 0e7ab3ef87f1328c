// FP32 Chebyshev step of the precision forms on the operator in its spin
// structure, rounded to FP32 (cn_spin.cu describes the operator, the split of
// the work and the pipeline).
//
// The inner solve A^H e = r runs the semi-iteration from e_0 = 0:
//   e_1 = r / theta,   e_{k+1} = e_k + c1 (e_k - e_{k-1}) + c2 (r - A^H e_k),
// so e_1 needs no launch, m steps take m - 1, and a launch moves four FP32
// vectors (e_k, r, e_{k-1} read; e_{k+1} over e_{k-1}) where the recurrence
// on (d, r, e) moved seven and its last launch only added d.  r - A^H e is
// formed as (r - e) - (A^H - 1) e, whose rounding is that of the small part.
// The last launch adds e_{k+1} to the FP64 iterate in place of a pass of its
// own, and stores the step's history x - (2b - psi) from it, the FP64
// difference rounded once (the learned form and the batch add e_{k+1} to what
// their start put there instead).
//
// Bound: 64^3, 3.1 KB a site: 0.12 ms at the copy rate, 0.08 ms of FP32
// FMAs; it takes 0.24 ms (the (d, r, e) recurrence on dense 6x6 blocks 0.36,
// and 0.10 more for the final addition), 32 fields at 24^3 0.43 ms (0.74).  The
// last launch, 6.1 KB a site with the history, takes 0.37 ms (0.31 adding to an
// FP32 history; two blocks an SM, 131 registers and no spill: 0.42).
// Four blocks an SM (80 registers) hide the latency of the loads only in
// part.
#include "cn_spin.cuh"

namespace nrq {

namespace {
using namespace spin;

// one launch: the vectors of a field
struct Step32 {
  const float2 *in, *r;  // e_k (first: r itself), r
  const float2 *prev;    // e_{k-1}; null: r / theta
  float2 *out;           // e_{k+1}
  double2 *x;            // last: x += e_{k+1}
  float2 *hist;          // last: history += e_{k+1} (may be null), or with b
  const double2 *b, *psi;  //   history = x - (2b - psi)
  cplx c1[2], c2[2], it[2];
};
struct Batch32 {
  const BatchField *tab;
  int nf, nunits, order, step;
};
__device__ __forceinline__ cx<float> f2(cplx a) { return {(float)a.re, (float)a.im}; }
__device__ __forceinline__ cx<float> cmul(cx<float> a, cx<float> b) {
  return {fmaf(a.re, b.re, -a.im * b.im), fmaf(a.re, b.im, a.im * b.re)};
}

// FIRST: e_2 from r alone (A^H e_1 = A^H r / theta); LAST: into x and the
// history instead of out, 2: the history anew from b and psi.
template <bool FIRST, int LAST, bool BATCH>
__global__ void __launch_bounds__(kUnit *kWarps, LAST ? 3 : 4)
    k_cheb_spin(Lat L, SpinOp32 op, Step32 A, Batch32 Bt, int *err, long long wait_cycles, bool early) {
  constexpr int kAhead = Num<float>::kAhead;
  __shared__ __align__(16) Smem<float> sm;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int V = (int)L.V;
  int u = (int)blockIdx.x;
  if (BATCH) {
    int f;
    batch_item(Bt.nf, Bt.nunits, Bt.order, f, u);
    const BatchField *F = Bt.tab + f;
    if (batch_field_done(*F)) return;
    op.W += (int64_t)F->wblk * 81 * V;
    op.S0 += (int64_t)F->wblk * 9 * V;
    op.S1 += (int64_t)F->wblk * 9 * V;
    // e_{step+2} goes to dA for even steps, dB for odd ones
    const int k = Bt.step;
    A.in = FIRST ? F->r32 : (k & 1) ? F->dA : F->dB;
    A.r = F->r32;
    A.prev = FIRST || k == 1 ? nullptr : (k & 1) ? F->dB : F->dA;
    A.out = (k & 1) ? F->dB : F->dA;
    A.x = F->x;
    A.hist = F->hnew;
#pragma unroll
    for (int sp = 0; sp < 2; ++sp) {
      A.c1[sp] = F->cheb[k].c1[sp];
      A.c2[sp] = F->cheb[k].c2[sp];
      A.it[sp] = F->inv_theta[sp];
    }
  }
  init_barriers(sm);
  const int s = unit_start(L, u) + lane;
  const bool act = s < V;
  const int x = act ? s : V - 1;  // a valid site for the addresses of idle lanes
  cx<float> acc[4][3];
  float2 own[kAhead][4];
  // a negative bound: the test of the timeout path, which stages no matrices
  // from the fourth neighbour on
  const bool ok = apply<float>(L, op.W, op.S0, op.S1, A.in, x, warp, sm, err, llabs(wait_cycles),
                               wait_cycles < 0 ? 3 : -1, early, acc, own);
  cp_async_wait_all();
  if (!ok || !act) return;
#pragma unroll
  for (int sp = 0; sp < 2; ++sp) {
    const cx<float> c1 = f2(A.c1[sp]), c2 = f2(A.c2[sp]), it = f2(A.it[sp]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // three rows at a time
      const int64_t off = (int64_t)(sp * 36 + warp * 6 + 3 * h) * V + x;
      float2 rv[3], pv[3], hv[3];
      double2 xv[3], bv[3], sv[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int64_t o = off + (int64_t)q * V;
        if (!FIRST) rv[q] = __ldca(A.r + o);
        if (!FIRST && A.prev) pv[q] = A.prev[o];
        if (LAST) xv[q] = A.x[o];
        if (LAST == 1 && A.hist) hv[q] = A.hist[o];
        if (LAST == 2) bv[q] = __ldca(A.b + o);
        if (LAST == 2) sv[q] = __ldca(A.psi + o);
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int64_t o = off + (int64_t)q * V;
        const int row = 3 * h + q;
        const float2 w = own[(18 + (row >> 1)) % kAhead][2 * sp + (row & 1)];
        const cx<float> n = acc[2 * sp + (row & 1)][row >> 1];
        cx<float> e, d, res;  // e_k, e_k - e_{k-1}, r - A^H e_k
        if (FIRST) {
          e = cmul(it, {w.x, w.y});
          d = e;
          const cx<float> t = cmul(it, n);
          res = {(w.x - e.re) - t.re, (w.y - e.im) - t.im};
        } else {
          e = {w.x, w.y};
          const cx<float> p = A.prev ? cx<float>{pv[q].x, pv[q].y} : cmul(it, {rv[q].x, rv[q].y});
          d = {e.re - p.re, e.im - p.im};
          res = {(rv[q].x - e.re) - n.re, (rv[q].y - e.im) - n.im};
        }
        const cx<float> a = cmul(c1, d), b = cmul(c2, res);
        const float2 en = make_float2(e.re + (a.re + b.re), e.im + (a.im + b.im));
        if (LAST) {
          const double2 xn = make_double2(xv[q].x + (double)en.x, xv[q].y + (double)en.y);
          A.x[o] = xn;
          if (LAST == 2)
            A.hist[o] = make_float2((float)(xn.x - (2.0 * bv[q].x - sv[q].x)), (float)(xn.y - (2.0 * bv[q].y - sv[q].y)));
          else if (A.hist)
            A.hist[o] = make_float2(hv[q].x + en.x, hv[q].y + en.y);
        } else {
          A.out[o] = en;
        }
      }
    }
  }
}

// m = 1: x += r / theta, and the history as above (n elements a field)
template <bool BATCH>
__global__ void k_cheb_one(int64_t n, Step32 A, const BatchField *__restrict__ tab) {
  if (BATCH) {
    const BatchField *F = tab + blockIdx.y;
    if (batch_field_done(*F)) return;
    A.r = F->r32;
    A.x = F->x;
    A.hist = F->hnew;
    A.it[0] = F->inv_theta[0];
    A.it[1] = F->inv_theta[1];
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float2 r = A.r[i];
    const cx<float> e = cmul(f2(i >= n / 2 ? A.it[1] : A.it[0]), {r.x, r.y});
    const double2 x = A.x[i];
    const double2 xn = make_double2(x.x + (double)e.re, x.y + (double)e.im);
    A.x[i] = xn;
    if (!BATCH && A.b) {
      const double2 b = A.b[i], p = A.psi[i];
      A.hist[i] = make_float2((float)(xn.x - (2.0 * b.x - p.x)), (float)(xn.y - (2.0 * b.y - p.y)));
    } else if (A.hist) {
      const float2 h = A.hist[i];
      A.hist[i] = make_float2(h.x + e.re, h.y + e.im);
    }
  }
}

template <bool BATCH>
void go(bool first, bool last, int64_t blocks, Lat L, const SpinOp32 &op, const Step32 &A, const Batch32 &Bt, int *err,
        cudaStream_t st, long long wait_cycles, bool early) {
  auto run = [&](auto kern) {
    if (BATCH)
      kern<<<(unsigned)blocks, kUnit * kWarps, 0, st>>>(L, op, A, Bt, err, wait_cycles, false);
    else
      launch_pdl(kern, (unsigned)blocks, kUnit * kWarps, 0, st, L, op, A, Bt, err, wait_cycles, early);
  };
  // (a batch's fields carry no b and psi here)
  const bool store = !BATCH && A.b != nullptr;
  if (!last) {
    if (first)
      run(k_cheb_spin<true, 0, BATCH>);
    else
      run(k_cheb_spin<false, 0, BATCH>);
  } else if (store) {
    if (first)
      run(k_cheb_spin<true, BATCH ? 1 : 2, BATCH>);
    else
      run(k_cheb_spin<false, BATCH ? 1 : 2, BATCH>);
  } else {
    if (first)
      run(k_cheb_spin<true, 1, BATCH>);
    else
      run(k_cheb_spin<false, 1, BATCH>);
  }
}
}  // namespace

// The kernel serves any lattice; the line is the one that callers who force the
// step were given (nrq_cn_set_cheb_stencil), and the default choice keeps to it.
bool cheb_spin_applicable(const Lat &L) {
  return L.V >= 36 && L.V <= 0x7fffffffLL && (L.V % 4) == 0 && (L.nx % 2) == 0;
}

void launch_cheb_spin(int step, bool last, Lat L, const SpinOp32 &op, const float2 *r, float2 *ea, float2 *eb,
                      double2 *x, float2 *hist, const double2 *b, const double2 *psi, const ChebCoef &K,
                      const cplx inv_theta[2], bool early, int *err, cudaStream_t st, long long wait_cycles) {
  Step32 A{};
  A.in = step == 0 ? r : (step & 1) ? ea : eb;
  A.r = r;
  A.prev = step <= 1 ? nullptr : (step & 1) ? eb : ea;
  A.out = (step & 1) ? eb : ea;
  A.x = x;
  A.hist = hist;
  A.b = b;
  A.psi = psi;
  for (int sp = 0; sp < 2; ++sp) {
    A.c1[sp] = K.c1[sp];
    A.c2[sp] = K.c2[sp];
    A.it[sp] = inv_theta[sp];
  }
  go<false>(step == 0, last, (L.V + kUnit - 1) / kUnit, L, op, A, Batch32{}, err, st, wait_cycles, early);
}

void launch_cheb_one(int64_t n, const float2 *r, double2 *x, float2 *hist, const double2 *b, const double2 *psi,
                     const cplx inv_theta[2], cudaStream_t st) {
  Step32 A{};
  A.r = r;
  A.x = x;
  A.hist = hist;
  A.b = b;
  A.psi = psi;
  A.it[0] = inv_theta[0];
  A.it[1] = inv_theta[1];
  k_cheb_one<false><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, A, nullptr);
}

void launch_batch_cheb_spin(int step, bool last, int order, Lat L, const SpinOp32 &op, const BatchField *tab,
                            int nfields, int *err, cudaStream_t st, long long wait_cycles) {
  const int nunits = (int)((L.V + kUnit - 1) / kUnit);
  go<true>(step == 0, last, (int64_t)nunits * nfields, L, op, Step32{}, Batch32{tab, nfields, nunits, order, step},
           err, st, wait_cycles, false);
}

void launch_batch_cheb_one(int64_t n, const BatchField *tab, int nfields, cudaStream_t st) {
  const int64_t nb = (n + 255) / 256;
  k_cheb_one<true><<<dim3((unsigned)(nb < 2048 ? nb : 2048), (unsigned)nfields), 256, 0, st>>>(n, Step32{}, tab);
}

}  // namespace nrq
