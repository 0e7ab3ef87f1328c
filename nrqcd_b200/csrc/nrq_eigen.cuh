// Complex Jacobi eigen-decomposition of a general 3x3 matrix on the device,
// shared by the CN preparation (field strength via LogU) and the gluon
// observables (ArgLogU of the links).
#pragma once
#include "nrq_common.cuh"

namespace nrq {

// ------------------------------------------------------------ Jacobi log
// Complex Jacobi eigen-decomposition of a general 3x3 matrix, the algorithm
// of src/matrixoperations.f90:327-459 (d = U A U^+, rows of U normalised).
__device__ inline void eigenc3(const m3 &Ain, cplx d[3], m3 &U) {
  const double EPS = 9.860761315262648e-32;  // 2^-103
  m3 A = Ain;
  cplx ev0[3], ev1[3];
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    ev0[p] = {0.0, 0.0};
    ev1[p] = A.e[p * 4];
    d[p] = ev1[p];
  }
  U = m3_id();
  const double red = 0.01 / 81.0;
  for (int sweep = 1; sweep <= 50; ++sweep) {
    double off = 0.0;
    for (int q = 1; q < 3; ++q)
      for (int p = 0; p < q; ++p) {
        double a1 = cabs_(A.e[p * 3 + q]), a2 = cabs_(A.e[q * 3 + p]);
        off = off + a1 * a1 + a2 * a2;
      }
    if (off <= EPS) break;
    double thresh = (sweep < 4) ? off * red : 0.0;
    for (int q = 1; q < 3; ++q) {
      for (int p = 0; p < q; ++p) {
        double a1 = cabs_(A.e[p * 3 + q]), a2 = cabs_(A.e[q * 3 + p]);
        off = a1 * a1 + a2 * a2;
        double e1 = cabs_(ev1[p]), e2 = cabs_(ev1[q]);
        if (sweep > 4 && off < EPS * (e1 * e1 + e2 * e2)) {
          A.e[p * 3 + q] = {0.0, 0.0};
          A.e[q * 3 + p] = {0.0, 0.0};
        } else if (off > thresh) {
          cplx delta = A.e[p * 3 + q] * A.e[q * 3 + p];
          cplx x = 0.5 * (ev1[p] - ev1[q]);
          cplx y = csqrt_(x * x + delta);
          cplx t = x - y;
          cplx s = x + y;
          if (cabs_(t) < cabs_(s)) t = s;
          t = cdiv({1.0, 0.0}, t);
          delta = delta * t;
          ev0[p] = ev0[p] + delta;
          ev1[p] = d[p] + ev0[p];
          ev0[q] = ev0[q] - delta;
          ev1[q] = d[q] + ev0[q];
          cplx invc = csqrt_(delta * t + cplx{1.0, 0.0});
          s = cdiv(t, invc);
          t = cdiv(t, invc + cplx{1.0, 0.0});
          cplx sx = s * A.e[p * 3 + q], ty = t * A.e[p * 3 + q];
          cplx sy = s * A.e[q * 3 + p], tx = t * A.e[q * 3 + p];
          for (int j = 0; j < 3; ++j) {
            x = A.e[j * 3 + p];
            y = A.e[j * 3 + q];
            A.e[j * 3 + p] = x + sy * (y - ty * x);
            A.e[j * 3 + q] = y - sx * (x + tx * y);
            x = A.e[p * 3 + j];
            y = A.e[q * 3 + j];
            A.e[p * 3 + j] = x + sx * (y - tx * x);
            A.e[q * 3 + j] = y - sy * (x + ty * y);
          }
          A.e[p * 3 + q] = {0.0, 0.0};
          A.e[q * 3 + p] = {0.0, 0.0};
          for (int j = 0; j < 3; ++j) {
            x = U.e[p * 3 + j];
            y = U.e[q * 3 + j];
            U.e[p * 3 + j] = x + sx * (y - tx * x);
            U.e[q * 3 + j] = y - sy * (x + ty * y);
          }
        }
      }
    }
    for (int p = 0; p < 3; ++p) {
      ev0[p] = {0.0, 0.0};
      d[p] = ev1[p];
    }
  }
  for (int p = 0; p < 3; ++p) {
    double nrm = 0.0;
    for (int q = 0; q < 3; ++q) nrm += norm2(U.e[p * 3 + q]);
    nrm = 1.0 / sqrt(nrm);
    for (int q = 0; q < 3; ++q) U.e[p * 3 + q] = nrm * U.e[p * 3 + q];
  }
}

// ------------------------------------------------------------ unitary log
// c_n = 2^2n (n!)^2 / (2n+1)!, the coefficients of the series below
constexpr int kLogTerms = 144;
struct LogCoef {
  double c[kLogTerms];
};
constexpr LogCoef make_log_coef() {
  LogCoef t{};
  t.c[0] = 1.0;
  for (int n = 1; n < kLogTerms; ++n) t.c[n] = t.c[n - 1] * (2.0 * n) / (2.0 * n + 1.0);
  return t;
}
static __constant__ LogCoef c_log = make_log_coef();

// H with P = exp(iH) and eigenphases theta in (-pi, pi), for unitary P whose
// sin^2(theta/2) stay below 3/4, without an eigen-decomposition.  Euler's
// series of the arctangent at tan(theta/2) reads
//   theta = sin(theta) sum_n c_n y^n,   y = sin^2(theta/2),
// so H = K sum_n c_n Y^n with K = (P - P^+)/(2i) = sin H and
// Y = (2 - P - P^+)/4 = sin^2(H/2), which commute.  The sum is taken by
// Horner's rule on three real coefficients (Y^3 = t1 Y^2 - t2 Y + t3 by
// Cayley-Hamilton, Y hermitian), as many terms as the largest eigenvalue,
// bounded by rho = |Y|_F, needs for 1e-17: about 20 for plaquettes of a
// thermal field.  The Jacobi route takes any unitary matrix but diverges
// over a warp and costs 2-3 times the rest of the preparation: false asks
// for it.  The line rho = 3/4 needs 137 terms, still under the Jacobi
// sweeps' time; beyond it the terms grow as 1 / (1 - rho).
// The Jacobi route takes the phases of the eigenvalues, whatever their moduli;
// the series sees a defect |P^+ P - 1| as an error of up to three times that,
// so it takes what is unitary to 1e-12, and with small_angle also plaquettes
// of FP32 links (defects of some 1e-7) below |sin H| = 0.3, where the error
// stays below the defect times the angle.
__device__ __forceinline__ bool log_unitary(const m3 &P, m3 &H, bool small_angle) {
  double defect = 0.0;
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = r; c < 3; ++c) {
      cplx q = {r == c ? -1.0 : 0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 3; ++k) cmac_cj(q, P.e[k * 3 + r], P.e[k * 3 + c]);
      defect = fma(r == c ? 1.0 : 2.0, norm2(q), defect);
    }
  m3 K, Y;
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const cplx a = P.e[r * 3 + c], b = conj(P.e[c * 3 + r]);
      K.e[r * 3 + c] = {0.5 * (a.im - b.im), -0.5 * (a.re - b.re)};
      Y.e[r * 3 + c] = {(r == c ? 0.5 : 0.0) - 0.25 * (a.re + b.re), -0.25 * (a.im + b.im)};
    }
  const m3 Y2 = mul(Y, Y);
  const double t1 = Y.e[0].re + Y.e[4].re + Y.e[8].re;
  const double ty2 = Y2.e[0].re + Y2.e[4].re + Y2.e[8].re;
  if (!(ty2 <= 0.5625) || !(defect <= (small_angle && ty2 <= 5.5e-4 ? 1e-10 : 1e-24))) return false;
  const double t2 = 0.5 * (t1 * t1 - ty2);
  const cplx det = Y.e[0] * (Y.e[4] * Y.e[8] - Y.e[5] * Y.e[7]) - Y.e[1] * (Y.e[3] * Y.e[8] - Y.e[5] * Y.e[6]) +
                   Y.e[2] * (Y.e[3] * Y.e[7] - Y.e[4] * Y.e[6]);
  const double t3 = det.re;
  // terms: rho^n < 1e-17, rho = sqrt(ty2) <= 3/4
  const int n = min(kLogTerms - 1, (int)(78.3f / -__logf(fmaxf((float)ty2, 1e-34f))) + 2);
  double a = c_log.c[n], b = 0.0, d = 0.0;
  for (int k = n - 1; k >= 0; --k) {
    const double an = fma(d, t3, c_log.c[k]), bn = fma(-d, t2, a), dn = fma(d, t1, b);
    a = an;
    b = bn;
    d = dn;
  }
  m3 f;
#pragma unroll
  for (int k = 0; k < 9; ++k) f.e[k] = b * Y.e[k] + d * Y2.e[k];
  f.e[0].re += a;
  f.e[4].re += a;
  f.e[8].re += a;
  H = mul(K, f);
  return true;
}

}  // namespace nrq
