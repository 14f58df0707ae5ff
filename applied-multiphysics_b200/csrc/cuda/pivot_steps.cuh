// Eight-column pivot steps shared by the group panel's POTRF and the whole-front kernel: right-looking elimination on the
// unscaled columns with the trailing triangle in C fragments of 8 x 8 tiles. Per step, some warps with one row per lane
// factor the 8 x 8 diagonal tile redundantly in registers -- so no value of the pivot chain crosses lanes -- and eliminate
// their own rows with it (eliminate8), publishing -a and a / d of the step's columns; the trailing tiles then take the
// rank-8 product of the two (step_tile).
#pragma once
#include <cuda_runtime.h>

namespace amp {

// D += A B on an 8 x 8 tile, K = 4: lane (g, t) = (lane / 4, lane % 4) holds A(g, t), B(t, g), D(g, 2 t) and D(g, 2 t + 1)
__device__ __forceinline__ void mma884(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// 1 / d as x f. FP64: Newton's iteration on the hardware estimate x (relative error e below 2^-20):
// 1 / d = x / (1 - e) = x (1 + e)(1 + e^2) up to e^4, x and f apart, so that a product with x can run beside f's chain;
// the estimate flushes results outside the normal range, so it returns false for |d| below 2^-975 or above 2^960 (an
// integer test of the exponent, off the FP64 pipe). Exact: the quotient.
template <bool Exact>
__device__ __forceinline__ bool recip_parts(double d, double &x, double &f) {
  if constexpr (Exact) {
    x = 1.0 / d;
    f = 1.0;
    return true;
  }
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
  const double e = fma(-d, x, 1.0), s = 1.0 + e;
  f = fma(s, e * e, s);
  return ((unsigned)__double2hiint(d) & 0x7fffffffu) - 0x03000000u <= 0x79000000u;
}
// Row stride of the step buffers (8 columns): 16-byte rows, few bank conflicts
constexpr int kColLd = 10;

// C(g, 2 t ..) -= A(g, .) B(., 2 t ..) on an 8 x 8 tile, K = 8: P the negated rows of A, Q the rows of B^T (stride ld)
__device__ __forceinline__ void step_tile(double (&c)[2], const double *P, const double *Q, int ld, int g, int t) {
  const double2 a = *reinterpret_cast<const double2 *>(P + g * ld + 2 * t);
  const double2 b = *reinterpret_cast<const double2 *>(Q + g * ld + 2 * t);
  mma884(c, a.x, b.x);
  mma884(c, a.y, b.y);
}
// One pivot step for row r (one row per lane of the calling warps; rows past the block repeat its last one): the columns
// [k8, k8 + 8) in R (row stride kColLd), their diagonal tile in R's rows k8 ... The first `pivots` columns are pivots
// (all eight unless Partial); the others only take the pivots' updates. Writes -a to Pk and a / d (0 for a column that is
// no pivot) to Qk. LDL^T: |d| < tau counts as -+tau by d's sign (ldlt.mjs:513-522). Returns false, R being unchanged, when
// a pivot is out of the reciprocal estimate's range (then to be repeated with Exact).
// The chain per column is one reciprocal (the hardware estimate and three dependent products) and two products, 58
// clocks in FP64; a step's FP64 issue takes 790 clocks of a warp alone on its scheduler. No branch inside: one around
// the exact reciprocals made a step 1,115 clocks.
template <bool Exact, bool LDLT, bool Partial>
__device__ __forceinline__ bool eliminate8(const double *R, double *Pk, double *Qk, int k8, int r, int pivots, double tau) {
  constexpr int CL = kColLd;
  double dg[8][8], a[8], iv[8];
  bool fine = true;
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j <= i; j += 2) {
      const double2 v = *reinterpret_cast<const double2 *>(R + (k8 + i) * CL + j);
      dg[i][j] = v.x;
      dg[i][j + 1] = v.y;
    }
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    const double2 v = *reinterpret_cast<const double2 *>(R + r * CL + j);
    a[j] = v.x;
    a[j + 1] = v.y;
  }
#pragma unroll
  for (int kk = 0; kk < 8; kk++) {
    double d = dg[kk][kk], x, fr;
    if (LDLT && !(fabs(d) >= tau)) d = d < 0.0 ? -tau : tau;
    if (Partial && kk >= pivots) d = 1.0;
    fine &= recip_parts<Exact>(d, x, fr);
    if (Partial && kk >= pivots) x = 0.0;
    iv[kk] = x * fr;
#pragma unroll
    for (int j = kk + 1; j < 8; j++) {
      const double lj = (dg[j][kk] * x) * fr;  // the update scale; L is scaled with the exact quotient when written
#pragma unroll
      for (int i = j; i < 8; i++) dg[i][j] -= dg[i][kk] * lj;
      a[j] -= a[kk] * lj;
    }
  }
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    double2 v;
    v.x = -a[j];
    v.y = -a[j + 1];
    *reinterpret_cast<double2 *>(Pk + r * CL + j) = v;
    v.x = a[j] * iv[j];
    v.y = a[j + 1] * iv[j + 1];
    *reinterpret_cast<double2 *>(Qk + r * CL + j) = v;
  }
  return fine;
}

}  // namespace amp
