// quotient.cuh -- several quotients by one divisor.
//
// Plain C++ besides the qualifiers, so that the host tests can compile it.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define DEM_HD __host__ __device__ __forceinline__
#else
#define DEM_HD inline
#endif

namespace demb {

// Several quotients by one divisor, each rounded as the IEEE division rounds
// it.  The contact arithmetic has up to eight by two divisors.  The divisor's
// reciprocal is divided out once and each quotient takes five multiply-adds
// that run side by side: a product within two units in the last place, one
// correction that brings it within one, and a last one whose remainder is
// exact, so that the sum rounds correctly (P. Markstein, Computation of
// elementary functions on the IBM RISC System/6000 processor, IBM J. Res. Dev.
// 34 (1990), theorems on the remainder and on the final rounding).  This holds
// while neither the remainders underflow nor the products overflow:
// quotients() divides plainly unless the divisor and the quotients pass
// div_range() and no numerator is small_num(), conditions joined without
// branches (200 steps of the bed of 1,000,000 spheres: 64.2 ms with one for
// each, 63.1 ms so; 500 of 4,000 spheres, whose forces are zero more often than
// not, 8.03 ms with a branch that sets zeros apart, 7.97 ms so).  Per step,
// plain divisions and so: that bed 354 and 342 us, split 260 and 249 us;
// 150,001 with Adams-Bashforth 72.9 and 68.3 us; gas of 200,003 59.6 and
// 57.5 us; a batch of 16 columns 117 and 111 us.
DEM_HD double quotient(double a, double b, double y) {
  double q = a * y;
  q = fma(fma(-b, q, a), y, q);
  q = fma(fma(-b, q, a), y, q);
  return copysign(q, a);  // of a zero: the divisors here are positive
}
// Divisor b and the sum of the quotients' magnitudes: in the range of quotient()?
constexpr double QUOTIENT_SUM = 0x1p600;
DEM_HD bool div_range(double b, double sum) { return (b > 0x1p-400) & (b < 0x1p400) & (sum < QUOTIENT_SUM); }
// A numerator under 2^-500: with a divisor of that range a quotient by it may
// be subnormal and its remainder inexact.  Zero is exact either way.
constexpr double SMALL_NUM = 0x1p-500;
DEM_HD bool small_num(double a) { return (fabs(a) < SMALL_NUM) & (a != 0.0); }

// q = a / b with y = 1 / b; returns whether the reciprocal served.
template <int N>
DEM_HD bool quotients(const double* a, double b, double y, double* q) {
  double sum = 0.0;
  bool ok = true;
#pragma unroll
  for (int c = 0; c < N; ++c) {
    q[c] = quotient(a[c], b, y);
    sum = sum + fabs(q[c]);
    ok = ok & !small_num(a[c]);
  }
  ok = ok & div_range(b, sum);
  if (!ok) {
#pragma unroll
    for (int c = 0; c < N; ++c) q[c] = a[c] / b;
  }
  return ok;
}
DEM_HD void div3(const double a[3], double b, double y, double q[3]) {
  double d[3];
  quotients<3>(a, b, y, d);
#pragma unroll
  for (int c = 0; c < 3; ++c) q[c] = d[c];  // q may be a
}
DEM_HD void div3(const double a[3], double b, double q[3]) { div3(a, b, 1.0 / b, q); }

// The quotients of a contact by the distance dmag = |dist| of its centres, at
// most rl + ri: the normal dist / dmag, and the lever arms (dmag^2 + rl^2 -
// ri^2) / (2 dmag) and (rl^2 - ri^2) / (2 dmag) (half a quotient is the
// quotient by twice the divisor).  |nrm| is at most one.  With dmag past 2^-200
// the arms' numerators are zero or past 2^-458: differences of doubles, the
// larger of which is at least the square of dmag / 2.
DEM_HD void contact_quotients(const double dist[3], double dmag, double rl, double ri, double nrm[3], double& dcl,
                              double& half) {
  const double num_dcl = dmag * dmag + rl * rl - ri * ri, num_half = rl * rl - ri * ri;
  const double y = 1.0 / dmag;
#pragma unroll
  for (int c = 0; c < 3; ++c) nrm[c] = quotient(dist[c], dmag, y);
  dcl = 0.5 * quotient(num_dcl, dmag, y);
  half = 0.5 * quotient(num_half, dmag, y);
  const bool range = (dmag > 0x1p-200) & div_range(dmag, fabs(dcl) + fabs(half));
  if (!(range & (fabs(dist[0]) >= SMALL_NUM) & (fabs(dist[1]) >= SMALL_NUM) & (fabs(dist[2]) >= SMALL_NUM))) {
    if (!range || small_num(dist[0]) || small_num(dist[1]) || small_num(dist[2])) {
#pragma unroll
      for (int c = 0; c < 3; ++c) nrm[c] = dist[c] / dmag;
      dcl = num_dcl / (2.0 * dmag);
      half = num_half / (2.0 * dmag);
    }
  }
}

}  // namespace demb
