// rbx_phase.cuh -- FP64 sine and cosine of k-space phases.
#pragma once
#include <cuda_runtime.h>

namespace rbx {

// sin and cos of t quarter turns (angle t pi / 2): t minus its nearest integer
// is exact for |t| < 2^51, and two polynomials in r^2 on |r| <= 1/2 follow, the
// interpolants of sin(pi r / 2) / r and (cos(pi r / 2) - 1) / r^2 at the seven
// Chebyshev nodes of r^2 in [0, 1/4], computed in 60-digit arithmetic
// (truncation 3.5e-18 and 1.2e-19; evaluated in FP64 2.2e-16 at most, relative).
// About 21 FP64 instructions; sincos of the phase in radians takes about 85
// (its reduction by pi covers any argument), and FP64 issue bounds both passes:
// with the neutral atoms left out, 46 -> 11 us for the structure factor and
// 38 -> 10 us for the force of 100,003 atoms (10 % charged) x 100 vectors.
__device__ __forceinline__ void sincos_quarter(double t, double* s, double* c) {
  const double kShift = 6755399441055744.0;  // 1.5 * 2^52
  const double b = __dadd_rn(t, kShift);
  const int n = __double2loint(b);  // nearest integer, modulo 2^32
  const double r = __dsub_rn(t, __dsub_rn(b, kShift));
  const double z = r * r;
  double p = 5.633933781537854e-08;
  p = fma(p, z, -3.59864335298231e-06);
  p = fma(p, z, 0.0001604411507421909);
  p = fma(p, z, -0.004681754132340976);
  p = fma(p, z, 0.07969262624604301);
  p = fma(p, z, -0.6459640975062443);
  p = fma(p, z, 1.5707963267948966);
  p *= r;
  double q = -6.329396344967424e-09;
  q = fma(q, z, 4.710678405505227e-07);
  q = fma(q, z, -2.5202039028029178e-05);
  q = fma(q, z, 0.0009192602745468447);
  q = fma(q, z, -0.020863480763340773);
  q = fma(q, z, 0.2536695079010478);
  q = fma(q, z, -1.2337005501361697);
  q = fma(q, z, 1.0);
  const bool odd = n & 1;
  const double ss = odd ? q : p, cc = odd ? p : q;
  *s = __hiloint2double(__double2hiint(ss) ^ ((n << 30) & 0x80000000), __double2loint(ss));
  *c = __hiloint2double(__double2hiint(cc) ^ (((n + 1) << 30) & 0x80000000), __double2loint(cc));
}

}  // namespace rbx
