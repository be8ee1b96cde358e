// rbx_phase.cuh -- FP64 sine and cosine of k-space phases.
#pragma once
#include <cuda_runtime.h>

namespace rbx {

// Largest phase that sincos_phase takes.  A pass checks its atoms and k-vectors
// against it before its loops (a check a phase costs the structure factor a third)
// and leaves what lies beyond, NaN and infinities to the library's sincos.
constexpr double PHASE_MAX = 35184372088832.0;  // 2^45

// |k.r| is at most norm1(k) times norm1(r).
__device__ __forceinline__ double norm1(double x, double y, double z) {
  return fabs(x) + fabs(y) + fabs(z);
}

// sin and cos of t radians, |t| <= PHASE_MAX.  t less its nearest multiple n of pi/2, pi/2 in two
// FP64 parts (Cody and Waite): n times the first part is exact in the fused
// multiply-add and cancels against t without rounding, so the remainder r is
// rounded once.  Then polynomials in r^2 on |r| <= pi/4: the interpolants of
// (sin(r) / r - 1) / r^2 and (cos(r) - 1) / r^2 at the six and seven Chebyshev
// nodes of r^2 in [0, pi^2/16], computed in 60-digit arithmetic (truncation
// 1.3e-17 and 1.2e-19 relative).  Some 20 FP64 instructions, where the library's
// sincos takes about 85, and FP64 issue bounds the passes that call it.
__device__ __forceinline__ void sincos_phase(double t, double* s, double* c) {
  const double kShift = 6755399441055744.0;                 // 1.5 * 2^52
  const double b = fma(t, 0.6366197723675814, kShift);      // 2 / pi
  const int n = __double2loint(b);  // nearest integer, modulo 2^32
  const double m = __dsub_rn(b, kShift);
  double r = fma(m, -1.5707963267948966, t);
  r = fma(m, -6.123233995736766e-17, r);
  const double z = r * r;
  double p = 1.5918129294866608e-10;
  p = fma(p, z, -2.5051131845003624e-08);
  p = fma(p, z, 2.755731610255244e-06);
  p = fma(p, z, -0.00019841269836758574);
  p = fma(p, z, 0.008333333333330948);
  p = fma(p, z, -0.16666666666666666);
  p = fma(r * z, p, r);
  double q = -1.1367998654022494e-11;
  q = fma(q, z, 2.0875886738047052e-09);
  q = fma(q, z, -2.7557315566341895e-07);
  q = fma(q, z, 2.480158729369346e-05);
  q = fma(q, z, -0.0013888888888880775);
  q = fma(q, z, 0.04166666666666664);
  q = fma(q, z, -0.5);
  q = fma(q, z, 1.0);
  const bool odd = n & 1;
  const double ss = odd ? q : p, cc = odd ? p : q;
  *s = __hiloint2double(__double2hiint(ss) ^ ((n << 30) & 0x80000000), __double2loint(ss));
  *c = __hiloint2double(__double2hiint(cc) ^ (((n + 1) << 30) & 0x80000000), __double2loint(cc));
}

// The same for any phase, checked here.
__device__ __forceinline__ void sincos_phase_any(double t, double* s, double* c) {
  if (fabs(t) <= PHASE_MAX)
    sincos_phase(t, s, c);
  else
    sincos(t, s, c);
}

}  // namespace rbx
