// rbx_pair_device.cuh -- device helpers shared by the pair-force and the
// adjoint kernels: warp sums, the exact FP64 RBL pair classification and its
// fixed-point screen.
#pragma once
#include "rbx_common.cuh"
#include "rbx_kernels.h"

namespace rbx {

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct Classified {
  bool core_active;    // core list and lj126_rs window (r^2 > EPS)
  bool shell_window;   // shell list and rcs window (r_core^2 < r^2 < cut_off^2)
};

__device__ __forceinline__ Classified classify_exact(double d2, const PairParams& pp) {
  Classified c;
  const bool A = d2 < pp.core2_list;
  c.core_active = A && d2 > RBX_EPSILON;  // d2 < rs2 holds: core2_list < rs2
  c.shell_window = !A && d2 < pp.force2_list && d2 > pp.rs2;  // force2_list < rc2
  return c;
}

__device__ __forceinline__ double exact_d2(const PairParams& pp, const double* __restrict__ x,
                                           const double* __restrict__ y,
                                           const double* __restrict__ z, int i, int j) {
  return dist2_list(pp.box, __ldg(x + i), __ldg(y + i), __ldg(z + i), __ldg(x + j),
                    __ldg(y + j), __ldg(z + j));
}

// LJ 12-6 term: sd6 = s6 / r^6 and force/r (lj126_rs,
// src/force/src/lj_op/rocm/lj_op.hip.cu:40-54); r2i = 1 / d2.  Both quotients are
// rounded as a division rounds them: with plain products of r2i the force's error
// is 2.1e-16 of the larger term (rms), with divisions or this 1.2e-16.
struct LjTerm {
  double sd6, f;
};
__device__ __forceinline__ LjTerm lj_term(double eps_ij, double s6, double d2, double r2i) {
  const double d6 = d2 * d2 * d2;
  LjTerm t;
  t.sd6 = d6 == 0.0 ? INFINITY : quotient(s6, d6, r2i * r2i * r2i);
  t.f = quotient(-24.0 * eps_ij * ((2.0 * t.sd6 - 1.0) * t.sd6), d2, r2i);
  return t;
}

// ---------------------------------------------------------------------------
// Candidate classification shared by both forms.
//
// The pair vector in fixed point, d = u_j - u_i (wrapped int32), is the exact
// minimum image of the FP64 pair vector to within 3 units of s_d = L_d/2^32
// per coordinate.  |d|^2 is formed in FP32 in units of s^2, s = L_max/2^32
// (on a box with unequal edges each coordinate is first weighted by
// L_d/L_max, which keeps its error below 3 units of s), and each predicate
// "r^2 < C" is decided when |d|^2 lies outside a guard band [lo, hi] around
// C/s^2 that exceeds every rounding and quantisation error; inside the band
// the reference's FP64 expression (CaculateDistance: i minus j, min image, no
// FMA) decides.  The outcome is therefore identical to the FP64 predicate on
// every pair, in both precision forms.
// ---------------------------------------------------------------------------
// Screened classification; *unsure is set when a threshold band is hit.  The
// band around core2_list and the one around rs2 (which lies just above it)
// are merged into one undecided interval, as are d2 values at or below the
// EPS band: each undecided pair is settled by the FP64 predicate, so five
// comparisons classify a pair.
__device__ __forceinline__ Classified classify_screen(const PairParams& pp, float d2s,
                                                      bool* unsure) {
  const bool A = d2s < pp.sc_core.lo;    // certainly d2 < core2_list
  const bool B = d2s <= pp.sc_rs.hi;     // not certainly d2 > rs2
  const bool C = d2s < pp.sc_force.lo;   // certainly d2 < force2_list
  const bool D = d2s < pp.sc_force.hi;   // not certainly d2 >= force2_list
  const bool E = d2s <= pp.sc_eps.hi;    // not certainly d2 > EPS
  *unsure = (!A && B) || (!C && D) || E;
  Classified c;
  c.core_active = A;
  c.shell_window = !B && C;
  return c;
}

__device__ __forceinline__ float fixed_d2(const uint4& ai, const uint4& aj) {
  const float dx = (float)(int)(aj.x - ai.x), dy = (float)(int)(aj.y - ai.y),
              dz = (float)(int)(aj.z - ai.z);
  return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}
// The same in units of the longest edge's fixed-point step on a box with
// unequal edges (each difference weighted by L_d / L_max).
__device__ __forceinline__ float fixed_d2_weighted(const PairParams& pp, const uint4& ai,
                                                   const uint4& aj) {
  const float dx = (float)(int)(aj.x - ai.x) * pp.sw[0], dy = (float)(int)(aj.y - ai.y) * pp.sw[1],
              dz = (float)(int)(aj.z - ai.z) * pp.sw[2];
  return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

}  // namespace rbx
