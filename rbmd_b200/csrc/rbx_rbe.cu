// rbx_rbe.cu -- Random Batch Ewald k-space kernels for sm_100a.
//
// Work per step is 2 * N * P (atom, k) phase evaluations: one pass builds the
// structure factors rho(k_p) = sum_j q_j exp(i k_p . r_j), one pass scatters
// F_i = q_i sum_p c_p (cos(k_p.r_i) Im rho_p - sin(k_p.r_i) Re rho_p) k_p
// (src/force/src/kspace_calculator_op/rocm/kspace_calculator_op.hip.cu:98-125,
// 238-289, 678-738).  Both passes are SFU/issue bound, not HBM bound: the
// 16-32 B/atom inputs stay in L2.
//
// An atom without a charge adds nothing to rho and feels no k-space force, so
// both passes evaluate phases for the charged atoms only (10 % of an LJ
// electrolyte's atoms, all of a water's).
//
// Plain form: FP64 positions and phases k.r, FP64 sine and cosine.
// Mixed form: 32-bit fixed-point fractional coordinates u = frac((x-lo)/L)*2^32
// so the phase m.u mod 2^32 is exact integer arithmetic; the angle goes to the
// SFU (__sincosf) in FP32; per-thread FP32 partial sums are folded with a
// TwoSum-compensated pair; the cross-block reduction, energy and virial are FP64.
#include <math.h>

#include <type_traits>

#include "rbx_common.cuh"
#include "rbx_kernels.h"
#include "rbx_phase.cuh"

namespace rbx {

// Whether an atom takes part in the k-space sums: a charge, or a coordinate
// that is not finite (which then shows in the sums).
__device__ __forceinline__ bool kspace_atom(double q, double x, double y, double z) {
  return q + 0.0 * (x + y + z) != 0.0;
}

// The largest double with this high word: a bound of nonnegative doubles by the
// integer maximum of their high words (NaN and infinity come out as NaN).
__device__ __forceinline__ double bound_of_hi(unsigned hi) {
  return __hiloint2double((int)hi, -1);
}

// ---------------------------------------------------------------------------
// rho(k) partial sums: block (bx, by) covers atom chunk bx and k-group by.
// A thread owns KPT k-vectors {kg*32*KPT + lane + 32*t} (KPT a template
// parameter, default 4); warps of the block take disjoint atom sub-ranges; the
// block combines its warps in fixed order and writes one partial per k.  No
// atomics: the result is deterministic.
// ---------------------------------------------------------------------------
constexpr int RBE_BLOCK = 256;
constexpr int RBE_WARPS = RBE_BLOCK / 32;

__device__ __forceinline__ int table_pick(const double* cdf, int cnt, double total, uint64_t u53) {
  const double target = (double)u53 * (1.0 / 9007199254740992.0) * total;
  int lo = 0, hi = cnt - 1;  // first index with target < cdf[idx], else cnt - 1
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (target < cdf[mid])
      hi = mid;
    else
      lo = mid + 1;
  }
  const int idx = lo;
  if (idx == 0) return 0;
  return (idx & 1) ? (idx + 1) / 2 : -(idx / 2);
}

// One RBE k-sample s of MD step `step` (RBESampleMH's density, drawn exactly
// per axis): Philox4x32-10 of counter {s, attempt, step} under key (k0, k1),
// the three inverse-CDF picks, |m| = 0 redrawn (at most 64 attempts).  false
// when every attempt gave m = 0.
__device__ __forceinline__ bool rbe_draw(int s, const SampleArgs& sa, const double* w0,
                                         uint64_t step, int m[3]) {
  const double* w1 = w0 + sa.c0;
  const double* w2 = w1 + sa.c1;
  for (int a = 0; a < 64; ++a) {
    uint32_t c[4] = {(uint32_t)s, (uint32_t)(2 * a), (uint32_t)step, (uint32_t)(step >> 32)};
    philox4x32_10(c, sa.key0, sa.key1);
    uint32_t d[4] = {(uint32_t)s, (uint32_t)(2 * a + 1), (uint32_t)step, (uint32_t)(step >> 32)};
    philox4x32_10(d, sa.key0, sa.key1);
    m[0] = table_pick(w0, sa.c0, sa.t0, ((((uint64_t)c[0]) << 32) | c[1]) >> 11);
    m[1] = table_pick(w1, sa.c1, sa.t1, ((((uint64_t)c[2]) << 32) | c[3]) >> 11);
    m[2] = table_pick(w2, sa.c2, sa.t2, ((((uint64_t)d[0]) << 32) | d[1]) >> 11);
    if (m[0] != 0 || m[1] != 0 || m[2] != 0) return true;
  }
  return false;
}

// With sa.tables the k-vectors of the block's k-group are drawn here (one
// per thread, into shared memory) instead of read, from the cumulative tables
// staged in shared memory when they fit: block column 0 also writes them out
// (double and integer copies) and raises sa.status on a failed draw.
constexpr int SAMPLE_TAB_SMEM = 768;  // table entries staged in shared memory

template <int KPT>
__device__ __forceinline__ void rbe_group_samples(const SampleArgs& sa, int p, int kbase,
                                                  int (*s_m)[32 * KPT], bool col0) {
  __shared__ double s_cdf[SAMPLE_TAB_SMEM];
  const int ent = sa.c0 + sa.c1 + sa.c2;
  const bool staged = ent <= SAMPLE_TAB_SMEM;
  if (staged)
    for (int e = threadIdx.x; e < ent; e += blockDim.x) s_cdf[e] = sa.tables[e];
  __syncthreads();
  const double* w0 = staged ? s_cdf : sa.tables;
  const uint64_t step = sa.step_dev ? (uint64_t)(int64_t)*sa.step_dev : sa.step_arg;
  for (int slot = threadIdx.x; slot < 32 * KPT; slot += blockDim.x) {
    const int k = kbase + slot;
    int m[3] = {0, 0, 0};
    if (k < p) {
      const bool ok = rbe_draw(k, sa, w0, step, m);
      if (col0) {
        if (!ok) atomicOr(sa.status, 1);
        sa.mx[k] = m[0];
        sa.my[k] = m[1];
        sa.mz[k] = m[2];
        if (sa.mi) {
          sa.mi[3 * k] = m[0];
          sa.mi[3 * k + 1] = m[1];
          sa.mi[3 * k + 2] = m[2];
        }
      }
    }
    s_m[0][slot] = m[0];
    s_m[1][slot] = m[1];
    s_m[2][slot] = m[2];
  }
  __syncthreads();
}

template <int KPT>
__global__ void __launch_bounds__(RBE_BLOCK)
k_rbe_rho_partial_f64(int n, int p, int chunk, double Lx, double Ly, double Lz, double rLx,
                      double rLy, double rLz,
                      const double* __restrict__ mx, const double* __restrict__ my,
                      const double* __restrict__ mz, const double* __restrict__ q,
                      const double* __restrict__ x, const double* __restrict__ y,
                      const double* __restrict__ z, double* __restrict__ part_re,
                      double* __restrict__ part_im, SampleArgs sa) {
  __shared__ double s_re[RBE_WARPS][(32 * KPT)];
  __shared__ double s_im[RBE_WARPS][(32 * KPT)];
  __shared__ int s_m[3][32 * KPT];
  __shared__ double s_k[3][32 * KPT];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kbase = blockIdx.y * (32 * KPT);
  if (sa.tables) rbe_group_samples<KPT>(sa, p, kbase, s_m, blockIdx.x == 0);
  // the block's k-vectors, k = 2 pi m / L evaluated as (2 pi * m) / L like the
  // reference (rL = 1 / L): formed once, since every warp's own took a fifth of the
  // kernel at 400 vectors
  for (int t = threadIdx.x; t < 96 * KPT; t += RBE_BLOCK) {
    const int d = t / (32 * KPT), s = t % (32 * KPT);
    const double* const m = d == 0 ? mx : (d == 1 ? my : mz);
    const double md = sa.tables ? (double)s_m[d][s] : (kbase + s < p ? m[kbase + s] : 0.0);
    s_k[d][s] = quotient(2 * RBX_PI * md, d == 0 ? Lx : (d == 1 ? Ly : Lz),
                         d == 0 ? rLx : (d == 1 ? rLy : rLz));
  }
  __syncthreads();
  double kx[KPT], ky[KPT], kz[KPT], sr[KPT], si[KPT];
  unsigned kmax_hi = 0;
#pragma unroll
  for (int t = 0; t < KPT; ++t) {
    kx[t] = s_k[0][lane + 32 * t];
    ky[t] = s_k[1][lane + 32 * t];
    kz[t] = s_k[2][lane + 32 * t];
    kmax_hi = max(kmax_hi, (unsigned)__double2hiint(norm1(kx[t], ky[t], kz[t])));
    sr[t] = 0.0;
    si[t] = 0.0;
  }
  const double kmax = bound_of_hi(__reduce_max_sync(0xffffffffu, kmax_hi));
  const int a0 = blockIdx.x * chunk;
  const int a1 = min(n, a0 + chunk);
  const int sub = (chunk + RBE_WARPS - 1) / RBE_WARPS;
  const int w0 = a0 + warp * sub, w1 = min(a1, w0 + sub);
  // 32 atoms at a time, one a lane; the charged ones are then broadcast in
  // atom order
  for (int jt = w0; jt < w1; jt += 32) {
    const int j = jt + lane;
    double xl = 0.0, yl = 0.0, zl = 0.0, ql = 0.0;
    if (j < w1) {
      xl = x[j];
      yl = y[j];
      zl = z[j];
      ql = q[j];
    }
    unsigned m = __ballot_sync(0xffffffffu, kspace_atom(ql, xl, yl, zl));
    if (m == 0) continue;
    const bool small =
        __all_sync(0xffffffffu, norm1(xl, yl, zl) * kmax <= PHASE_MAX);
    auto add = [&](auto phase) {
      for (unsigned left = m; left; left &= left - 1) {
        const int src = __ffs(left) - 1;
        const double xj = __shfl_sync(0xffffffffu, xl, src), yj = __shfl_sync(0xffffffffu, yl, src),
                     zj = __shfl_sync(0xffffffffu, zl, src), qj = __shfl_sync(0xffffffffu, ql, src);
#pragma unroll
        for (int t = 0; t < KPT; ++t) {
          double s, c;
          phase(kx[t] * xj + ky[t] * yj + kz[t] * zj, &s, &c);
          sr[t] += qj * c;
          si[t] += qj * s;
        }
      }
    };
    if (small)
      add([](double t, double* s, double* c) { sincos_phase(t, s, c); });
    else
      add([](double t, double* s, double* c) { sincos(t, s, c); });
  }
#pragma unroll
  for (int t = 0; t < KPT; ++t) {
    s_re[warp][lane + 32 * t] = sr[t];
    s_im[warp][lane + 32 * t] = si[t];
  }
  __syncthreads();
  for (int s = threadIdx.x; s < (32 * KPT); s += RBE_BLOCK) {
    const int k = kbase + s;
    if (k >= p) continue;
    double r = 0.0, im = 0.0;
    for (int w = 0; w < RBE_WARPS; ++w) {
      r += s_re[w][s];
      im += s_im[w][s];
    }
    part_re[(size_t)k * gridDim.x + blockIdx.x] = r;
    part_im[(size_t)k * gridDim.x + blockIdx.x] = im;
  }
}

// TwoSum (Knuth): s + e == a + b exactly.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// Mixed form.  Atom record: {ux, uy, uz, float bits of q}.  Lanes own k-vectors
// (integer m), atoms stream through the warp as broadcast loads.  Every
// RBE_TILE atoms the plain FP32 tile sums are folded into a compensated
// (hi, lo) pair.
constexpr int RBE_TILE = 32;

struct RhoMixedArgs {
  int n, p, chunk;
  const int* mi;
  const uint4* atoms;
  double *part_re, *part_im;
  SampleArgs sa;
  int gx;  // atom chunks (the grid is gx x k-groups)
};

// Block (bx, by) of the replica's grid.
template <int KPT>
__device__ __forceinline__ void rho_mixed_body(const RhoMixedArgs& A, int bx, int by) {
  const int n = A.n, p = A.p, chunk = A.chunk, gx = A.gx;
  const int* __restrict__ mi = A.mi;
  const uint4* __restrict__ atoms = A.atoms;
  double* __restrict__ part_re = A.part_re;
  double* __restrict__ part_im = A.part_im;
  const SampleArgs& sa = A.sa;
  __shared__ double s_re[RBE_WARPS][(32 * KPT)];
  __shared__ double s_im[RBE_WARPS][(32 * KPT)];
  __shared__ int s_m[3][32 * KPT];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kbase = by * (32 * KPT);
  if (sa.tables) rbe_group_samples<KPT>(sa, p, kbase, s_m, bx == 0);
  int m0[KPT], m1[KPT], m2[KPT];
  float hr[KPT], lr[KPT], hi[KPT], li[KPT];
#pragma unroll
  for (int t = 0; t < KPT; ++t) {
    const int k = kbase + lane + 32 * t;
    const bool ok = k < p;
    m0[t] = sa.tables ? s_m[0][lane + 32 * t] : (ok ? mi[3 * k] : 0);
    m1[t] = sa.tables ? s_m[1][lane + 32 * t] : (ok ? mi[3 * k + 1] : 0);
    m2[t] = sa.tables ? s_m[2][lane + 32 * t] : (ok ? mi[3 * k + 2] : 0);
    hr[t] = lr[t] = hi[t] = li[t] = 0.f;
  }
  const float ang = (float)(2.0 * RBX_PI / 4294967296.0);
  const int a0 = bx * chunk;
  const int a1 = min(n, a0 + chunk);
  const int sub = (chunk + RBE_WARPS - 1) / RBE_WARPS;
  const int w0 = a0 + warp * sub, w1 = min(a1, w0 + sub);
  for (int jt = w0; jt < w1; jt += RBE_TILE) {
    const int je = min(w1, jt + RBE_TILE);
    float tr[KPT], ti[KPT];
#pragma unroll
    for (int t = 0; t < KPT; ++t) tr[t] = ti[t] = 0.f;
    // the charged atoms of the tile, in atom order; a mostly charged tile takes
    // every atom (a neutral one adds exact zeros) in a loop without the search
    static_assert(RBE_TILE == 32, "one atom a lane");
    const float ql = jt + lane < je ? __uint_as_float(__ldg(&atoms[jt + lane].w)) : 0.f;
    unsigned m = __ballot_sync(0xffffffffu, ql != 0.f);
    if (m == 0) continue;  // nothing to add to the compensated sums
    auto add = [&](int j) {
      const uint4 a = __ldg(atoms + j);
      const float qj = __uint_as_float(a.w);
#pragma unroll
      for (int t = 0; t < KPT; ++t) {
        const unsigned ph = (unsigned)m0[t] * a.x + (unsigned)m1[t] * a.y + (unsigned)m2[t] * a.z;
        float s, c;
        __sincosf((float)(int)ph * ang, &s, &c);
        tr[t] = fmaf(qj, c, tr[t]);
        ti[t] = fmaf(qj, s, ti[t]);
      }
    };
    if (__popc(m) >= 20) {
      for (int j = jt; j < je; ++j) add(j);
    } else {
      for (; m; m &= m - 1) add(jt + __ffs(m) - 1);
    }
#pragma unroll
    for (int t = 0; t < KPT; ++t) {
      float s, e;
      two_sum(hr[t], tr[t], s, e);
      hr[t] = s;
      lr[t] += e;
      two_sum(hi[t], ti[t], s, e);
      hi[t] = s;
      li[t] += e;
    }
  }
#pragma unroll
  for (int t = 0; t < KPT; ++t) {
    s_re[warp][lane + 32 * t] = (double)hr[t] + (double)lr[t];
    s_im[warp][lane + 32 * t] = (double)hi[t] + (double)li[t];
  }
  __syncthreads();
  for (int s = threadIdx.x; s < (32 * KPT); s += RBE_BLOCK) {
    const int k = kbase + s;
    if (k >= p) continue;
    double r = 0.0, im = 0.0;
    for (int w = 0; w < RBE_WARPS; ++w) {
      r += s_re[w][s];
      im += s_im[w][s];
    }
    part_re[(size_t)k * gx + bx] = r;
    part_im[(size_t)k * gx + bx] = im;
  }
}

template <int KPT>
__global__ void __launch_bounds__(RBE_BLOCK) k_rbe_rho_partial_mixed(RhoMixedArgs a) {
  rho_mixed_body<KPT>(a, blockIdx.x, blockIdx.y);
}

template <int KPT>
__global__ void __launch_bounds__(RBE_BLOCK)
k_rbe_rho_partial_mixed_batch(const RhoMixedArgs* __restrict__ a, const int* __restrict__ start,
                              int nrep) {
  const int r = batch_replica(start, nrep, blockIdx.x);
  const int b = blockIdx.x - __ldg(start + r), gx = a[r].gx;
  rho_mixed_body<KPT>(a[r], b % gx, b / gx);
}

// ---------------------------------------------------------------------------
// Finalize: rho_p = sum over the k-major partials; energy/virial terms
// (ComputeRBEVirial0, kspace_calculator_op.hip.cu:573-674) summed over k in
// fixed order; force table tab[p] = {kx, ky, kz, coef*Re, coef*Im} with coef =
// -4 pi qqr2e S / (P V k^2); optional mean of a force-partial array (RBL mean
// removal).
// ---------------------------------------------------------------------------
constexpr int FIN_BLOCK = 256;

// Energy and virial of structure factors that are already sums: a thread a k,
// then a fixed tree.  (A warp a k with one lane at work, and one thread adding
// the warps' sums, took 9.1 us at 100 vectors.)
__global__ void __launch_bounds__(FIN_BLOCK)
k_rbe_energy_virial(int p, const double* __restrict__ re, const double* __restrict__ im,
                    const double* __restrict__ mx, const double* __restrict__ my,
                    const double* __restrict__ mz, double Lx, double Ly, double Lz, double alpha,
                    double S, double qqr2e, double qsq, double qsum, double* __restrict__ energy,
                    double* __restrict__ virial) {
  __shared__ double s_w[7][FIN_BLOCK / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double V = Lx * Ly * Lz;
  const double coef = (2 * RBX_PI * S) / (p * V);
  double t[7] = {0, 0, 0, 0, 0, 0, 0};
  for (int k = threadIdx.x; k < p; k += FIN_BLOCK) {
    const double r = re[k], i = im[k];
    const double kx = 2 * RBX_PI * mx[k] / Lx;
    const double ky = 2 * RBX_PI * my[k] / Ly;
    const double kz = 2 * RBX_PI * mz[k] / Lz;
    const double k2 = kx * kx + ky * ky + kz * kz;
    const double base = coef * (r * r + i * i) / k2;
    const double inner = (1.0 / (4 * alpha)) + (1.0 / k2);
    t[0] += base;
    t[1] += base * (1.0 - 2 * kx * kx * inner);
    t[2] += base * (1.0 - 2 * ky * ky * inner);
    t[3] += base * (1.0 - 2 * kz * kz * inner);
    t[4] += base * (-2 * kx * ky * inner);
    t[5] += base * (-2 * kx * kz * inner);
    t[6] += base * (-2 * ky * kz * inner);
  }
#pragma unroll
  for (int c = 0; c < 7; ++c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t[c] += __shfl_down_sync(0xffffffffu, t[c], o);
    if (lane == 0) s_w[c][warp] = t[c];
  }
  __syncthreads();
  if (threadIdx.x >= 7) return;
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < FIN_BLOCK / 32; ++w) s += s_w[threadIdx.x][w];
  if (threadIdx.x == 0) {
    const double MY_PIS = 1.77245385090551602729, MY_PI2 = 1.57079632679489661923;
    s -= sqrt(alpha) * qsq / MY_PIS + MY_PI2 * qsum * qsum / (alpha * V);
    *energy = s * qqr2e;
  } else {
    virial[threadIdx.x - 1] = s * qqr2e;
  }
}

// Parallel finalize: block k < p reduces the partials of k-vector k (fixed
// strided order, then a fixed tree) and writes rho(k), the force table entry
// and its seven energy/virial terms to kterm[k][0..6]; blocks p..p+2 reduce
// the per-block pair-force sums into the mean force.  The per-k terms are then
// added in increasing k by one warp in a fixed order (energy_job): in
// k_energy_sum, or in an extra block of the force pass that follows, where
// nothing waits for it (as the finalize's last block, behind a fence and a
// counter, it was 2 us of a 6 us launch that the forces wait for).
constexpr int FK_BLOCK = 128;

__device__ __forceinline__ void energy_job(const EnergyJob& job) {
  const int lane = threadIdx.x & 31, p = job.p;
  double t[7] = {0, 0, 0, 0, 0, 0, 0};
  if (job.kind == EnergyJob::RBE) {
    // each lane adds its k in increasing order; the seven loads of a k are independent
    for (int k = lane; k < p; k += 32)
#pragma unroll
      for (int c = 0; c < 7; ++c) t[c] += job.kterm[(size_t)k * 8 + c];
  } else {
    for (int k = lane; k < p; k += 32) {
      if (job.energy) t[0] += job.kterm[k];
      if (job.vterm)
#pragma unroll
        for (int c = 0; c < 6; ++c) t[1 + c] += job.vterm[6 * (size_t)k + c];
    }
  }
#pragma unroll
  for (int c = 0; c < 7; ++c)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t[c] += __shfl_down_sync(0xffffffffu, t[c], o);
  if (lane != 0) return;
  if (job.kind == EnergyJob::RBE) {
    const double MY_PIS = 1.77245385090551602729, MY_PI2 = 1.57079632679489661923;
    const double etot = t[0] - (sqrt(job.alpha) * job.qsq / MY_PIS +
                                MY_PI2 * job.qsum * job.qsum / (job.alpha * job.V));
    *job.energy = etot * job.qqr2e;
    for (int c = 0; c < 6; ++c) job.virial[c] = t[1 + c] * job.qqr2e;
  } else {
    if (job.energy) *job.energy = t[0] + job.self_energy;
    if (job.vterm)
      for (int c = 0; c < 6; ++c) job.virial[c] = t[1 + c];
  }
}

__global__ void __launch_bounds__(32) k_energy_sum(EnergyJob job) { energy_job(job); }

int launch_energy_sum(const EnergyJob& job, cudaStream_t st) {
  k_energy_sum<<<1, 32, 0, st>>>(job);
  count_launch();
  return check_launch("energy_sum");
}

__device__ void rbe_finalize_one(int k, int p, int nparts, const double* __restrict__ part_re,
                                 const double* __restrict__ part_im, const double* __restrict__ mx,
                                 const double* __restrict__ my, const double* __restrict__ mz,
                                 double Lx, double Ly, double Lz, double alpha, double S,
                                 double qqr2e, double* __restrict__ rho_re,
                                 double* __restrict__ rho_im, KTab* __restrict__ tab,
                                 double* __restrict__ kterm, double* sh);

struct FinalizeArgs {
  int p, nparts;
  const double *part_re, *part_im, *mx, *my, *mz;
  double Lx, Ly, Lz, alpha, S, qqr2e;
  double *rho_re, *rho_im;
  KTab* tab;
  double* kterm;
  int mean_parts;
  const double* fpart;
  double n_atoms;
  double* mean_out;
};

// Block blk.
__device__ __forceinline__ void finalize_k_body(const FinalizeArgs& A, int blk) {
  const int p = A.p, nparts = A.nparts, mean_parts = A.mean_parts;
  const double* __restrict__ part_re = A.part_re;
  const double* __restrict__ part_im = A.part_im;
  const double* __restrict__ fpart = A.fpart;
  double* __restrict__ kterm = A.kterm;
  double* __restrict__ mean_out = A.mean_out;
  const double n_atoms = A.n_atoms;
  __shared__ double sh[2 * FK_BLOCK / 32];
  if (blk >= p) {  // mean of the pair-force block sums, one component per block
    const int d = blk - p;
    double s = 0.0;
    constexpr int U = 16;  // loads in flight per thread
    for (int b0 = threadIdx.x; b0 < mean_parts; b0 += U * FK_BLOCK) {
      double v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int b = b0 + u * FK_BLOCK;
        v[u] = b < mean_parts ? fpart[(size_t)b * 3 + d] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) s += v[u];
    }
    s = block_sum_det<FK_BLOCK>(s, sh);
    if (threadIdx.x == 0) mean_out[d] = s / n_atoms;
  } else {
    rbe_finalize_one(blk, p, nparts, part_re, part_im, A.mx, A.my, A.mz, A.Lx, A.Ly, A.Lz,
                     A.alpha, A.S, A.qqr2e, A.rho_re, A.rho_im, A.tab, kterm, sh);
  }
}

__global__ void __launch_bounds__(FK_BLOCK) k_rbe_finalize_k(FinalizeArgs a) {
  finalize_k_body(a, blockIdx.x);
}

__global__ void __launch_bounds__(FK_BLOCK)
k_rbe_finalize_k_batch(const FinalizeArgs* __restrict__ a, const int* __restrict__ start,
                       int nrep) {
  const int r = batch_replica(start, nrep, blockIdx.x);
  finalize_k_body(a[r], blockIdx.x - __ldg(start + r));
}

// Block k's part of the finalize (all threads of the block call it).
__device__ void rbe_finalize_one(int k, int p, int nparts, const double* __restrict__ part_re,
                                 const double* __restrict__ part_im, const double* __restrict__ mx,
                                 const double* __restrict__ my, const double* __restrict__ mz,
                                 double Lx, double Ly, double Lz, double alpha, double S,
                                 double qqr2e, double* __restrict__ rho_re,
                                 double* __restrict__ rho_im, KTab* __restrict__ tab,
                                 double* __restrict__ kterm, double* sh) {
  // a chain of latencies: every load is issued before the sums, the per-k
  // constants (their FP64 divides) are formed while the loads are in flight,
  // and one barrier serves both sums
  constexpr int U = 8;
  double r = 0.0, im = 0.0;
  const double* pr = part_re + (size_t)k * nparts;
  const double* pi = part_im + (size_t)k * nparts;
  for (int b0 = threadIdx.x; b0 < nparts; b0 += U * FK_BLOCK) {
    double vr[U], vi[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int b = b0 + u * FK_BLOCK;
      vr[u] = b < nparts ? pr[b] : 0.0;
      vi[u] = b < nparts ? pi[b] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      r += vr[u];
      im += vi[u];
    }
  }
  const double V = Lx * Ly * Lz;
  const double kx = 2 * RBX_PI * mx[k] / Lx;
  const double ky = 2 * RBX_PI * my[k] / Ly;
  const double kz = 2 * RBX_PI * mz[k] / Lz;
  const double k2 = kx * kx + ky * ky + kz * kz;
  const double c = (-4 * RBX_PI * qqr2e * S / p) / (V * k2);
  const double e_scale = (2 * RBX_PI * S) / (p * V) / k2;
  const double inner = (1.0 / (4 * alpha)) + (1.0 / k2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    r += __shfl_down_sync(0xffffffffu, r, o);
    im += __shfl_down_sync(0xffffffffu, im, o);
  }
  if ((threadIdx.x & 31) == 0) {
    sh[threadIdx.x >> 5] = r;
    sh[FK_BLOCK / 32 + (threadIdx.x >> 5)] = im;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
#pragma unroll
  for (int w = 1; w < FK_BLOCK / 32; ++w) {
    r += sh[w];
    im += sh[FK_BLOCK / 32 + w];
  }
  if (rho_re) {
    rho_re[k] = r;
    rho_im[k] = im;
  }
  if (kterm) {
    const double base = e_scale * (r * r + im * im);
    double* t = kterm + (size_t)k * 8;
    t[0] = base;
    t[1] = base * (1.0 - 2 * kx * kx * inner);
    t[2] = base * (1.0 - 2 * ky * ky * inner);
    t[3] = base * (1.0 - 2 * kz * kz * inner);
    t[4] = base * (-2 * kx * ky * inner);
    t[5] = base * (-2 * kx * kz * inner);
    t[6] = base * (-2 * ky * kz * inner);
  }
  if (tab) {
    KTab t;
    t.kx = kx;
    t.ky = ky;
    t.kz = kz;
    t.a = c * r;
    t.b = c * im;
    t.m[0] = (int)mx[k];
    t.m[1] = (int)my[k];
    t.m[2] = (int)mz[k];
    t.m[3] = 0;
    tab[k] = t;
  }
}

// ---------------------------------------------------------------------------
// Force scatter over the charged atoms of a block, compacted onto its first
// threads.  FP64: where few are charged, the idle threads share the atoms'
// k-vectors.  An atom's k-vectors fall into eight classes (k modulo 8), each
// summed in increasing k, and the eight sums meet in one tree, in a thread's
// registers or in shuffles: the force is the same to the bit however many
// threads share it, so it depends neither on the block size nor on the charges
// around the atom.  Mixed: one thread an atom, k in increasing order, since FP32
// sums in another order move a force by 1e-7.  The k table is staged in shared
// memory.
// Epilogue variants: plain store of F_k, or the fused combine
// F = F_pair - mean + F_k with the second velocity-Verlet half kick.
// ---------------------------------------------------------------------------
constexpr int FRC_TABLE = 512;  // k entries staged per pass

struct ForceEpilogue {
  const double* f_pair_x;  // may be null: store F_k only
  const double* f_pair_y;
  const double* f_pair_z;
  const double* mean;      // may be null
  double* f_out_x;         // total (or k-space only)
  double* f_out_y;
  double* f_out_z;
  double* fk_x;            // optional copy of the k-space part
  double* fk_y;
  double* fk_z;
  double* vx;              // optional half kick
  double* vy;
  double* vz;
  const int* type;
  const double* inv_mass;  // per type
  double half_dt;
  EnergyJob job;           // the launch's last block, when there is one
};

__device__ __forceinline__ void force_epilogue(const ForceEpilogue& ep, int i, double fx,
                                               double fy, double fz) {
  if (ep.fk_x) {
    ep.fk_x[i] = fx;
    ep.fk_y[i] = fy;
    ep.fk_z[i] = fz;
  }
  if (ep.f_pair_x) {
    double mx = 0, my = 0, mz = 0;
    if (ep.mean) {
      mx = ep.mean[0];
      my = ep.mean[1];
      mz = ep.mean[2];
    }
    fx += ep.f_pair_x[i] - mx;
    fy += ep.f_pair_y[i] - my;
    fz += ep.f_pair_z[i] - mz;
  }
  ep.f_out_x[i] = fx;
  ep.f_out_y[i] = fy;
  ep.f_out_z[i] = fz;
  if (ep.vx) {
    const double im = ep.inv_mass[ep.type[i]] * ep.half_dt;
    ep.vx[i] += fx * im;
    ep.vy[i] += fy * im;
    ep.vz[i] += fz * im;
  }
}

// The charged atoms of a block of FB, in atom order: s_list[0..count).  All
// threads call it; live threads pass their atom's flag.  Ends with a barrier.
template <int FB>
__device__ __forceinline__ int block_compact(bool take, unsigned short* s_list, int* s_cnt) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned m = __ballot_sync(0xffffffffu, take);
  if (lane == 0) s_cnt[warp] = __popc(m);
  __syncthreads();
  int before = 0, count = 0;
#pragma unroll
  for (int w = 0; w < FB / 32; ++w) {
    const int c = s_cnt[w];
    before += w < warp ? c : 0;
    count += c;
  }
  if (take) s_list[before + __popc(m & ((1u << lane) - 1u))] = (unsigned short)threadIdx.x;
  __syncthreads();
  return count;
}

// Threads that share one charged atom's k-vectors: the largest power of two
// (at most the number of classes) that the block has threads for.
constexpr int K_CLASSES = 8;
template <int FB>
__device__ __forceinline__ int threads_per_atom(int count) {
  int s = 1;
  while (s < K_CLASSES && 2 * s * count <= FB) s *= 2;
  return s;
}

// FP64 table entry in shared memory: k, coef Re / Im rho.
struct KTabD {
  double kx, ky, kz, a, b;
};

template <int FB>
__global__ void __launch_bounds__(FB)
k_rbe_force_f64(int n, int p, const KTab* __restrict__ tab, const double* __restrict__ q,
                const double* __restrict__ x, const double* __restrict__ y,
                const double* __restrict__ z, ForceEpilogue ep) {
  if (ep.job.kind != EnergyJob::NONE && blockIdx.x == gridDim.x - 1) {
    if (threadIdx.x < 32) energy_job(ep.job);
    return;
  }
  __shared__ KTabD s_tab[FRC_TABLE];
  __shared__ double s_x[FB], s_y[FB], s_z[FB];  // positions, then forces
  __shared__ unsigned short s_list[FB];
  __shared__ int s_cnt[FB / 32];
  __shared__ unsigned s_far[FB / 32];  // the warps' farthest charged atoms
  const int i = blockIdx.x * FB + threadIdx.x;
  const bool live = i < n;
  const double xi = live ? x[i] : 0.0, yi = live ? y[i] : 0.0, zi = live ? z[i] : 0.0;
  const double qi = live ? q[i] : 0.0;
  const bool take = live && kspace_atom(qi, xi, yi, zi);
  if (take) {
    s_x[threadIdx.x] = xi;
    s_y[threadIdx.x] = yi;
    s_z[threadIdx.x] = zi;
  }
  const int count = block_compact<FB>(take, s_list, s_cnt);
  const unsigned far_hi = __reduce_max_sync(
      0xffffffffu, take ? (unsigned)__double2hiint(norm1(xi, yi, zi)) : 0u);
  if ((threadIdx.x & 31) == 0) s_far[threadIdx.x >> 5] = far_hi;
  const int share = threads_per_atom<FB>(count);
  const int slot = (int)threadIdx.x / share, part = (int)threadIdx.x % share;
  const bool mine = slot < count;
  const int own = mine ? s_list[slot] : 0;
  const double xo = s_x[own], yo = s_y[own], zo = s_z[own];
  // a thread that has its atom to itself does what two would, one after the
  // other: half the accumulators, twice the resident blocks
  double fx = 0.0, fy = 0.0, fz = 0.0;
  for (int half = 0; half < (share == 1 ? 2 : 1); ++half) {
    const int first = share == 1 ? half : part;
    double f[K_CLASSES / 2][3];  // classes first + max(share, 2) c
#pragma unroll
    for (int c = 0; c < K_CLASSES / 2; ++c) f[c][0] = f[c][1] = f[c][2] = 0.0;
    for (int k0 = 0; k0 < p && count > 0; k0 += FRC_TABLE) {
      const int kn = min(FRC_TABLE, p - k0);
      const int kpad = (kn + K_CLASSES - 1) / K_CLASSES * K_CLASSES;
      __syncthreads();
      unsigned rmax_hi = 0;
      for (int w = 0; w < FB / 32; ++w) rmax_hi = max(rmax_hi, s_far[w]);
      const double rmax = bound_of_hi(rmax_hi);
      bool large = false;
      for (int s = threadIdx.x; s < kpad; s += FB) {
        if (s < kn) {
          const KTab& t = tab[k0 + s];
          s_tab[s] = KTabD{t.kx, t.ky, t.kz, t.a, t.b};
          large |= !(norm1(t.kx, t.ky, t.kz) * rmax <= PHASE_MAX);
        } else {
          s_tab[s] = KTabD{0.0, 0.0, 0.0, 0.0, 0.0};  // adds 0 to its class
        }
      }
      large = __syncthreads_or(large);
      auto add = [&](int s, double* fc, auto phase) {
        const KTabD t = s_tab[s];
        double sn, cs;
        phase(t.kx * xo + t.ky * yo + t.kz * zo, &sn, &cs);
        const double g = cs * t.b - sn * t.a;
        fc[0] += g * t.kx;
        fc[1] += g * t.ky;
        fc[2] += g * t.kz;
      };
      auto classes = [&](auto step, auto phase) {
        constexpr int STEP = decltype(step)::value;
#pragma unroll 2
        for (int s = first; s < kpad; s += K_CLASSES)
#pragma unroll
          for (int c = 0; c < K_CLASSES / STEP; ++c) add(s + STEP * c, f[c], phase);
      };
      auto all = [&](auto phase) {
        if (share <= 2)
          classes(std::integral_constant<int, 2>(), phase);
        else if (share == 4)
          classes(std::integral_constant<int, 4>(), phase);
        else
          classes(std::integral_constant<int, 8>(), phase);
      };
      if (mine && !large)
        all([](double t, double* s, double* c) { sincos_phase(t, s, c); });
      else if (mine)
        all([](double t, double* s, double* c) { sincos(t, s, c); });
    }
    // the tree: classes c and c + 4, then c + 2, then c + 1, first those that a
    // thread holds, then those of its neighbours (a share never crosses a warp)
#pragma unroll
    for (int h = K_CLASSES / 4; h > 0; h >>= 1)
      if (share * h < K_CLASSES)
#pragma unroll
        for (int c = 0; c < h; ++c)
          for (int d = 0; d < 3; ++d) f[c][d] += f[c + h][d];
    fx += f[0][0];
    fy += f[0][1];
    fz += f[0][2];
  }
  for (int o = share >> 1; o > 0; o >>= 1) {
    fx += __shfl_xor_sync(0xffffffffu, fx, o);
    fy += __shfl_xor_sync(0xffffffffu, fy, o);
    fz += __shfl_xor_sync(0xffffffffu, fz, o);
  }
  __syncthreads();  // every position has been read
  if (mine && part == 0) {
    s_x[own] = fx;
    s_y[own] = fy;
    s_z[own] = fz;
  }
  __syncthreads();
  if (live)
    force_epilogue(ep, i, take ? s_x[threadIdx.x] * qi : 0.0, take ? s_y[threadIdx.x] * qi : 0.0,
                   take ? s_z[threadIdx.x] * qi : 0.0);
}

// Mixed-form force table entry (FP32 coefficients, integer m).
struct KTabF {
  int m0, m1, m2;
  float a, b, kx, ky, kz;
};

struct ForceMixedArgs {
  int n, p;
  const KTab* tab;
  const uint4* atoms;
  ForceEpilogue ep;
};

// Block bx of a grid of gx blocks.
template <int FB>
__device__ __forceinline__ void force_mixed_body(const ForceMixedArgs& A, int bx, int gx) {
  if (A.ep.job.kind != EnergyJob::NONE && bx == gx - 1) {
    if (threadIdx.x < 32) energy_job(A.ep.job);
    return;
  }
  const int n = A.n, p = A.p;
  const KTab* __restrict__ tab = A.tab;
  const uint4* __restrict__ atoms = A.atoms;
  const ForceEpilogue& ep = A.ep;
  __shared__ KTabF s_tab[FRC_TABLE];
  __shared__ uint4 s_atom[FB];          // records of the charged atoms
  __shared__ float s_f[3][FB];
  __shared__ unsigned short s_list[FB];
  __shared__ int s_cnt[FB / 32];
  const int i = bx * FB + threadIdx.x;
  const bool live = i < n;
  const uint4 ai = live ? atoms[i] : make_uint4(0, 0, 0, 0);
  const bool take = __uint_as_float(ai.w) != 0.f;
  if (take) s_atom[threadIdx.x] = ai;
  const int count = block_compact<FB>(take, s_list, s_cnt);
  const bool mine = (int)threadIdx.x < count;
  const int own = mine ? s_list[threadIdx.x] : 0;
  const uint4 a = mine ? s_atom[own] : make_uint4(0, 0, 0, 0);
  const float ang = (float)(2.0 * RBX_PI / 4294967296.0);
  float fx = 0.f, fy = 0.f, fz = 0.f;
  for (int k0 = 0; k0 < p && count > 0; k0 += FRC_TABLE) {
    const int kn = min(FRC_TABLE, p - k0);
    __syncthreads();
    for (int s = threadIdx.x; s < kn; s += FB) {
      const KTab& t = tab[k0 + s];
      KTabF f;
      f.m0 = t.m[0];
      f.m1 = t.m[1];
      f.m2 = t.m[2];
      f.a = (float)t.a;
      f.b = (float)t.b;
      f.kx = (float)t.kx;
      f.ky = (float)t.ky;
      f.kz = (float)t.kz;
      s_tab[s] = f;
    }
    __syncthreads();
    if (mine) {
#pragma unroll 4
      for (int s = 0; s < kn; ++s) {
        const KTabF t = s_tab[s];
        const unsigned ph = (unsigned)t.m0 * a.x + (unsigned)t.m1 * a.y + (unsigned)t.m2 * a.z;
        float sn, cs;
        __sincosf((float)(int)ph * ang, &sn, &cs);
        const float f = cs * t.b - sn * t.a;
        fx = fmaf(f, t.kx, fx);
        fy = fmaf(f, t.ky, fy);
        fz = fmaf(f, t.kz, fz);
      }
    }
  }
  if (mine) {
    s_f[0][own] = fx;
    s_f[1][own] = fy;
    s_f[2][own] = fz;
  }
  __syncthreads();
  if (live) {
    const double qi = (double)__uint_as_float(ai.w);
    force_epilogue(ep, i, take ? (double)s_f[0][threadIdx.x] * qi : 0.0,
                   take ? (double)s_f[1][threadIdx.x] * qi : 0.0,
                   take ? (double)s_f[2][threadIdx.x] * qi : 0.0);
  }
}

template <int FB>
__global__ void __launch_bounds__(FB) k_rbe_force_mixed(ForceMixedArgs a) {
  force_mixed_body<FB>(a, blockIdx.x, gridDim.x);
}

template <int FB>
__global__ void __launch_bounds__(FB)
k_rbe_force_mixed_batch(const ForceMixedArgs* __restrict__ a, const int* __restrict__ start,
                        int nrep) {
  const int r = batch_replica(start, nrep, blockIdx.x);
  const int b0 = __ldg(start + r);
  force_mixed_body<FB>(a[r], blockIdx.x - b0, __ldg(start + r + 1) - b0);
}

// ---------------------------------------------------------------------------
// Philox k-sampler: one thread per sample; per-axis inverse-CDF tables built
// on the host (order m = 0, +1, -1, +2, -2, ...).
// ---------------------------------------------------------------------------
// cdf[t] = w[0] + ... + w[t], accumulated left to right on the host exactly as
// the oracle's linear scan accumulates, so the first t with target < cdf[t]
// (binary search) is the oracle's pick.

constexpr int kSampleSmemTables = 6144;  // staged table entries (48 KB)
constexpr int SAMPLE_BLOCK = 128;

__global__ void __launch_bounds__(SAMPLE_BLOCK)
k_rbe_sample(int p, const double* __restrict__ tables, int c0, int c1, int c2, double t0,
             double t1, double t2, uint32_t key0, uint32_t key1, uint64_t step_arg,
             const int* __restrict__ step_dev, double* __restrict__ mx, double* __restrict__ my,
             double* __restrict__ mz, int* __restrict__ mi, int* __restrict__ status) {
  // the three cumulative tables are staged in shared memory when they fit
  // (dynamic size (c0 + c1 + c2) doubles), so the binary searches run there
  extern __shared__ double s_tab[];
  const int tot = c0 + c1 + c2;
  const bool staged = tot <= kSampleSmemTables;
  if (staged) {
    for (int t = threadIdx.x; t < tot; t += blockDim.x) s_tab[t] = tables[t];
    __syncthreads();
  }
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= p) return;
  // the MD step: a device copy inside a step graph
  const uint64_t step = step_dev ? (uint64_t)(int64_t)*step_dev : step_arg;
  SampleArgs sa{};
  sa.c0 = c0;
  sa.c1 = c1;
  sa.c2 = c2;
  sa.t0 = t0;
  sa.t1 = t1;
  sa.t2 = t2;
  sa.key0 = key0;
  sa.key1 = key1;
  int m[3];
  if (!rbe_draw(s, sa, staged ? s_tab : tables, step, m)) {
    atomicOr(status, 1);
    return;
  }
  if (mx) {
    mx[s] = m[0];
    my[s] = m[1];
    mz[s] = m[2];
  }
  if (mi) {
    mi[3 * s] = m[0];
    mi[3 * s + 1] = m[1];
    mi[3 * s + 2] = m[2];
  }
}

// Integer copy of injected samples (for the mixed kernels).
__global__ void k_m_to_int(int p, const double* __restrict__ mx, const double* __restrict__ my,
                           const double* __restrict__ mz, int* __restrict__ mi) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= p) return;
  mi[3 * s] = (int)mx[s];
  mi[3 * s + 1] = (int)my[s];
  mi[3 * s + 2] = (int)mz[s];
}

// ---------------------------------------------------------------------------
// Exact Ewald over the kmax box (oracle support / statistical reference).
// ---------------------------------------------------------------------------
// A warp owns EW_KPT k-vectors, a block EW_BLOCK / 32 warps: the block streams
// the atoms once for its 32 k-vectors, keeping the charged ones of each
// tile in shared memory, and lanes take atoms.  (One block a k-vector reads every
// atom nk times and is bound by L2.)  Where the k-vectors make fewer blocks than
// fit the chip, the atoms are split over blockIdx.y as well: without that, 26
// vectors are one block's work, and 200,000 atoms took it 3.4 ms.
// Measured, B200, rho, force and energy (with the charges' copy to the host, some
// 75 us) of 20,000 all-charged atoms, kmax 1 / 2 / 4 / 8: 115 / 129 / 237 / 939 us;
// a block a k-vector 144 / 182 / 479 / 2,600, without the split 390 / 404 / 484 / 1,190.
// Part blockIdx.y writes its sums to re, im[blockIdx.y][nk]; with one part they
// are rho(k), and the k-vectors and the table are written too.
constexpr int EW_BLOCK = 256;
constexpr int EW_KPT = 4;
constexpr int EW_PER_BLOCK = EW_BLOCK / 32 * EW_KPT;

struct EwaldBox {
  int nk, kmax[3];
  double L[3], alpha, coef;
  // k index -> (i, j, l) in ExecuteOnKmax order, skipping the origin
  __device__ __forceinline__ void vector(int k, int m[3], double kv[3]) const {
    const int ny = 2 * kmax[1] + 1, nz = 2 * kmax[2] + 1;
    const int center = kmax[0] * ny * nz + kmax[1] * nz + kmax[2];
    const int flat = k < center ? k : k + 1;
    m[0] = flat / (ny * nz) - kmax[0];
    m[1] = (flat / nz) % ny - kmax[1];
    m[2] = flat % nz - kmax[2];
    for (int d = 0; d < 3; ++d) kv[d] = 2 * RBX_PI * m[d] / L[d];
  }
  // k-vector k and, with tab, the force table entry of coef exp(-k^2 / 4 alpha) / k^2
  __device__ __forceinline__ void entry(int k, double re, double im, double* __restrict__ kvec,
                                        KTab* __restrict__ tab) const {
    int m[3];
    double kv[3];
    vector(k, m, kv);
    for (int d = 0; d < 3; ++d) kvec[3 * k + d] = kv[d];
    if (!tab) return;
    const double k2 = kv[0] * kv[0] + kv[1] * kv[1] + kv[2] * kv[2];
    const double f = coef / k2 * exp(-0.25 * k2 / alpha);
    KTab e;
    e.kx = kv[0];
    e.ky = kv[1];
    e.kz = kv[2];
    e.a = f * re;
    e.b = f * im;
    for (int d = 0; d < 3; ++d) e.m[d] = m[d];
    e.m[3] = 0;
    tab[k] = e;
  }
};

int ewald_parts(int n, int nk) {
  const int blocks = (nk + EW_PER_BLOCK - 1) / EW_PER_BLOCK, tiles = (n + EW_BLOCK - 1) / EW_BLOCK;
  const int fit = 2 * sm_count();  // resident blocks
  const int parts = blocks > 0 ? (fit + blocks - 1) / blocks : 1;
  return parts < tiles ? parts : (tiles > 0 ? tiles : 1);
}

__global__ void __launch_bounds__(EW_BLOCK)
k_ewald_rho(int n, EwaldBox E, const double* __restrict__ q, const double* __restrict__ x,
            const double* __restrict__ y, const double* __restrict__ z, double* __restrict__ re,
            double* __restrict__ im, double* __restrict__ kvec, KTab* __restrict__ tab) {
  __shared__ double s_x[EW_BLOCK], s_y[EW_BLOCK], s_z[EW_BLOCK], s_q[EW_BLOCK];
  __shared__ unsigned short s_list[EW_BLOCK];
  __shared__ int s_cnt[EW_BLOCK / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k0 = blockIdx.x * EW_PER_BLOCK + warp * EW_KPT;
  double kx[EW_KPT], ky[EW_KPT], kz[EW_KPT], sr[EW_KPT], si[EW_KPT], kmax = 0.0;
#pragma unroll
  for (int t = 0; t < EW_KPT; ++t) {
    int m[3];
    double kv[3];
    E.vector(min(k0 + t, E.nk - 1), m, kv);
    kx[t] = kv[0];
    ky[t] = kv[1];
    kz[t] = kv[2];
    sr[t] = si[t] = 0.0;
    kmax = fmax(kmax, norm1(kx[t], ky[t], kz[t]));
  }
  const int tiles = (n + EW_BLOCK - 1) / EW_BLOCK;
  for (int tile = blockIdx.y; tile < tiles; tile += gridDim.y) {
    const int j = tile * EW_BLOCK + threadIdx.x;
    const bool live = j < n;
    const double xj = live ? x[j] : 0.0, yj = live ? y[j] : 0.0, zj = live ? z[j] : 0.0;
    const double qj = live ? q[j] : 0.0;
    const bool take = live && kspace_atom(qj, xj, yj, zj);
    __syncthreads();  // the previous tile has been read
    if (take) {
      s_x[threadIdx.x] = xj;
      s_y[threadIdx.x] = yj;
      s_z[threadIdx.x] = zj;
      s_q[threadIdx.x] = qj;
    }
    const int count = block_compact<EW_BLOCK>(take, s_list, s_cnt);
    for (int a = lane; a < count; a += 32) {
      const int o = s_list[a];
      const double xo = s_x[o], yo = s_y[o], zo = s_z[o], c = s_q[o];
      auto add = [&](auto phase) {
#pragma unroll
        for (int t = 0; t < EW_KPT; ++t) {
          double sn, cs;
          phase(kx[t] * xo + ky[t] * yo + kz[t] * zo, &sn, &cs);
          sr[t] += c * cs;
          si[t] += c * sn;
        }
      };
      if (norm1(xo, yo, zo) * kmax <= PHASE_MAX)
        add([](double t, double* s, double* c) { sincos_phase(t, s, c); });
      else
        add([](double t, double* s, double* c) { sincos(t, s, c); });
    }
  }
#pragma unroll
  for (int t = 0; t < EW_KPT; ++t) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sr[t] += __shfl_xor_sync(0xffffffffu, sr[t], o);
      si[t] += __shfl_xor_sync(0xffffffffu, si[t], o);
    }
    const int k = k0 + t;
    if (lane == 0 && k < E.nk) {
      re[(size_t)blockIdx.y * E.nk + k] = sr[t];
      im[(size_t)blockIdx.y * E.nk + k] = si[t];
      if (gridDim.y == 1) E.entry(k, sr[t], si[t], kvec, tab);
    }
  }
}

// rho(k) = the sum over the parts, left in part 0.
__global__ void __launch_bounds__(128)
k_ewald_parts(int parts, EwaldBox E, double* __restrict__ re, double* __restrict__ im,
              double* __restrict__ kvec, KTab* __restrict__ tab) {
  const int k = blockIdx.x * 128 + threadIdx.x;
  if (k >= E.nk) return;
  double r = 0.0, i = 0.0;
#pragma unroll 8
  for (int b = 0; b < parts; ++b) {
    r += re[(size_t)b * E.nk + k];
    i += im[(size_t)b * E.nk + k];
  }
  re[k] = r;
  im[k] = i;
  E.entry(k, r, i, kvec, tab);
}

__global__ void k_ewald_energy(int nk, double V, double alpha, double qqr2e, double qsq,
                               const double* __restrict__ kvec, const double* __restrict__ re,
                               const double* __restrict__ im, double* __restrict__ energy) {
  __shared__ double sh[FIN_BLOCK / 32];
  double e = 0;
  for (int k = threadIdx.x; k < nk; k += FIN_BLOCK) {
    const double kx = kvec[3 * k], ky = kvec[3 * k + 1], kz = kvec[3 * k + 2];
    const double k2 = kx * kx + ky * ky + kz * kz;
    e += exp(-0.25 * k2 / alpha) / k2 * (re[k] * re[k] + im[k] * im[k]);
  }
  e = block_sum_det<FIN_BLOCK>(e, sh);
  if (threadIdx.x == 0) *energy = qqr2e * (2 * RBX_PI / V) * e + qqr2e * (-sqrt(alpha / RBX_PI) * qsq);
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
int rbe_partial_blocks(int n) {
  // about four waves of 256-thread blocks on the 148 SMs, at least 64 atoms each
  const int target = sm_count() * 4;
  int blocks = (n + 63) / 64;
  if (blocks > target) blocks = target;
  return blocks < 1 ? 1 : blocks;
}

// kpt: k-vectors per thread (1, 2, 4 or 8; 32 kpt per block); the partial
// sums do not depend on it.
int launch_rbe_rho_partial_f64(const DBox& b, int n, int p, const double* mx, const double* my,
                               const double* mz, const double* q, const double* x,
                               const double* y, const double* z, double* part_re,
                               double* part_im, int nblocks, cudaStream_t st, int kpt,
                               const SampleArgs* sample) {
  if (n <= 0 || p <= 0) return RBX_OK;
  const int chunk = (n + nblocks - 1) / nblocks;
  dim3 grid(nblocks, (p + 32 * kpt - 1) / (32 * kpt));
  const SampleArgs sa = sample ? *sample : SampleArgs{};
#define RHO_F64(K)                                                                             \
  k_rbe_rho_partial_f64<K><<<grid, RBE_BLOCK, 0, st>>>(                                        \
      n, p, chunk, b.len[0], b.len[1], b.len[2], 1.0 / b.len[0], 1.0 / b.len[1],               \
      1.0 / b.len[2], mx, my, mz, q, x, y, z, part_re, part_im, sa)
  switch (kpt) {
    case 1: RHO_F64(1); break;
    case 2: RHO_F64(2); break;
    case 8: RHO_F64(8); break;
    default: RHO_F64(4); break;
  }
#undef RHO_F64
  count_launch();
  return check_launch("rbe_rho_partial_f64");
}

int launch_rbe_rho_partial_mixed(int n, int p, const int* mi, const uint4* atoms,
                                 double* part_re, double* part_im, int nblocks, cudaStream_t st,
                                 int kpt, const SampleArgs* sample) {
  if (n <= 0 || p <= 0) return RBX_OK;
  const int chunk = (n + nblocks - 1) / nblocks;
  dim3 grid(nblocks, (p + 32 * kpt - 1) / (32 * kpt));
  RhoMixedArgs a;
  a.n = n;
  a.p = p;
  a.chunk = chunk;
  a.mi = mi;
  a.atoms = atoms;
  a.part_re = part_re;
  a.part_im = part_im;
  a.sa = sample ? *sample : SampleArgs{};
  a.gx = nblocks;
  if (kpt != 1 && kpt != 2 && kpt != 8) kpt = 4;
  if (batch_recorder())
    return record_phase(PH_RHO, kpt, (int)(grid.x * grid.y), RBE_BLOCK, 0, &a, sizeof a);
#define RHO_MIX(K) k_rbe_rho_partial_mixed<K><<<grid, RBE_BLOCK, 0, st>>>(a)
  switch (kpt) {
    case 1: RHO_MIX(1); break;
    case 2: RHO_MIX(2); break;
    case 8: RHO_MIX(8); break;
    default: RHO_MIX(4); break;
  }
#undef RHO_MIX
  count_launch();
  return check_launch("rbe_rho_partial_mixed");
}

int launch_rbe_finalize(const DBox& b, int p, int nparts, const double* part_re,
                        const double* part_im, const double* mx, const double* my,
                        const double* mz, double alpha, double S, double qqr2e, double qsq,
                        double qsum, double* rho_re, double* rho_im, double* energy,
                        double* virial, KTab* tab, int mean_parts, const double* fpart,
                        int n_atoms, double* mean_out, double* kterm, cudaStream_t st,
                        EnergyJob* job) {
  if (energy && !kterm) {  // no per-k scratch: rho is given (one partial a k)
    if (nparts != 1 || tab || mean_out || rho_re) {
      set_error("rbe_finalize: energies without per-k scratch need finished structure factors");
      return RBX_ERR_INVALID;
    }
    k_rbe_energy_virial<<<1, FIN_BLOCK, 0, st>>>(p, part_re, part_im, mx, my, mz, b.len[0],
                                                 b.len[1], b.len[2], alpha, S, qqr2e, qsq, qsum,
                                                 energy, virial);
    count_launch();
    return check_launch("rbe_energy_virial");
  }
  const int grid = p + (mean_out ? 3 : 0);
  EnergyJob sum;
  if (energy) {
    sum.kind = EnergyJob::RBE;
    sum.p = p;
    sum.kterm = kterm;
    sum.alpha = alpha;
    sum.V = b.len[0] * b.len[1] * b.len[2];
    sum.qqr2e = qqr2e;
    sum.qsq = qsq;
    sum.qsum = qsum;
    sum.energy = energy;
    sum.virial = virial;
  }
  if (job) *job = sum;
  if (grid > 0) {
    FinalizeArgs a;
    a.p = p;
    a.nparts = nparts;
    a.part_re = part_re;
    a.part_im = part_im;
    a.mx = mx;
    a.my = my;
    a.mz = mz;
    a.Lx = b.len[0];
    a.Ly = b.len[1];
    a.Lz = b.len[2];
    a.alpha = alpha;
    a.S = S;
    a.qqr2e = qqr2e;
    a.rho_re = rho_re;
    a.rho_im = rho_im;
    a.tab = tab;
    a.kterm = energy ? kterm : nullptr;
    a.mean_parts = mean_parts;
    a.fpart = fpart;
    a.n_atoms = (double)n_atoms;
    a.mean_out = mean_out;
    if (batch_recorder()) {
      if (energy && !job) {
        set_error("rbe_finalize: a batched finalize leaves the energy sum to the force pass");
        return RBX_ERR_INVALID;
      }
      return record_phase(PH_FINALIZE, 0, grid, FK_BLOCK, 0, &a, sizeof a);
    }
    k_rbe_finalize_k<<<grid, FK_BLOCK, 0, st>>>(a);
    count_launch();
    const int rc = check_launch("rbe_finalize_k");
    if (rc) return rc;
  }
  return energy && !job ? launch_energy_sum(sum, st) : RBX_OK;
}

static ForceEpilogue make_ep(const RbeForceOut& o) {
  ForceEpilogue ep;
  ep.f_pair_x = o.f_pair_x;
  ep.f_pair_y = o.f_pair_y;
  ep.f_pair_z = o.f_pair_z;
  ep.mean = o.mean;
  ep.f_out_x = o.f_out_x;
  ep.f_out_y = o.f_out_y;
  ep.f_out_z = o.f_out_z;
  ep.fk_x = o.fk_x;
  ep.fk_y = o.fk_y;
  ep.fk_z = o.fk_z;
  ep.vx = o.vx;
  ep.vy = o.vy;
  ep.vz = o.vz;
  ep.type = o.type;
  ep.inv_mass = o.inv_mass;
  ep.half_dt = o.half_dt;
  ep.job = o.job;
  return ep;
}

// block: atoms per block (128, 256 or 512); the forces do not depend on it.
int launch_rbe_force_f64(int n, int p, const KTab* tab, const double* q, const double* x,
                         const double* y, const double* z, const RbeForceOut& out,
                         cudaStream_t st, int block) {
  const int extra = out.job.kind != EnergyJob::NONE;  // the energy's block
  if (n <= 0) return extra ? launch_energy_sum(out.job, st) : RBX_OK;
  const ForceEpilogue ep = make_ep(out);
  if (block != 128 && block != 512) block = 256;
  const auto kern = block == 128 ? k_rbe_force_f64<128>
                                 : (block == 512 ? k_rbe_force_f64<512> : k_rbe_force_f64<256>);
  kern<<<(n + block - 1) / block + extra, block, 0, st>>>(n, p, tab, q, x, y, z, ep);
  count_launch();
  return check_launch("rbe_force_f64");
}

int launch_rbe_force_mixed(int n, int p, const KTab* tab, const uint4* atoms,
                           const RbeForceOut& out, cudaStream_t st, int block) {
  const int extra = out.job.kind != EnergyJob::NONE;  // the energy's block
  if (n <= 0) return extra ? launch_energy_sum(out.job, st) : RBX_OK;
  ForceMixedArgs a;
  a.n = n;
  a.p = p;
  a.tab = tab;
  a.atoms = atoms;
  a.ep = make_ep(out);
  if (block != 128 && block != 512) block = 256;
  const int grid = (n + block - 1) / block + extra;
  if (batch_recorder()) return record_phase(PH_FORCE, block, grid, block, 0, &a, sizeof a);
  const auto kern = block == 128 ? k_rbe_force_mixed<128>
                                 : (block == 512 ? k_rbe_force_mixed<512> : k_rbe_force_mixed<256>);
  kern<<<grid, block, 0, st>>>(a);
  count_launch();
  return check_launch("rbe_force_mixed");
}

int launch_rho_mixed_batch(int variant, const void* args, const int* start, int nrep, int total,
                           cudaStream_t st) {
  const RhoMixedArgs* a = static_cast<const RhoMixedArgs*>(args);
  switch (variant) {
    case 1: k_rbe_rho_partial_mixed_batch<1><<<total, RBE_BLOCK, 0, st>>>(a, start, nrep); break;
    case 2: k_rbe_rho_partial_mixed_batch<2><<<total, RBE_BLOCK, 0, st>>>(a, start, nrep); break;
    case 8: k_rbe_rho_partial_mixed_batch<8><<<total, RBE_BLOCK, 0, st>>>(a, start, nrep); break;
    default: k_rbe_rho_partial_mixed_batch<4><<<total, RBE_BLOCK, 0, st>>>(a, start, nrep); break;
  }
  count_launch();
  return check_launch("rbe_rho_partial_mixed_batch");
}

int launch_finalize_batch(const void* args, const int* start, int nrep, int total,
                          cudaStream_t st) {
  k_rbe_finalize_k_batch<<<total, FK_BLOCK, 0, st>>>(static_cast<const FinalizeArgs*>(args),
                                                     start, nrep);
  count_launch();
  return check_launch("rbe_finalize_k_batch");
}

int launch_force_mixed_batch(int variant, const void* args, const int* start, int nrep,
                             int total, cudaStream_t st) {
  const ForceMixedArgs* a = static_cast<const ForceMixedArgs*>(args);
  if (variant == 128)
    k_rbe_force_mixed_batch<128><<<total, 128, 0, st>>>(a, start, nrep);
  else if (variant == 512)
    k_rbe_force_mixed_batch<512><<<total, 512, 0, st>>>(a, start, nrep);
  else
    k_rbe_force_mixed_batch<256><<<total, 256, 0, st>>>(a, start, nrep);
  count_launch();
  return check_launch("rbe_force_mixed_batch");
}

int launch_rbe_sample(int p, const double* tables, const int cnt[3], const double tot[3],
                      uint64_t seed, int64_t step, const int* step_dev, double* mx, double* my,
                      double* mz, int* mi, int* status, cudaStream_t st) {
  if (p <= 0) return RBX_OK;
  const int entries = cnt[0] + cnt[1] + cnt[2];
  const size_t smem = entries <= kSampleSmemTables ? sizeof(double) * entries : 0;
  k_rbe_sample<<<(p + SAMPLE_BLOCK - 1) / SAMPLE_BLOCK, SAMPLE_BLOCK, smem, st>>>(
      p, tables, cnt[0], cnt[1], cnt[2], tot[0], tot[1], tot[2], (uint32_t)seed,
      (uint32_t)(seed >> 32), (uint64_t)step, step_dev, mx, my, mz, mi, status);
  count_launch();
  return check_launch("rbe_sample");
}

SampleArgs make_sample_args(const double* tables, const int cnt[3], const double tot[3],
                            uint64_t seed, int64_t step, const int* step_dev, double* mx,
                            double* my, double* mz, int* mi, int* status) {
  SampleArgs sa{};
  sa.tables = tables;
  sa.c0 = cnt[0];
  sa.c1 = cnt[1];
  sa.c2 = cnt[2];
  sa.t0 = tot[0];
  sa.t1 = tot[1];
  sa.t2 = tot[2];
  sa.key0 = (uint32_t)seed;
  sa.key1 = (uint32_t)(seed >> 32);
  sa.step_arg = (uint64_t)step;
  sa.step_dev = step_dev;
  sa.mx = mx;
  sa.my = my;
  sa.mz = mz;
  sa.mi = mi;
  sa.status = status;
  return sa;
}

int launch_m_to_int(int p, const double* mx, const double* my, const double* mz, int* mi,
                    cudaStream_t st) {
  if (p <= 0) return RBX_OK;
  k_m_to_int<<<(p + 127) / 128, 128, 0, st>>>(p, mx, my, mz, mi);
  count_launch();
  return check_launch("m_to_int");
}

int launch_ewald(const DBox& b, int n, const int kmax[3], double alpha, double qqr2e,
                 double qsq, const double* q, const double* x, const double* y, const double* z,
                 double* re, double* im, double* kvec, KTab* tab, double* fx, double* fy,
                 double* fz, double* energy, cudaStream_t st) {
  const int nk = (2 * kmax[0] + 1) * (2 * kmax[1] + 1) * (2 * kmax[2] + 1) - 1;
  if (nk <= 0) return RBX_OK;
  const double V = b.len[0] * b.len[1] * b.len[2];
  EwaldBox E;
  E.nk = nk;
  for (int d = 0; d < 3; ++d) {
    E.kmax[d] = kmax[d];
    E.L[d] = b.len[d];
  }
  E.alpha = alpha;
  E.coef = -4.0 * RBX_PI * qqr2e / V;
  const int parts = ewald_parts(n, nk);
  k_ewald_rho<<<dim3((nk + EW_PER_BLOCK - 1) / EW_PER_BLOCK, parts), EW_BLOCK, 0, st>>>(
      n, E, q, x, y, z, re, im, kvec, tab);
  count_launch();
  int rc = check_launch("ewald_rho");
  if (rc) return rc;
  if (parts > 1) {
    k_ewald_parts<<<(nk + 127) / 128, 128, 0, st>>>(parts, E, re, im, kvec, tab);
    count_launch();
    rc = check_launch("ewald_parts");
    if (rc) return rc;
  }
  if (n > 0 && tab) {
    RbeForceOut o;
    o.f_out_x = fx;
    o.f_out_y = fy;
    o.f_out_z = fz;
    rc = launch_rbe_force_f64(n, nk, tab, q, x, y, z, o, st, 256);
    if (rc) return rc;
  }
  if (energy) {
    k_ewald_energy<<<1, FIN_BLOCK, 0, st>>>(nk, V, alpha, qqr2e, qsq, kvec, re, im, energy);
    count_launch();
    rc = check_launch("ewald_energy");
  }
  return rc;
}

}  // namespace rbx
