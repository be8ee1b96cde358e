// rbx_adjoint.cu -- adjoint (vector-Jacobian product) of the RBL + RBE force
// for force-field fitting: plain FP64 for FP64 engines; FP32 pair terms and
// FP32 k-space terms on exact fixed-point phases with FP64 sums for engines
// in the mixed form.
//
// For an upstream g = dL/dF it gives dL/d(eps_t, sigma_t) per type, dL/dq_i,
// dL/dalpha and dL/dr_i (the Hessian-vector product), for the lists, batch
// selection and k-samples of the engine's last force evaluation.  Nothing is
// stored per pair: the pair terms and the k-space phases are recomputed.
//
// Force (ComputeLJCutCoulRBLForce, lj_cut_coul_kspace_op.hip.cu:569-683; mean
// removal lj_cut_coul_kspace.cpp:537-563; ComputeRBEForce,
// kspace_calculator_op.hip.cu:98-125, 678-738):
//   F_i = P_i - mean(P) + K_i,  P_i = sum_{j in L(i)} s_ij f(r^2) (r_j - r_i)
// With g' = g - mean(g), pair (i, j) adds s (df/dtheta)(g'_i . d) to the
// parameter gradient and c = s (f g'_i + 2 f'(g'_i . d) d) to dL/dr_j, -c to
// dL/dr_i.  The pair kernel runs a warp per atom m over its candidate row,
// which is symmetric, and tests both m in L(j) and j in L(m) (the same
// distance windows; the shell batch hash evaluated from either side), so each
// atom gathers its own gradient without atomics.  The k-space part uses
// a_k = sum_i q_i (g_i.k) cos(k.r_i), b_k = sum_i q_i (g_i.k) sin(k.r_i).
#include <math.h>

#include "rbx_common.cuh"
#include "rbx_kernels.h"
#include "rbx_pair_device.cuh"
#include "rbx_phase.cuh"

namespace rbx {

constexpr int ADJ_WARPS = 8;
constexpr int ADJ_BLOCK = 32 * ADJ_WARPS;
constexpr int ADJ_MAX_TYPES = 16;

// Pair terms of one (i, j) at squared distance r2 (windows already applied):
// f, f' = df/d(r^2), df/deps_ij, df/dsigma_ij, the Coulomb shape h (f_C = q q h)
// and dh/dalpha.
struct PairTerms {
  double f, fp, df_de, df_ds, h, dh_da;
};

__device__ __forceinline__ PairTerms pair_terms(double e, double sg, double qq, double r2,
                                                double alpha, double qqr2e) {
  PairTerms t;
  const double ui = 1.0 / r2;
  const double s6 = sg * sg * sg * sg * sg * sg;
  const double u = s6 * ui * ui * ui;  // sigma^6 / r^6
  t.df_de = -24.0 * (2.0 * u * u - u) * ui;  // f_lj / e, also where e = 0
  const double f_lj = e * t.df_de;
  const double ui2 = ui * ui, ui4 = ui2 * ui2;
  const double fp_lj = 24.0 * e * (14.0 * s6 * s6 * ui4 * ui4 - 4.0 * s6 * ui4 * ui);
  const double r = sqrt(r2);
  const double b = sqrt(alpha);
  const double ex = exp(-alpha * r2);
  const double ec = erfc(b * r);
  const double two_b_pi = 2.0 * b / 1.77245385090551602729;  // 2 b / sqrt(pi)
  t.h = -qqr2e * (ec * ui + two_b_pi * ex / r) / r;
  const double dh_dr = qqr2e * (3.0 * ec * ui2 + two_b_pi * ex * (3.0 * ui + 2.0 * alpha) / r);
  t.dh_da = qqr2e * two_b_pi * ex;
  t.f = f_lj + qq * t.h;
  t.fp = fp_lj + qq * dh_dr / (2.0 * r);
  t.df_ds = -144.0 * e * (4.0 * u * u - u) * ui / sg;
  return t;
}

// The same pair terms in FP32 (mixed form), returned widened to FP64 for the
// FP64 sums of the adjoint.
__device__ __forceinline__ PairTerms pair_terms_f32(float e, float sg, float qq, float r2,
                                                    float alpha, float qqr2e) {
  const float ui = 1.0f / r2;
  const float s2 = sg * sg, s6 = s2 * s2 * s2;
  const float u = s6 * ui * ui * ui;
  const float df_de = -24.0f * (2.0f * u * u - u) * ui;
  const float f_lj = e * df_de;
  const float ui2 = ui * ui, ui4 = ui2 * ui2;
  const float fp_lj = 24.0f * e * (14.0f * s6 * s6 * ui4 * ui4 - 4.0f * s6 * ui4 * ui);
  const float r = sqrtf(r2);
  const float b = sqrtf(alpha);
  const float ex = expf(-alpha * r2);
  const float ec = erfcf(b * r);
  const float two_b_pi = 2.0f * b / 1.77245385090551602729f;
  const float h = -qqr2e * (ec * ui + two_b_pi * ex / r) / r;
  const float dh_dr = qqr2e * (3.0f * ec * ui2 + two_b_pi * ex * (3.0f * ui + 2.0f * alpha) / r);
  PairTerms t;
  t.h = h;
  t.dh_da = qqr2e * two_b_pi * ex;
  t.f = f_lj + qq * h;
  t.fp = fp_lj + qq * dh_dr / (2.0f * r);
  t.df_de = df_de;
  t.df_ds = -144.0f * e * (4.0f * u * u - u) * ui / sg;
  return t;
}

// Block partials: [block][2 * ntypes + 1] = d_eps[0..nt), d_sigma[0..nt), d_alpha.
// F32: pair terms in FP32 (mixed form), sums in FP64 either way.
//
// A warp per atom.  Candidates are screened in batches (fixed-point |d|^2, the
// FP64 predicate inside its guard bands) and hashed from both sides; the 44 %
// that carry a gradient wait in a per-warp queue, so that the pair terms run on
// full warps.  The parameter sums of the partner's type live in shared memory,
// one column a lane (an array indexed by a run-time type is local memory: the
// kernel was bound by it and by idle lanes).  Four blocks an SM, some words
// spilled, beat two without: 20,000 atoms, 417 us before, 247 at two blocks, 185
// at four (FP64: 275).
constexpr int ADJ_U = 2;           // 32-candidate groups per batch
constexpr int AQ_M = (int)0x80000000;  // j is in m's list
constexpr int AQ_J = 0x40000000;       // m is in j's list
constexpr int AQ_CORE = 0x20000000;    // core pair: scale 1, not freq
constexpr int AQ_INDEX = 0x1fffffff;   // atom index (n < 2^29)

template <bool F32>
__global__ void __launch_bounds__(ADJ_BLOCK, 4)
k_adj_pair(PairParams pp, int n, const uint4* __restrict__ atoms, const double* __restrict__ x,
           const double* __restrict__ y, const double* __restrict__ z,
           const double* __restrict__ q, const int* __restrict__ type,
           const double* __restrict__ sigma_t, const double* __restrict__ eps_t,
           const unsigned long long* __restrict__ key_a,
           const unsigned long long* __restrict__ key_b, int epoch, Rows rows,
           const double* __restrict__ gx, const double* __restrict__ gy,
           const double* __restrict__ gz, double mgx, double mgy, double mgz,
           double* __restrict__ d_rx, double* __restrict__ d_ry, double* __restrict__ d_rz,
           double* __restrict__ d_q, double* __restrict__ part) {
  extern __shared__ double s_lane[];  // [2 * nt][ADJ_BLOCK]: d_eps, d_sigma sums of a lane
  __shared__ double s_part[ADJ_WARPS][2 * ADJ_MAX_TYPES + 1];
  __shared__ int s_q[ADJ_WARPS][32 + 32 * ADJ_U];
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int nt = pp.ntypes, npar = 2 * nt + 1;
  const unsigned lt = (1u << lane) - 1u;
  int* const wq = s_q[warp];
  double* const mine = s_lane + threadIdx.x;
  for (int t = 0; t < 2 * nt; ++t) mine[t * ADJ_BLOCK] = 0.0;
  double d_alpha = 0.0;
  const double freq = (double)pp.freq;
  for (int m = blockIdx.x * ADJ_WARPS + warp; m < n; m += gridDim.x * ADJ_WARPS) {
    const uint4 am = atoms[m];
    const double xm = x[m], ym = y[m], zm = z[m], qm = q[m];
    const int tm = type[m];
    const double eps_m = eps_t[tm], sig_m = sigma_t[tm];
    const double gpx = gx[m] - mgx, gpy = gy[m] - mgy, gpz = gz[m] - mgz;
    const unsigned long long ea_m = key_a[m] ^ (unsigned long long)(long long)epoch;
    const unsigned long long kb_m = key_b[m];
    double rx = 0.0, ry = 0.0, rz = 0.0, dq = 0.0, de_m = 0.0, ds_m = 0.0;
    int nf, nb;
    row_extent(rows, m, nf, nb);
    const int cnt = nf + nb;
    const int* row = rows.idx + (size_t)m * rows.cap;
    int qn = 0;
    auto pair = [&](int slot) {
      const int c = wq[slot];
      const int j = c & AQ_INDEX;
      const bool in_m = c < 0, in_j = c & AQ_J;
      const double s = (c & AQ_CORE) ? 1.0 : freq;
      // r_j - r_m, MinImageDistance (box.h:51-73), as in the force kernel
      const double dx = min_image1(x[j] - xm, pp.box.len[0], pp.box.half[0]);
      const double dy = min_image1(y[j] - ym, pp.box.len[1], pp.box.half[1]);
      const double dz = min_image1(z[j] - zm, pp.box.len[2], pp.box.half[2]);
      const double r2 = dx * dx + dy * dy + dz * dz;
      const int tj = type[j];
      const double eps_j = eps_t[tj];
      const double e = sqrt(eps_m * eps_j);
      const double sg = 0.5 * (sig_m + sigma_t[tj]);
      const double qj = q[j];
      const PairTerms pt =
          F32 ? pair_terms_f32((float)e, (float)sg, (float)(qm * qj), (float)r2, (float)pp.alpha,
                               (float)pp.qqr2e)
              : pair_terms(e, sg, qm * qj, r2, pp.alpha, pp.qqr2e);
      if (in_m) {  // pair (m, j) of m's force: parameters and -c on r_m
        const double gd = gpx * dx + gpy * dy + gpz * dz;
        const double w = s * gd;
        const double cf = s * pt.f, cd = 2.0 * s * pt.fp * gd;
        rx -= cf * gpx + cd * dx;
        ry -= cf * gpy + cd * dy;
        rz -= cf * gpz + cd * dz;
        dq += w * pt.h * qj;
        const double we = w * pt.df_de * e, ws = 0.5 * w * pt.df_ds;
        // sqrt(eps_m eps_j) has no derivative in an eps that is 0
        de_m += eps_m > 0.0 ? we : NAN;
        ds_m += ws;
        mine[tj * ADJ_BLOCK] += eps_j > 0.0 ? we : NAN;
        mine[(nt + tj) * ADJ_BLOCK] += ws;
        d_alpha += w * qm * qj * pt.dh_da;
      }
      if (in_j) {  // pair (j, m) of j's force: +c on r_m, and its q_m factor
        const double gjx = gx[j] - mgx, gjy = gy[j] - mgy, gjz = gz[j] - mgz;
        const double gd = gjx * dx + gjy * dy + gjz * dz;  // d = r_j - r_m: g'_j . (-(r_m - r_j))
        const double cf = s * pt.f, cd = 2.0 * s * pt.fp * gd;
        rx += cf * gjx + cd * dx;
        ry += cf * gjy + cd * dy;
        rz += cf * gjz + cd * dz;
        dq -= s * gd * pt.h * qj;  // w_j = s g'_j . (r_m - r_j) = -s gd
      }
    };
    for (int k0 = 0; k0 < cnt; k0 += 32 * ADJ_U) {
      int j[ADJ_U];
      uint4 aj[ADJ_U];
#pragma unroll
      for (int u = 0; u < ADJ_U; ++u) {
        const int k = k0 + 32 * u + lane;
        j[u] = k < cnt ? row_at(row, rows.cap, nf, nb, k) : m;
      }
#pragma unroll
      for (int u = 0; u < ADJ_U; ++u) aj[u] = __ldg(atoms + j[u]);
#pragma unroll
      for (int u = 0; u < ADJ_U; ++u) {
        bool unsure;
        Classified c = classify_screen(pp, pp.cubic ? fixed_d2(am, aj[u])
                                                    : fixed_d2_weighted(pp, am, aj[u]), &unsure);
        if (unsure && j[u] != m) c = classify_exact(exact_d2(pp, x, y, z, m, j[u]), pp);
        int f = c.core_active ? AQ_M | AQ_J | AQ_CORE : 0;
        if (c.shell_window) {
          if (rbl_selected(ea_m, __ldg(key_b + j[u]), pp.div)) f |= AQ_M;
          if (rbl_selected(__ldg(key_a + j[u]) ^ (unsigned long long)(long long)epoch, kb_m,
                           pp.div))
            f |= AQ_J;
        }
        const bool push = f != 0 && j[u] != m;
        const unsigned mk = __ballot_sync(0xffffffffu, push);
        if (push) wq[qn + __popc(mk & lt)] = j[u] | f;
        qn += __popc(mk);
      }
      __syncwarp();
      while (qn >= 32) {  // full batches from the tail of the queue
        qn -= 32;
        pair(qn + lane);
      }
      __syncwarp();
    }
    if (lane < qn) pair(lane);
    __syncwarp();
    // d(eps_ij)/d(eps_m) = e / (2 eps_m); the partner's side below
    mine[tm * ADJ_BLOCK] += de_m;
    mine[(nt + tm) * ADJ_BLOCK] += ds_m;
    rx = warp_sum(rx);
    ry = warp_sum(ry);
    rz = warp_sum(rz);
    dq = warp_sum(dq);
    if (lane == 0) {
      d_rx[m] = rx;
      d_ry[m] = ry;
      d_rz[m] = rz;
      d_q[m] = dq;
    }
  }
  for (int t = 0; t < npar; ++t) {
    double v = warp_sum(t < 2 * nt ? mine[t * ADJ_BLOCK] : d_alpha);
    // a type without force-carrying pairs sums to 0, also with eps = 0; with
    // eps = 0 and pairs the sum is NaN
    if (t < nt && v != 0.0) v /= 2.0 * eps_t[t];
    if (lane == 0) s_part[warp][t] = v;
  }
  __syncthreads();
  if (threadIdx.x < npar) {
    double v = 0.0;
    for (int w = 0; w < ADJ_WARPS; ++w) v += s_part[w][threadIdx.x];
    part[(size_t)blockIdx.x * npar + threadIdx.x] = v;
  }
}

// k-space, pass 1: per-block partial sums of a_k and b_k, part[k][block].
constexpr int ADJK_BLOCK = 128;
__global__ void __launch_bounds__(ADJK_BLOCK)
k_adj_k_ab(int n, int p, int chunk, const KTab* __restrict__ tab, const double* __restrict__ q,
           const double* __restrict__ x, const double* __restrict__ y,
           const double* __restrict__ z, const double* __restrict__ gx,
           const double* __restrict__ gy, const double* __restrict__ gz,
           double* __restrict__ part_a, double* __restrict__ part_b) {
  const int k = blockIdx.y * ADJK_BLOCK + threadIdx.x;
  if (k >= p) return;
  const double kx = tab[k].kx, ky = tab[k].ky, kz = tab[k].kz;
  const int a0 = blockIdx.x * chunk, a1 = min(n, a0 + chunk);
  double sa = 0.0, sb = 0.0;
  for (int i = a0; i < a1; ++i) {
    double s, c;
    if (q[i] + 0.0 * (x[i] + y[i] + z[i] + gx[i] + gy[i] + gz[i]) == 0.0)
      continue;  // a neutral atom's weight q_i (g_i . k) is zero
    sincos_phase_any(kx * x[i] + ky * y[i] + kz * z[i], &s, &c);
    const double w = q[i] * (gx[i] * kx + gy[i] * ky + gz[i] * kz);
    sa += w * c;
    sb += w * s;
  }
  part_a[(size_t)k * gridDim.x + blockIdx.x] = sa;
  part_b[(size_t)k * gridDim.x + blockIdx.x] = sb;
}

// k-space, pass 2: per-atom dL/dq and dL/dr, and per-block sums of g . K
// (for dL/dalpha).  ab[k] = {a_k, b_k} reduced in fixed order beforehand.
__global__ void __launch_bounds__(ADJK_BLOCK)
k_adj_k_scatter(int n, int p, double cscale, const KTab* __restrict__ tab,
                const double* __restrict__ ab, const double* __restrict__ q,
                const double* __restrict__ x, const double* __restrict__ y,
                const double* __restrict__ z, const double* __restrict__ gx,
                const double* __restrict__ gy, const double* __restrict__ gz,
                double* __restrict__ d_rx, double* __restrict__ d_ry, double* __restrict__ d_rz,
                double* __restrict__ d_q, double* __restrict__ part_gk) {
  struct K64 {  // per-k constants, formed once a block
    double kx, ky, kz, ta, tb, ca, cb;
  };
  constexpr int kTile = 128;
  __shared__ K64 s_k[kTile];
  __shared__ double s_sum[ADJK_BLOCK / 32];
  const int i = blockIdx.x * ADJK_BLOCK + threadIdx.x;
  const bool live = i < n;
  const double xi = live ? x[i] : 0.0, yi = live ? y[i] : 0.0, zi = live ? z[i] : 0.0,
               qi = live ? q[i] : 0.0;
  const double gix = live ? gx[i] : 0.0, giy = live ? gy[i] : 0.0, giz = live ? gz[i] : 0.0;
  double rx = 0.0, ry = 0.0, rz = 0.0, dq = 0.0, gk_sum = 0.0;
  for (int k0 = 0; k0 < p; k0 += kTile) {
    const int kn = min(kTile, p - k0);
    __syncthreads();
    for (int k = threadIdx.x; k < kn; k += ADJK_BLOCK) {
      const KTab& t = tab[k0 + k];
      const double ck = cscale / (t.kx * t.kx + t.ky * t.ky + t.kz * t.kz);
      // t.a = c_k Re rho_k, t.b = c_k Im rho_k, c_k = -4 pi qqr2e S / (P V k^2)
      s_k[k] = K64{t.kx, t.ky, t.kz, t.a, t.b,
                   ck * ab[2 * (k0 + k)], ck * ab[2 * (k0 + k) + 1]};
    }
    __syncthreads();
    for (int k = 0; k < kn; ++k) {
      const K64 t = s_k[k];
      double s, c;
      sincos_phase_any(t.kx * xi + t.ky * yi + t.kz * zi, &s, &c);
      const double gk = gix * t.kx + giy * t.ky + giz * t.kz;
      const double g1 = gk * (c * t.tb - s * t.ta);
      dq += g1 + (t.ca * s - t.cb * c);
      const double coef = -gk * (s * t.tb + c * t.ta) + (t.ca * c + t.cb * s);
      rx += coef * t.kx;
      ry += coef * t.ky;
      rz += coef * t.kz;
      gk_sum += g1;
    }
  }
  if (live) {
    d_rx[i] += qi * rx;
    d_ry[i] += qi * ry;
    d_rz[i] += qi * rz;
    d_q[i] += dq;
  }
  gk_sum = block_sum_det<ADJK_BLOCK>(live ? gk_sum * qi : 0.0, s_sum);
  if (threadIdx.x == 0) part_gk[blockIdx.x] = gk_sum;
}

// Mixed form of the k-space passes: the phase k.r_i = 2 pi (m . u_i) / 2^32 from
// the 32-bit fixed-point record u_i exactly in integer arithmetic, sin and
// cos on the SFU, every term in FP32 and every sum in FP64.
__global__ void __launch_bounds__(ADJK_BLOCK)
k_adj_k_ab_mixed(int n, int p, int chunk, const KTab* __restrict__ tab,
                 const uint4* __restrict__ atoms, const double* __restrict__ gx,
                 const double* __restrict__ gy, const double* __restrict__ gz,
                 double* __restrict__ part_a, double* __restrict__ part_b) {
  const int k = blockIdx.y * ADJK_BLOCK + threadIdx.x;
  if (k >= p) return;
  const KTab t = tab[k];
  const unsigned m0 = (unsigned)t.m[0], m1 = (unsigned)t.m[1], m2 = (unsigned)t.m[2];
  const float kx = (float)t.kx, ky = (float)t.ky, kz = (float)t.kz;
  const float ang = (float)(2.0 * RBX_PI / 4294967296.0);
  const int a0 = blockIdx.x * chunk, a1 = min(n, a0 + chunk);
  double sa = 0.0, sb = 0.0;
  for (int i = a0; i < a1; ++i) {
    const uint4 a = atoms[i];
    const unsigned ph = m0 * a.x + m1 * a.y + m2 * a.z;
    float sn, cs;
    __sincosf((float)(int)ph * ang, &sn, &cs);
    const float w = __uint_as_float(a.w) *
                    ((float)gx[i] * kx + (float)gy[i] * ky + (float)gz[i] * kz);
    sa += (double)(w * cs);
    sb += (double)(w * sn);
  }
  part_a[(size_t)k * gridDim.x + blockIdx.x] = sa;
  part_b[(size_t)k * gridDim.x + blockIdx.x] = sb;
}

__global__ void __launch_bounds__(ADJK_BLOCK)
k_adj_k_scatter_mixed(int n, int p, double cscale, const KTab* __restrict__ tab,
                      const double* __restrict__ ab, const uint4* __restrict__ atoms,
                      const double* __restrict__ gx, const double* __restrict__ gy,
                      const double* __restrict__ gz, double* __restrict__ d_rx,
                      double* __restrict__ d_ry, double* __restrict__ d_rz,
                      double* __restrict__ d_q, double* __restrict__ part_gk) {
  // the per-k constants in FP32, formed once a block (c_k took an FP64 divide
  // per atom and k)
  struct K32 {
    unsigned m0, m1, m2;
    float kx, ky, kz, ck, ta, tb, ak, bk;
  };
  constexpr int kTile = 256;
  __shared__ K32 s_k[kTile];
  __shared__ double s_sum[ADJK_BLOCK / 32];
  const int i = blockIdx.x * ADJK_BLOCK + threadIdx.x;
  double gk_sum = 0.0;
  const bool live = i < n;
  const uint4 a = live ? atoms[i] : make_uint4(0, 0, 0, 0);
  const float qi = __uint_as_float(a.w);
  const float gix = live ? (float)gx[i] : 0.f, giy = live ? (float)gy[i] : 0.f,
              giz = live ? (float)gz[i] : 0.f;
  const float ang = (float)(2.0 * RBX_PI / 4294967296.0);
  double rx = 0.0, ry = 0.0, rz = 0.0, dq = 0.0;
  for (int k0 = 0; k0 < p; k0 += kTile) {
    const int kn = min(kTile, p - k0);
    __syncthreads();
    for (int k = threadIdx.x; k < kn; k += ADJK_BLOCK) {
      const KTab& t = tab[k0 + k];
      K32 c;
      c.m0 = (unsigned)t.m[0];
      c.m1 = (unsigned)t.m[1];
      c.m2 = (unsigned)t.m[2];
      c.kx = (float)t.kx;
      c.ky = (float)t.ky;
      c.kz = (float)t.kz;
      c.ck = (float)(cscale / (t.kx * t.kx + t.ky * t.ky + t.kz * t.kz));
      c.ta = (float)t.a;
      c.tb = (float)t.b;
      c.ak = (float)ab[2 * (k0 + k)];
      c.bk = (float)ab[2 * (k0 + k) + 1];
      s_k[k] = c;
    }
    __syncthreads();
    for (int k = 0; k < kn; ++k) {
      const K32 c = s_k[k];
      const unsigned ph = c.m0 * a.x + c.m1 * a.y + c.m2 * a.z;
      float sn, cs;
      __sincosf((float)(int)ph * ang, &sn, &cs);
      const float gk = gix * c.kx + giy * c.ky + giz * c.kz;
      const float g1 = gk * (cs * c.tb - sn * c.ta);
      dq += (double)(g1 + c.ck * (c.ak * sn - c.bk * cs));
      const float coef = -gk * (sn * c.tb + cs * c.ta) + c.ck * (c.ak * cs + c.bk * sn);
      rx += (double)(coef * c.kx);
      ry += (double)(coef * c.ky);
      rz += (double)(coef * c.kz);
      gk_sum += (double)g1;
    }
  }
  if (live) {
    d_rx[i] += (double)qi * rx;
    d_ry[i] += (double)qi * ry;
    d_rz[i] += (double)qi * rz;
    d_q[i] += dq;
  }
  gk_sum = live ? gk_sum * (double)qi : 0.0;
  gk_sum = block_sum_det<ADJK_BLOCK>(gk_sum, s_sum);
  if (threadIdx.x == 0) part_gk[blockIdx.x] = gk_sum;
}

// Fixed-order reduction of part[k][nb] into out[2 * k + which].
__global__ void k_adj_reduce_k(int p, int nb, const double* __restrict__ part_a,
                               const double* __restrict__ part_b, double* __restrict__ ab) {
  __shared__ double sh[32];
  const int k = blockIdx.x;
  double a = 0.0, b = 0.0;
  for (int t = threadIdx.x; t < nb; t += blockDim.x) {
    a += part_a[(size_t)k * nb + t];
    b += part_b[(size_t)k * nb + t];
  }
  a = block_sum_det<128>(a, sh);
  b = block_sum_det<128>(b, sh);
  if (threadIdx.x == 0) {
    ab[2 * k] = a;
    ab[2 * k + 1] = b;
  }
}

__global__ void k_gather_vec3(int n, const int* __restrict__ orig, const double* __restrict__ src,
                              double* __restrict__ x, double* __restrict__ y,
                              double* __restrict__ z) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const size_t o = (size_t)orig[i] * 3;
  x[i] = src[o];
  y[i] = src[o + 1];
  z[i] = src[o + 2];
}

int launch_gather_vec3(int n, const int* orig, const double* src, double* x, double* y, double* z,
                       cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_gather_vec3<<<(n + 255) / 256, 256, 0, st>>>(n, orig, src, x, y, z);
  count_launch();
  return check_launch("gather_vec3");
}

int adj_pair_blocks(int n) {
  // up to four waves of the four resident blocks: the scheduler evens out the
  // atoms' work
  const int b = (n + ADJ_WARPS - 1) / ADJ_WARPS;
  return b < 16 * sm_count() ? (b < 1 ? 1 : b) : 16 * sm_count();
}

int launch_adj_pair(const PairParams& pp, int n, const uint4* atoms, const double* x,
                    const double* y, const double* z, const double* q, const int* type, const double* sigma_t,
                    const double* eps_t, const unsigned long long* key_a,
                    const unsigned long long* key_b, int epoch, const Rows& rows,
                    const double* gx, const double* gy,
                    const double* gz, const double mean_g[3], double* d_rx, double* d_ry,
                    double* d_rz, double* d_q, double* part, int nblocks, cudaStream_t st,
                    bool f32) {
  if (pp.ntypes > ADJ_MAX_TYPES) {
    set_error("adjoint: at most %d atom types", ADJ_MAX_TYPES);
    return RBX_ERR_INVALID;
  }
  if (n > AQ_INDEX) {
    set_error("adjoint: at most %d atoms", AQ_INDEX);
    return RBX_ERR_INVALID;
  }
  auto kern = f32 ? k_adj_pair<true> : k_adj_pair<false>;
  const size_t smem = sizeof(double) * 2 * pp.ntypes * ADJ_BLOCK;  // at most 64 KB
  if (smem > 32 * 1024 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess)
    return check_launch("adj_pair (shared memory)");
  kern<<<nblocks, ADJ_BLOCK, smem, st>>>(pp, n, atoms, x, y, z, q, type, sigma_t, eps_t, key_a,
                                         key_b, epoch, rows, gx, gy, gz, mean_g[0], mean_g[1],
                                         mean_g[2], d_rx, d_ry, d_rz, d_q, part);
  count_launch();
  return check_launch("adj_pair");
}

int adj_k_blocks(int n) { return (n + ADJK_BLOCK - 1) / ADJK_BLOCK; }

int launch_adj_kspace(int n, int p, double cscale, const KTab* tab, const double* q,
                      const double* x, const double* y, const double* z, const double* gx,
                      const double* gy, const double* gz, double* part_a, double* part_b,
                      int nparts, double* ab, double* d_rx, double* d_ry, double* d_rz,
                      double* d_q, double* part_gk, cudaStream_t st) {
  if (p <= 0 || n <= 0) return RBX_OK;
  const int chunk = (n + nparts - 1) / nparts;
  const int nb = (n + chunk - 1) / chunk;
  k_adj_k_ab<<<dim3(nb, (p + ADJK_BLOCK - 1) / ADJK_BLOCK), ADJK_BLOCK, 0, st>>>(
      n, p, chunk, tab, q, x, y, z, gx, gy, gz, part_a, part_b);
  count_launch();
  int rc = check_launch("adj_k_ab");
  if (rc) return rc;
  k_adj_reduce_k<<<p, 128, 0, st>>>(p, nb, part_a, part_b, ab);
  count_launch();
  rc = check_launch("adj_reduce_k");
  if (rc) return rc;
  k_adj_k_scatter<<<adj_k_blocks(n), ADJK_BLOCK, 0, st>>>(n, p, cscale, tab, ab, q, x, y, z, gx,
                                                          gy, gz, d_rx, d_ry, d_rz, d_q, part_gk);
  count_launch();
  return check_launch("adj_k_scatter");
}

int launch_adj_kspace_mixed(int n, int p, double cscale, const KTab* tab, const uint4* atoms,
                            const double* gx, const double* gy, const double* gz, double* part_a,
                            double* part_b, int nparts, double* ab, double* d_rx, double* d_ry,
                            double* d_rz, double* d_q, double* part_gk, cudaStream_t st) {
  if (p <= 0 || n <= 0) return RBX_OK;
  const int chunk = (n + nparts - 1) / nparts;
  const int nb = (n + chunk - 1) / chunk;
  k_adj_k_ab_mixed<<<dim3(nb, (p + ADJK_BLOCK - 1) / ADJK_BLOCK), ADJK_BLOCK, 0, st>>>(
      n, p, chunk, tab, atoms, gx, gy, gz, part_a, part_b);
  count_launch();
  int rc = check_launch("adj_k_ab_mixed");
  if (rc) return rc;
  k_adj_reduce_k<<<p, 128, 0, st>>>(p, nb, part_a, part_b, ab);
  count_launch();
  rc = check_launch("adj_reduce_k");
  if (rc) return rc;
  k_adj_k_scatter_mixed<<<adj_k_blocks(n), ADJK_BLOCK, 0, st>>>(
      n, p, cscale, tab, ab, atoms, gx, gy, gz, d_rx, d_ry, d_rz, d_q, part_gk);
  count_launch();
  return check_launch("adj_k_scatter_mixed");
}

}  // namespace rbx
