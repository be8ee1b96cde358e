// rbx_capi_f32.cu -- the op-level entry points for the reference's default
// build, where rbmd::Real is float (cmake/option.cmake: ENABLE_DOUBLE OFF,
// src/common/types.h:4-8).  Same argument order as the FP64 entries; every
// Real buffer and scalar is float.
//
// k-space: the structure factor and the RBE force run the mixed-form kernels
// (32-bit fixed-point fractional coordinates, exact integer phase m.u mod
// 2^32, FP32 sincos, FP64 cross-block reduction), so their error is that of
// the FP32 arithmetic on the phase, not of an FP32 k.r.  Energy and virial
// are summed in FP64.  Real space: every membership test (list predicate,
// force windows) is evaluated in float exactly as the float build evaluates
// it, so lists and kept pairs are the float build's; force values are FP64
// sums stored in float.
#include <cuda_runtime.h>

#include <initializer_list>

#include "rbx.h"
#include "rbx_capi_util.h"
#include "rbx_common.cuh"
#include "rbx_kernels.h"

namespace rbx {

// Up to eight float arrays of one length widened into consecutive runs of
// dst, in one launch (blockIdx.y: the array).
struct FloatSet {
  const float* src[8];
};
__global__ void k_widen(int n, FloatSet s, double* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[(size_t)n * blockIdx.y + i] = (double)s.src[blockIdx.y][i];
}
// Consecutive runs of src narrowed into up to eight float arrays.
struct FloatOut {
  float* dst[8];
};
__global__ void k_narrow(int n, const double* __restrict__ src, FloatOut o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) o.dst[blockIdx.y][i] = (float)src[(size_t)n * blockIdx.y + i];
}

// Fixed-point records {u_x, u_y, u_z, q} of float positions and charges, and
// (in the blocks after the atoms') the k-vectors and any further p-element
// arrays widened, the integer k-vectors: one launch prepares a whole call.
constexpr int PREP_BLOCK = 256;
__global__ void __launch_bounds__(PREP_BLOCK)
k_prepare_f32(DBox b, int n, const float* __restrict__ q, const float* __restrict__ x,
              const float* __restrict__ y, const float* __restrict__ z, uint4* __restrict__ atoms,
              int p, int narr, FloatSet s, double* __restrict__ wide, int* __restrict__ mi) {
  const int blocks_n = (n + PREP_BLOCK - 1) / PREP_BLOCK;
  if ((int)blockIdx.x < blocks_n) {
    const int i = blockIdx.x * PREP_BLOCK + threadIdx.x;
    if (i >= n) return;
    uint4 a;
    a.x = to_fixed((double)x[i], b.lo[0], 4294967296.0 / b.len[0]);
    a.y = to_fixed((double)y[i], b.lo[1], 4294967296.0 / b.len[1]);
    a.z = to_fixed((double)z[i], b.lo[2], 4294967296.0 / b.len[2]);
    a.w = __float_as_uint(q[i]);
    atoms[i] = a;
    return;
  }
  const int k = ((int)blockIdx.x - blocks_n) * PREP_BLOCK + threadIdx.x;
  if (k >= p) return;
  for (int a = 0; a < narr; ++a) wide[(size_t)p * a + k] = (double)s.src[a][k];
  if (mi)
    for (int d = 0; d < 3; ++d) mi[3 * k + d] = (int)s.src[d][k];
}

namespace {
// Device scratch freed on the stream when the call returns.
struct Scratch {
  cudaStream_t st;
  void* p[8] = {};
  int k = 0;
  explicit Scratch(cudaStream_t s) : st(s) {}
  template <typename T>
  int get(T** out, size_t count) {
    RBX_TRY(async_alloc(out, count, st));
    p[k++] = *out;
    return RBX_OK;
  }
  ~Scratch() {
    for (int i = 0; i < k; ++i) cudaFreeAsync(p[i], st);
  }
};

// Widened copies of n-element float arrays (contiguous, in argument order).
int widen_all(Scratch& s, int n, std::initializer_list<const float*> src, double** dst) {
  RBX_TRY(s.get(dst, (size_t)n * src.size()));
  FloatSet fs{};
  int k = 0;
  for (const float* a : src) fs.src[k++] = a;
  k_widen<<<dim3((n + 255) / 256, k), 256, 0, s.st>>>(n, fs, *dst);
  count_launch();
  return check_launch("widen");
}

int launch_narrow(int n, const double* src, std::initializer_list<float*> dst, cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  FloatOut o{};
  int k = 0;
  for (float* a : dst) o.dst[k++] = a;
  k_narrow<<<dim3((n + 255) / 256, k), 256, 0, st>>>(n, src, o);
  count_launch();
  return check_launch("narrow");
}

// Records of n atoms, p-element arrays widened (the first three are the
// k-vectors) and, with want_mi, the integer k-vectors.
int prepare(Scratch& s, const DBox& b, int n, const float* q, const float* x, const float* y,
            const float* z, uint4** atoms, int p, std::initializer_list<const float*> src,
            double** wide, int** mi) {
  RBX_TRY(s.get(atoms, (size_t)n));
  RBX_TRY(s.get(wide, (size_t)p * src.size()));
  if (mi) RBX_TRY(s.get(mi, (size_t)3 * p));
  FloatSet fs{};
  int k = 0;
  for (const float* a : src) fs.src[k++] = a;
  const int grid = (n + PREP_BLOCK - 1) / PREP_BLOCK + (p + PREP_BLOCK - 1) / PREP_BLOCK;
  k_prepare_f32<<<grid, PREP_BLOCK, 0, s.st>>>(b, n, q, x, y, z, *atoms, p, k, fs, *wide,
                                               mi ? *mi : nullptr);
  count_launch();
  return check_launch("prepare_f32");
}
}  // namespace
}  // namespace rbx

using namespace rbx;

extern "C" {

int rbx_rbe_structure_factor_f32(const rbx_box* box, int num_atoms, int p_number,
                                 const float* charge, const float* p_sample_x,
                                 const float* p_sample_y, const float* p_sample_z,
                                 const float* px, const float* py, const float* pz,
                                 float* density_real, float* density_imag, void* stream) {
  RBX_CHECK_BOX(box);
  if (num_atoms < 0 || p_number < 0) {
    set_error("rbx_rbe_structure_factor_f32: negative size");
    return RBX_ERR_INVALID;
  }
  if (p_number == 0) return RBX_OK;
  RBX_TRY(require_device());
  cudaStream_t st = (cudaStream_t)stream;
  Scratch s(st);
  const DBox b = make_dbox(*box);
  double* m = nullptr;  // samples widened: mx, my, mz
  const int nb = rbe_partial_blocks(num_atoms);
  double *part = nullptr, *rho = nullptr;
  RBX_TRY(s.get(&part, (size_t)2 * nb * p_number));
  RBX_TRY(s.get(&rho, (size_t)2 * p_number));
  double *pr = part, *pi = part + (size_t)nb * p_number;
  if (num_atoms > 0) {
    uint4* atoms = nullptr;
    int* mi = nullptr;
    RBX_TRY(prepare(s, b, num_atoms, charge, px, py, pz, &atoms, p_number,
                    {p_sample_x, p_sample_y, p_sample_z}, &m, &mi));
    RBX_TRY(launch_rbe_rho_partial_mixed(num_atoms, p_number, mi, atoms, pr, pi, nb, st));
  } else {
    RBX_TRY(widen_all(s, p_number, {p_sample_x, p_sample_y, p_sample_z}, &m));
    cudaMemsetAsync(part, 0, sizeof(double) * 2 * nb * p_number, st);
  }
  RBX_TRY(launch_rbe_finalize(b, p_number, nb, pr, pi, m, m + p_number, m + 2 * p_number, 1.0,
                              0.0, 1.0, 0.0, 0.0, rho, rho + p_number, nullptr, nullptr, nullptr,
                              0, nullptr, 0, nullptr, nullptr, st));
  return launch_narrow(p_number, rho, {density_real, density_imag}, st);
}

int rbx_rbe_force_f32(const rbx_box* box, int num_atoms, int p_number, float alpha,
                      float rbe_sum_gauss, float qqr2e, const float* real_array,
                      const float* imag_array, const float* charge, const float* p_sample_x,
                      const float* p_sample_y, const float* p_sample_z, const float* px,
                      const float* py, const float* pz, float* fx, float* fy, float* fz,
                      void* stream) {
  RBX_CHECK_BOX(box);
  if (num_atoms < 0 || p_number <= 0) {
    set_error("rbx_rbe_force_f32: need num_atoms >= 0 and p_number > 0");
    return RBX_ERR_INVALID;
  }
  if (num_atoms == 0) return RBX_OK;
  RBX_TRY(require_device());
  cudaStream_t st = (cudaStream_t)stream;
  Scratch s(st);
  const DBox b = make_dbox(*box);
  double *m = nullptr, *f = nullptr;
  uint4* atoms = nullptr;
  RBX_TRY(prepare(s, b, num_atoms, charge, px, py, pz, &atoms, p_number,
                  {p_sample_x, p_sample_y, p_sample_z, real_array, imag_array}, &m, nullptr));
  const double* rho = m + 3 * (size_t)p_number;
  KTab* tab = nullptr;
  RBX_TRY(s.get(&tab, (size_t)p_number));
  RBX_TRY(launch_rbe_finalize(b, p_number, 1, rho, rho + p_number, m, m + p_number,
                              m + 2 * p_number, alpha, rbe_sum_gauss, qqr2e, 0.0, 0.0, nullptr,
                              nullptr, nullptr, nullptr, tab, 0, nullptr, 0, nullptr, nullptr,
                              st));
  RBX_TRY(s.get(&f, (size_t)3 * num_atoms));
  RbeForceOut o;
  o.f_out_x = f;
  o.f_out_y = f + num_atoms;
  o.f_out_z = f + 2 * (size_t)num_atoms;
  RBX_TRY(launch_rbe_force_mixed(num_atoms, p_number, tab, atoms, o, st));
  return launch_narrow(num_atoms, f, {fx, fy, fz}, st);
}

int rbx_rbe_energy_virial_f32(const rbx_box* box, int p, float alpha, float rbe_sum_gauss,
                              float qqrd2e, float qsqsum, float qsum, const float* real_array,
                              const float* imag_array, const float* p_sample_x,
                              const float* p_sample_y, const float* p_sample_z,
                              float* virial_tensor, float* energy, void* stream) {
  RBX_CHECK_BOX(box);
  if (p <= 0 || !virial_tensor || !energy) {
    set_error("rbx_rbe_energy_virial_f32: need p > 0 and output pointers");
    return RBX_ERR_INVALID;
  }
  RBX_TRY(require_device());
  cudaStream_t st = (cudaStream_t)stream;
  Scratch s(st);
  const DBox b = make_dbox(*box);
  double *m = nullptr, *out = nullptr;
  RBX_TRY(widen_all(s, p, {p_sample_x, p_sample_y, p_sample_z, real_array, imag_array}, &m));
  const double* rho = m + 3 * (size_t)p;
  RBX_TRY(s.get(&out, 7));  // virial[6], energy
  RBX_TRY(launch_rbe_finalize(b, p, 1, rho, rho + p, m, m + p, m + 2 * p, alpha, rbe_sum_gauss,
                              qqrd2e, qsqsum, qsum, nullptr, nullptr, out + 6, out, nullptr, 0,
                              nullptr, 0, nullptr, nullptr, st));
  RBX_TRY(launch_narrow(6, out, {virial_tensor}, st));
  return launch_narrow(1, out + 6, {energy}, st);
}

int rbx_rbl_filter_f32(float core_cutoff_2, float force_cutoff_2, int total_atom_num,
                       const int* atoms_id, const float* px, const float* py, const float* pz,
                       const int* candidate_start, const int* candidate_end,
                       const int* candidate_neighbors, const int* max_core_neighbor_num,
                       const int* core_start, int* core_end, int* core_neighbors,
                       int random_neighbor_capacity, int* random_neighbors,
                       int* random_neighbors_num, int* required_random_neighbor_capacity,
                       const rbx_box* box, int* should_realloc, int selection_frequency,
                       int sample_epoch, void* stream) {
  RBX_CHECK_BOX(box);
  if (total_atom_num < 0 || random_neighbor_capacity < 0) {
    set_error("rbx_rbl_filter_f32: negative size");
    return RBX_ERR_INVALID;
  }
  RBX_TRY(require_device());
  return launch_ref_rbl_filter(core_cutoff_2, force_cutoff_2, total_atom_num, atoms_id, px, py,
                               pz, candidate_start, candidate_end, candidate_neighbors,
                               max_core_neighbor_num, core_start, core_end, core_neighbors,
                               random_neighbor_capacity, random_neighbors, random_neighbors_num,
                               required_random_neighbor_capacity, make_dbox(*box), should_realloc,
                               make_divtest(selection_frequency), sample_epoch,
                               (cudaStream_t)stream);
}

int rbx_pair_force_rbl_f32(const rbx_box* box, float rs, float rc, int num_atoms,
                           int neighbor_sample_num, int pice_num, float alpha, float qqr2e,
                           const int* atoms_type, const float* sigma, const float* eps,
                           const int* start_id, const int* end_id, const int* id_verletlist,
                           const int* id_random_neighbor, const int* random_neighbor_num,
                           const float* charge, const float* px, const float* py,
                           const float* pz, float* fx, float* fy, float* fz, void* stream) {
  (void)neighbor_sample_num;
  RBX_CHECK_BOX(box);
  if (num_atoms < 0) {
    set_error("rbx_pair_force_rbl_f32: negative num_atoms");
    return RBX_ERR_INVALID;
  }
  RBX_TRY(require_device());
  return launch_ref_pair_rbl(make_dbox(*box), rs, rc, num_atoms, pice_num, alpha, qqr2e,
                             atoms_type, sigma, eps, start_id, end_id, id_verletlist,
                             id_random_neighbor, random_neighbor_num, charge, px, py, pz, fx, fy,
                             fz, (cudaStream_t)stream);
}

int rbx_fix_rbl_force_f32(int num_atoms, float* fx, float* fy, float* fz, float* mean_out,
                          void* stream) {
  if (num_atoms <= 0) {
    set_error("rbx_fix_rbl_force_f32: num_atoms must be > 0");
    return RBX_ERR_INVALID;
  }
  RBX_TRY(require_device());
  cudaStream_t st = (cudaStream_t)stream;
  Scratch s(st);
  double* part = nullptr;
  RBX_TRY(s.get(&part, (size_t)3 * fix_rbl_parts(num_atoms)));
  return launch_fix_rbl(num_atoms, fx, fy, fz, mean_out, part, st);
}

int rbx_pair_force_verlet_f32(const rbx_box* box, float cut_off, int num_atoms, float alpha,
                              float qqr2e, const int* atoms_type, const float* sigma,
                              const float* eps, const int* start_id, const int* end_id,
                              const int* id_verletlist, const float* charge, const float* px,
                              const float* py, const float* pz, float* fx, float* fy, float* fz,
                              float* flat_virial, float* total_evdwl, float* total_ecoul,
                              void* stream) {
  RBX_CHECK_BOX(box);
  if (num_atoms < 0) {
    set_error("rbx_pair_force_verlet_f32: negative num_atoms");
    return RBX_ERR_INVALID;
  }
  if (num_atoms == 0) return RBX_OK;
  RBX_TRY(require_device());
  cudaStream_t st = (cudaStream_t)stream;
  Scratch s(st);
  double *epart = nullptr, *tot = nullptr;
  RBX_TRY(s.get(&epart, (size_t)2 * num_atoms));
  RBX_TRY(s.get(&tot, 2));
  RBX_TRY(launch_ref_pair_verlet(make_dbox(*box), cut_off, num_atoms, alpha, qqr2e, atoms_type,
                                 sigma, eps, start_id, end_id, id_verletlist, charge, px, py, pz,
                                 fx, fy, fz, flat_virial, epart, st));
  RBX_TRY(launch_reduce_cols(num_atoms, 2, epart, tot, 1.0, st));
  if (total_evdwl) RBX_TRY(launch_narrow(1, tot, {total_evdwl}, st));
  if (total_ecoul) RBX_TRY(launch_narrow(1, tot + 1, {total_ecoul}, st));
  return RBX_OK;
}

}  // extern "C"
