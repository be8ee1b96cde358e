// rbx_cells.cu -- cell binning, cell-sorted atom order, candidate (Verlet)
// lists and the velocity-Verlet integration kernels for sm_100a.
//
// Binning replaces LinkedCell::AssignAtomsToCell / SortAtomsByCellKey /
// ComputeCellRangesIndices (src/neighbor_list/src/linked_cell/linked_cell.cpp:428-670,
// src/neighbor_list/src/op/rocm/linked_cell_op.hip.cu:57-164) with a counting
// sort: atomic histogram, one-block scan, atomic scatter, then a per-cell
// bitonic sort.  Inside a cell atoms are ordered by a 4x4x4 Morton sub-cell
// code, then by old index (deterministic), so consecutive atoms are close in
// space: chunks of them have small bounding boxes for the list builder.
//
// The candidate list replaces Estimate/GenerateFullNeighborListOp
// (src/neighbor_list/src/op/rocm/full_neighbor_list_op.hip.cu:177-288): a
// block per 32 centre atoms stages the four-atom chunks of the 27 stencil
// cells that survive a bounding-box cull in shared memory and screens them in
// FP32; only pairs inside a guard band around the cutoff are
// settled with the reference's FP64 predicate, so the list is bit-identical
// (as a set) to the FP64 reference list.  Rows come out in stencil order,
// then in cell order.
#include <math.h>

#include <algorithm>

#include "rbx_common.cuh"
#include "rbx_kernels.h"

namespace rbx {

constexpr int SEG_MAX = 2048;  // atoms per cell handled by the segment sort

__device__ __forceinline__ int cell_coord(double v, double lo, double inv_edge, int dim) {
  int c = (int)floor((v - lo) * inv_edge);
  c = c < 0 ? 0 : c;
  return c > dim - 1 ? dim - 1 : c;
}

// Morton interleave of three 2-bit sub-cell coordinates.
__device__ __forceinline__ unsigned morton2(unsigned a, unsigned b, unsigned c) {
  unsigned m = 0;
#pragma unroll
  for (int bit = 0; bit < 2; ++bit)
    m |= ((a >> bit) & 1u) << (3 * bit) | ((b >> bit) & 1u) << (3 * bit + 1) |
         ((c >> bit) & 1u) << (3 * bit + 2);
  return m;
}

constexpr int SUB_SHIFT = 26;  // key = sub-cell code << 26 | old index (n < 2^26)

// Cell edge and its reciprocal per dimension, formed on the host as LinkedCell
// does (edge = box length / cells, reciprocal = 1 / edge).
struct CellGeom {
  double edge[3], inv[3];
};

// AssignAtomsToCell (linked_cell_op.hip.cu:57-138, no halo): floor((p - lo) *
// 1/edge) clamped, then, for a point outside that cell's bounds
// [lo + c edge, lo + (c + 1) edge) (products and sums rounded separately), a
// move of one cell per dimension that is kept only if the point lies inside
// the corrected cell.
__device__ __forceinline__ void assign_cell(const DBox& b, const CellGeom& g, const int dims[3],
                                            const double p[3], int c[3]) {
  bool inside = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    c[d] = cell_coord(p[d], b.lo[d], g.inv[d], dims[d]);
    const double cmin = __dadd_rn(__dmul_rn((double)c[d], g.edge[d]), b.lo[d]);
    const double cmax = __dadd_rn(__dmul_rn((double)(c[d] + 1), g.edge[d]), b.lo[d]);
    inside = inside && cmin <= p[d] && p[d] < cmax;
  }
  if (inside) return;
  int cc[3];
  bool ok = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double cmin = __dadd_rn(__dmul_rn((double)c[d], g.edge[d]), b.lo[d]);
    const double cmax = __dadd_rn(__dmul_rn((double)(c[d] + 1), g.edge[d]), b.lo[d]);
    cc[d] = c[d] + (p[d] < cmin ? -1 : (p[d] >= cmax ? 1 : 0));
    cc[d] = cc[d] < 0 ? 0 : (cc[d] > dims[d] - 1 ? dims[d] - 1 : cc[d]);
    const double nmin = __dadd_rn(__dmul_rn((double)cc[d], g.edge[d]), b.lo[d]);
    const double nmax = __dadd_rn(__dmul_rn((double)(cc[d] + 1), g.edge[d]), b.lo[d]);
    ok = ok && nmin <= p[d] && p[d] < nmax;
  }
  if (ok)
    for (int d = 0; d < 3; ++d) c[d] = cc[d];
}

__global__ void k_cell_assign(DBox b, CellGeom g, int dx, int dy, int dz, int n,
                              const double* __restrict__ x, const double* __restrict__ y,
                              const double* __restrict__ z, int* __restrict__ cell,
                              unsigned* __restrict__ sub, int* __restrict__ counts) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double fx = (x[i] - b.lo[0]) * (dx / b.len[0]);
  const double fy = (y[i] - b.lo[1]) * (dy / b.len[1]);
  const double fz = (z[i] - b.lo[2]) * (dz / b.len[2]);
  const int dims[3] = {dx, dy, dz};
  const double p[3] = {x[i], y[i], z[i]};
  int cc[3];
  assign_cell(b, g, dims, p, cc);
  const int cx = cc[0], cy = cc[1], cz = cc[2];
  const int c = (cz * dy + cy) * dx + cx;
  cell[i] = c;
  auto sub4 = [](double f, int c0) {
    int v = (int)floor((f - c0) * 4.0);
    return (unsigned)(v < 0 ? 0 : (v > 3 ? 3 : v));
  };
  sub[i] = n < (1 << SUB_SHIFT) ? morton2(sub4(fx, cx), sub4(fy, cy), sub4(fz, cz)) : 0u;
  // atoms still in the order of the last sort share cells along a warp: one
  // atomic per distinct cell of the warp
  const unsigned same = __match_any_sync(__activemask(), c);
  if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(counts + c, __popc(same));
}

// Exclusive scan of counts into start[0..ncell] (one block of 1024 threads).
__global__ void __launch_bounds__(1024)
k_cell_scan(int ncell, const int* __restrict__ counts, int* __restrict__ start,
            int* __restrict__ fill) {
  __shared__ int s_warp[32];
  __shared__ int s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int base = 0; base < ncell; base += 1024) {
    const int c = base + threadIdx.x;
    const int v = c < ncell ? counts[c] : 0;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    if (w == 0) {
      int ws = s_warp[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, ws, o);
        if (lane >= o) ws += t;
      }
      s_warp[lane] = ws;
    }
    __syncthreads();
    const int excl = s_carry + (w > 0 ? s_warp[w - 1] : 0) + incl - v;
    if (c < ncell) {
      start[c] = excl;
      fill[c] = excl;
    }
    __syncthreads();
    if (threadIdx.x == 1023) s_carry = excl + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) start[ncell] = s_carry;
}

__global__ void k_cell_scatter(int n, const int* __restrict__ cell,
                               const unsigned* __restrict__ sub, int* __restrict__ fill,
                               unsigned* __restrict__ tmp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  // one atomic per distinct cell of the warp; the order inside a cell is set
  // by the segment sort that follows
  const int c = cell[i];
  const unsigned same = __match_any_sync(__activemask(), c);
  const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(fill + c, __popc(same));
  base = __shfl_sync(same, base, leader);
  tmp[base + __popc(same & ((1u << lane) - 1u))] = (sub[i] << SUB_SHIFT) | (unsigned)i;
}

// One block per cell: bitonic sort of the cell's keys (sub-cell, old index).  128
// threads a block let many cells be resident at once; 512 shorten the passes over
// full cells.  Measured, B200, 200,000 atoms of 120 / 200 / 300 / 400 / 600 / 1,200 a
// cell: 13 / 11 / 18 / 18 / 35 / 75 us with 128, 21 / 16 / 19 / 15 / 21 / 30 with 512;
// 27 cells of 120 8.3 and 6.2, where all are resident either way.
constexpr int SORT_BLOCK = 128, SORT_BLOCK_FULL = 512;
static int sort_block(int n, int ncell) {
  const long long full = ncell <= 2 * sm_count() ? 100 : 350;  // atoms a cell
  return n < full * ncell ? SORT_BLOCK : SORT_BLOCK_FULL;
}
__global__ void __launch_bounds__(SORT_BLOCK_FULL)
k_cell_segsort(int ncell, int n, const int* __restrict__ start, const unsigned* __restrict__ tmp,
               int* __restrict__ perm, int* __restrict__ cell_of_sorted, int* __restrict__ status) {
  __shared__ unsigned s[SEG_MAX];
  const int c = blockIdx.x;
  const int a = start[c], cnt = start[c + 1] - a;
  const unsigned mask = n < (1 << SUB_SHIFT) ? (1u << SUB_SHIFT) - 1u : 0xffffffffu;
  if (cnt > SEG_MAX) {  // reported; the cell keeps a valid, unsorted permutation
    if (threadIdx.x == 0) atomicOr(status, 2);
    for (int t = threadIdx.x; t < cnt; t += blockDim.x) {
      perm[a + t] = (int)(tmp[a + t] & mask);
      cell_of_sorted[a + t] = c;
    }
    return;
  }
  int p2 = 1;
  while (p2 < cnt) p2 <<= 1;
  for (int t = threadIdx.x; t < p2; t += blockDim.x) s[t] = t < cnt ? tmp[a + t] : 0xffffffffu;
  __syncthreads();
  for (int k = 2; k <= p2; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = threadIdx.x; t < p2; t += blockDim.x) {
        const int u = t ^ j;
        if (u > t) {
          const bool up = (t & k) == 0;
          const unsigned va = s[t], vb = s[u];
          if ((va > vb) == up) {
            s[t] = vb;
            s[u] = va;
          }
        }
      }
      __syncthreads();
    }
  }
  for (int t = threadIdx.x; t < cnt; t += blockDim.x) {
    perm[a + t] = (int)(s[t] & mask);
    cell_of_sorted[a + t] = c;
  }
}

// ---------------------------------------------------------------------------
// Candidate list.  A block of eight warps builds the rows of one group of up
// to 32 consecutive centre atoms of a cell, four atoms a warp.
//
// The atoms of a cell are also cut into chunks of four (consecutive in the
// cell's Morton order); chunk k of cell c sits at table index
// (cell_start[c] >> 2) + c + k, which is unique and needs no scan (the
// indices of consecutive cells never overlap).  k_chunk_boxes writes each
// chunk's bounding box, rounded outwards to FP32.  Groups are numbered the
// same way with 32 in place of four; a group index between two cells has
// group_cell -1.
//
// Level 1: the block culls the chunks of the 27 stencil cells against the
// box of its centre atoms (directed rounding: a lower bound of the true box
// distance, so no pair within the cutoff is ever culled); the survivors, in
// stencil order, are staged in shared memory as {v, |v|^2}, FP32 coordinates
// relative to the centre cell's centre with the periodic image applied.
// Level 2: each warp culls the staged chunks against the box of its own four
// centre atoms.  Then a lane takes one staged atom (eight chunks an
// iteration) and tests it against the four centres as |v|^2 - 2 u.v <
// C - |u|^2: three FMAs per pair.  Pairs inside a guard band around the
// cutoff are settled with the reference's FP64 predicate, so the list equals
// the FP64 reference list as a set; hits are appended through a ballot
// prefix, so rows come out in stencil order, then in cell order.
//
// Split rows (RBL engines): a pair whose build distance is certainly at
// least r_near = r_core + skin cannot come within r_core before the next
// rebuild (no atom moves more than skin/2 before one), so the fused RBL
// kernel tests it with its batch hash first.  Such far pairs are written from
// the end of the row backwards; every other candidate from the front.
// count[i] is the number of candidates (above cap: overflow), far[i] the
// number of far ones; a row that overflows holds some cap of its candidates.
//
// Bound by issue and by the barriers between a block's phases: 70 % of the issue
// slots are taken (split rows 74 %) with half of the warp slots (64 registers,
// 52 KB: four blocks an SM), and of the ten cycles a warp spends on an instruction
// 2.3 are waits at a barrier, the largest share.  An append in half its
// instructions was no faster.  Four centres a warp and four-atom chunks leave
// about 1,400 tested slots an atom at rho* = 0.8, cutoff 5.3 (499 hits; 1,860 warp
// instructions, 2,350 with split rows), against 3,700 slots when one warp tests
// 32-atom chunks against 32 centres, one a lane; and a small box fills the chip.
// Measured, B200, rho* = 0.8, cutoff 5.3, one warp per 32 centres and this:
// 200,000 atoms 660 and 466 us (split rows 915 and 614), 20,000 atoms split 214
// and 92, 4,000 atoms split 171 and 42.
// ---------------------------------------------------------------------------
// W, the warps of a block (centre atoms 4 W): eight, or one where cells hold a few
// atoms, whose blocks would leave most of eight warps idle.
constexpr int NL_CH = 4;  // atoms of a chunk, centre atoms of a warp
template <int W>
struct ListShape {
  static constexpr int GROUP = NL_CH * W;            // centre atoms of a block
  static constexpr int BATCH = W == 8 ? 448 : 64;    // chunks staged at a time
  static constexpr int WORDS = W == 8 ? 256 : 64;    // 32-chunk cull words handled at a time
  static constexpr int RESIDENT = W == 8 ? 4 : 24;   // blocks of an SM
};

__device__ __forceinline__ int chunk_base(int c, int cs) { return cs / NL_CH + c; }
__device__ __forceinline__ int group_base(int c, int cs, int group) { return cs / group + c; }

static size_t full_list_groups(int n, int ncell, int group) { return (size_t)(n / group) + ncell; }
static size_t full_list_chunks(int n, int ncell) { return (size_t)(n / NL_CH) + ncell; }
// With fewer than LIST_DILUTE atoms a cell on average the cells of at most LIST_FEW
// atoms go to one-warp blocks (a second launch), the others to the eight-warp
// blocks, as all do in a denser box: a gas and a droplet in a large box each get
// the blocks that suit them.  The indices of the eight-warp groups are then
// gathered first: a block that finds none costs 1 ns, and most would.  Measured,
// B200, us, eight warps / one for all cells: 200,000 atoms of 0.3, 1, 3, 6 and 12 a
// cell 1779 / 545, 1252 / 556, 809 / 529, 475 / 469, 314 / 508; 4,000 atoms of 1, 2,
// 3 and 6 32 / 20, 28 / 24, 22 / 25, 18 / 27.
constexpr long long LIST_DILUTE = 3;
constexpr int LIST_FEW = 6;
static bool list_dilute(int n, int ncell) { return n < LIST_DILUTE * ncell; }
// Most groups that cells of more than LIST_FEW atoms can make.
static int list_many(int n) { return n / ListShape<8>::GROUP + n / (LIST_FEW + 1) + 1; }

// Device scratch of one list build.
struct ListTables {
  float4* rel;      // plain rows: an atom's FP32 position relative to its cell's centre
  float4 *lo, *hi;  // per chunk: its box relative to its cell's centre, rounded outwards
  int* group_cell;  // per group: its cell, -1 for an index without a group
  int* few_cell;    // the same for the one-warp blocks, null where there are none
  int* many;        // then: how many groups group_cell has, and their indices
};

__global__ void __launch_bounds__(128)
k_chunk_boxes(DBox b, int dimx, int dimy, int dimz, const double* __restrict__ x,
              const double* __restrict__ y, const double* __restrict__ z,
              const int* __restrict__ cell_start, ListTables T) {
  const int c = blockIdx.x;
  const int cs = cell_start[c], ce = cell_start[c + 1];
  const int base = chunk_base(c, cs);
  const int cz = c / (dimx * dimy), cy = (c / dimx) % dimy, cx = c % dimx;
  const double o[3] = {b.lo[0] + (cx + 0.5) * (b.len[0] / dimx),
                       b.lo[1] + (cy + 0.5) * (b.len[1] / dimy),
                       b.lo[2] + (cz + 0.5) * (b.len[2] / dimz)};
  // a lane an atom, a chunk four neighbouring lanes
  for (int a0 = cs; a0 < ce; a0 += blockDim.x) {
    const int a = a0 + threadIdx.x;
    const bool ok = a < ce;
    const double p[3] = {ok ? x[a] : 0.0, ok ? y[a] : 0.0, ok ? z[a] : 0.0};
    float lo[3], hi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      lo[d] = ok ? __double2float_rd(__dsub_rd(p[d], o[d])) : INFINITY;
      hi[d] = ok ? __double2float_ru(__dsub_ru(p[d], o[d])) : -INFINITY;
#pragma unroll
      for (int s = 1; s < NL_CH; s <<= 1) {
        lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], s));
        hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], s));
      }
    }
    if (!ok) continue;
    if (T.rel)
      T.rel[a] =
          make_float4((float)(p[0] - o[0]), (float)(p[1] - o[1]), (float)(p[2] - o[2]), 0.f);
    if (threadIdx.x % NL_CH == 0) {
      const int k = base + (a - cs) / NL_CH;
      T.lo[k] = make_float4(lo[0], lo[1], lo[2], 0.f);
      T.hi[k] = make_float4(hi[0], hi[1], hi[2], 0.f);
    }
  }
  const bool few = T.few_cell && ce - cs <= LIST_FEW;
  auto groups = [&](int* __restrict__ of, int size, bool taken) {
    const int g0 = group_base(c, cs, size), ng = taken ? (ce - cs + size - 1) / size : 0;
    const int g1 = group_base(c + 1, ce, size);  // first index of the next cell
    for (int g = g0 + threadIdx.x; g < g1; g += blockDim.x) of[g] = g < g0 + ng ? c : -1;
  };
  groups(T.group_cell, ListShape<8>::GROUP, !few);
  if (T.few_cell) groups(T.few_cell, ListShape<1>::GROUP, few);
  if (T.few_cell && c == 0 && threadIdx.x == 0) T.many[0] = 0;
}

// The indices of the groups in group_cell, in any order (rows do not depend on it).
__global__ void __launch_bounds__(256) k_many_groups(int groups, ListTables T) {
  __shared__ int s_at[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = blockIdx.x * 256 + threadIdx.x;
  const bool live = g < groups && T.group_cell[g] >= 0;
  const unsigned m = __ballot_sync(0xffffffffu, live);
  if (lane == 0) s_at[warp] = __popc(m);
  __syncthreads();
  if (threadIdx.x == 0) {
    int sum = 0;
    for (int w = 0; w < 8; ++w) {
      const int k = s_at[w];
      s_at[w] = sum;
      sum += k;
    }
    const int first = sum ? atomicAdd(T.many, sum) : 0;
    for (int w = 0; w < 8; ++w) s_at[w] += first;
  }
  __syncthreads();
  if (live) T.many[1 + s_at[warp] + __popc(m & ((1u << lane) - 1u))] = g;
}

// A store under a predicate, without a branch around it.
__device__ __forceinline__ void store_if(bool take, int* p, int v) {
  asm volatile(
      "{\n\t.reg .pred t;\n\tsetp.ne.u32 t, %0, 0;\n\t@t st.global.u32 [%1], %2;\n\t}" ::"r"(
          (unsigned)take),
      "l"(p), "r"(v)
      : "memory");
}

template <int W>
struct FullListSmem {
  static constexpr int BATCH = ListShape<W>::BATCH, WORDS = ListShape<W>::WORDS;
  float4 atom[(BATCH + 1) * NL_CH];  // staged chunks; the last one is empty
  float2 bx[BATCH], by[BATCH], bz[BATCH];  // {lo, hi} of a staged chunk
  int first[BATCH + 1];              // its first atom
  unsigned short meta[BATCH];        // stencil cell | atoms << 8
  unsigned short pick[W][BATCH + 8];  // a warp's surviving chunks
  float4 edge[27];                      // centre of a stencil cell's image, relative to the
  float shl[27][3], shh[27][3];         // centre cell's; and rounded down and up
  double shift[27][3];                  // its periodic image minus the centre cell's centre
  int cs[27], ce[27], cb[27];           // atom range and first chunk index of a stencil cell
  int word0[28];                        // first cull word of a stencil cell
  unsigned mask[WORDS];              // surviving chunks of a word
  int off[WORDS + 1];                // survivors before it
};

// SPLIT: RBL rows with a far segment; without it (Verlet lists) no far test.
template <bool SPLIT, int W>
__global__ void __launch_bounds__(32 * W, ListShape<W>::RESIDENT)
k_full_list(DBox b, int dimx, int dimy, int dimz, double cut2, float cut2_up, float lo_band,
            float hi_band, const double* __restrict__ x, const double* __restrict__ y,
            const double* __restrict__ z, const int* __restrict__ cell_start, ListTables T,
            int cap, int* __restrict__ count, int* __restrict__ nbrs, int* __restrict__ overflow,
            float near2, int* __restrict__ far, long long* __restrict__ total) {
  constexpr int BLOCK = 32 * W, GROUP = ListShape<W>::GROUP;
  constexpr int BATCH = ListShape<W>::BATCH, WORDS = ListShape<W>::WORDS;
  extern __shared__ __align__(16) unsigned char s_list[];
  FullListSmem<W>& S = *reinterpret_cast<FullListSmem<W>*>(s_list);
  int block = blockIdx.x;
  if (W == 8 && T.few_cell) {
    if (block >= T.many[0]) return;
    block = T.many[1 + block];
  }
  const int c = (W == 1 ? T.few_cell : T.group_cell)[block];
  if (c < 0) return;  // an index without a group
  // the warp's index through a shuffle, so that the compiler knows the loops
  // below to be uniform over the warp
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const unsigned lt = (1u << lane) - 1u;
  const int cs = cell_start[c], ce = cell_start[c + 1];
  const int g = block - group_base(c, cs, GROUP);
  const int i0 = cs + GROUP * g + NL_CH * warp;  // this warp's first centre atom
  const int cz = c / (dimx * dimy), cy = (c / dimx) % dimy, cx = c % dimx;
  const double ox = b.lo[0] + (cx + 0.5) * (b.len[0] / dimx);  // the centre cell's centre
  const double oy = b.lo[1] + (cy + 0.5) * (b.len[1] / dimy);
  const double oz = b.lo[2] + (cz + 0.5) * (b.len[2] / dimz);
  if (warp == 0) {  // the stencil cells, and their cull words
    int words = 0;
    if (lane < 27) {
      // stencil order of ComputeFullNeighborStencilCellOnTheFly:
      // offsets (s%3-1, (s/3)%3-1, s/9-1); the image's centre lies that many
      // cell edges away
      const int o[3] = {lane % 3 - 1, (lane / 3) % 3 - 1, lane / 9 - 1};
      const int dim[3] = {dimx, dimy, dimz}, at[3] = {cx + o[0], cy + o[1], cz + o[2]};
      const double cen[3] = {ox, oy, oz};
      int w[3];
      float ed[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        w[d] = at[d] < 0 ? at[d] + dim[d] : (at[d] >= dim[d] ? at[d] - dim[d] : at[d]);
        const double e = o[d] * (b.len[d] / dim[d]);
        ed[d] = (float)e;
        S.shift[lane][d] =
            (at[d] < 0 ? -b.len[d] : (at[d] >= dim[d] ? b.len[d] : 0.0)) - cen[d];
        // one FP64 rounding of the edge and of the two centres: 4 ulp of the
        // box's extent cover them
        const double slack = 1e-15 * (fabs(b.lo[d]) + b.len[d]);
        S.shl[lane][d] = __double2float_rd(__dsub_rd(e, slack));
        S.shh[lane][d] = __double2float_ru(__dadd_ru(e, slack));
      }
      S.edge[lane] = make_float4(ed[0], ed[1], ed[2], 0.f);
      const int nc = (w[2] * dimy + w[1]) * dimx + w[0];
      S.cs[lane] = cell_start[nc];
      S.ce[lane] = cell_start[nc + 1];
      S.cb[lane] = chunk_base(nc, S.cs[lane]);
      words = (S.ce[lane] - S.cs[lane] + 32 * NL_CH - 1) / (32 * NL_CH);
    }
    int incl = words;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, k);
      if (lane >= k) incl += t;
    }
    if (lane < 27) S.word0[lane + 1] = incl;
    if (lane == 0) S.word0[0] = 0;
  }
  if (threadIdx.x < NL_CH) S.atom[BATCH * NL_CH + threadIdx.x] =
      make_float4(0.f, 0.f, 0.f, INFINITY);  // an empty slot: never a hit
  if (threadIdx.x == NL_CH) S.first[BATCH] = 0;
  // this warp's centres i0 + q: their tests and their box (it is their chunk's)
  float ax[NL_CH], ay[NL_CH], az[NL_CH], lo_i[NL_CH], hi_i[NL_CH], near_i[NL_CH];
#pragma unroll
  for (int q = 0; q < NL_CH; ++q) {
    const bool live = i0 + q < ce;
    const int i = live ? i0 + q : cs;
    const float ux = (float)(x[i] - ox), uy = (float)(y[i] - oy), uz = (float)(z[i] - oz);
    const float uu = fmaf(ux, ux, fmaf(uy, uy, uz * uz));
    ax[q] = live ? -2.f * ux : 0.f;
    ay[q] = live ? -2.f * uy : 0.f;
    az[q] = live ? -2.f * uz : 0.f;
    lo_i[q] = live ? lo_band - uu : -INFINITY;
    hi_i[q] = live ? hi_band - uu : -INFINITY;
    near_i[q] = near2 - uu;  // far pairs: d above this
  }
  const int own = chunk_base(c, cs) + W * g;  // the group's first chunk
  float ulo[3], uhi[3], glo[3], ghi[3];                   // boxes of the group, of the warp
  {
    const bool ok = lane < W && cs + GROUP * g + NL_CH * lane < ce;
    const float4 l = T.lo[ok ? own + lane : own], h = T.hi[ok ? own + lane : own];
    const float ll[3] = {l.x, l.y, l.z}, hh[3] = {h.x, h.y, h.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      glo[d] = __shfl_sync(0xffffffffu, ll[d], warp);
      ghi[d] = __shfl_sync(0xffffffffu, hh[d], warp);
      ulo[d] = ll[d];  // lanes without a chunk repeat the first
      uhi[d] = hh[d];
#pragma unroll
      for (int s = 1; s < W; s <<= 1) {
        ulo[d] = fminf(ulo[d], __shfl_xor_sync(0xffffffffu, ulo[d], s));
        uhi[d] = fmaxf(uhi[d], __shfl_xor_sync(0xffffffffu, uhi[d], s));
      }
      ulo[d] = __shfl_sync(0xffffffffu, ulo[d], 0);
      uhi[d] = __shfl_sync(0xffffffffu, uhi[d], 0);
    }
  }
  int nfront[NL_CH], nback[NL_CH];
#pragma unroll
  for (int q = 0; q < NL_CH; ++q) nfront[q] = nback[q] = 0;
  int* const row = nbrs + (size_t)i0 * cap;  // NL_CH rows, back to back
  __syncthreads();

  // the box of chunk k of stencil cell s relative to the centre cell's centre
  auto chunk_box = [&](int s, int k, float rl[3], float rh[3]) {
    const float4 bl = T.lo[S.cb[s] + k], bh = T.hi[S.cb[s] + k];
    const float l[3] = {bl.x, bl.y, bl.z}, h[3] = {bh.x, bh.y, bh.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      rl[d] = __fadd_rd(l[d], S.shl[s][d]);
      rh[d] = __fadd_ru(h[d], S.shh[s][d]);
    }
  };
  // lower bound of the squared distance of boxes [al, ah] and [bl, bh]
  auto gap2 = [](const float al[3], const float ah[3], const float bl[3], const float bh[3]) {
    float e[3];
#pragma unroll
    for (int d = 0; d < 3; ++d)
      e[d] = fmaxf(0.f, fmaxf(__fsub_rd(bl[d], ah[d]), __fsub_rd(al[d], bh[d])));
    return __fadd_rd(__fadd_rd(__fmul_rd(e[0], e[0]), __fmul_rd(e[1], e[1])),
                     __fmul_rd(e[2], e[2]));
  };
  // stencil cell of cull word w
  auto word_cell = [&](int w) {
    return __popc(__ballot_sync(0xffffffffu, lane < 27 && S.word0[min(lane, 27)] <= w)) - 1;
  };

  const int nwords = S.word0[27];
  for (int wb = 0; wb < nwords; wb += WORDS) {
    const int nw = min(WORDS, nwords - wb);
    for (int w = warp; w < nw; w += W) {  // level 1
      const int s = word_cell(wb + w);
      const int k = (wb + w - S.word0[s]) * 32 + lane;
      bool near = false;
      if (k * NL_CH < S.ce[s] - S.cs[s]) {
        float rl[3], rh[3];
        chunk_box(s, k, rl, rh);
        near = gap2(ulo, uhi, rl, rh) < cut2_up;
      }
      const unsigned m = __ballot_sync(0xffffffffu, near);
      if (lane == 0) S.mask[w] = m;
    }
    __syncthreads();
    if (warp == 0) {  // survivors before each word
      int carry = 0;
      for (int w0 = 0; w0 < nw; w0 += 32) {
        const int v = w0 + lane < nw ? __popc(S.mask[w0 + lane]) : 0;
        int incl = v;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, k);
          if (lane >= k) incl += t;
        }
        if (w0 + lane < nw) S.off[w0 + lane] = carry + incl - v;
        carry += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) S.off[nw] = carry;
    }
    __syncthreads();
    const int found = S.off[nw];
    for (int b0 = 0; b0 < found; b0 += BATCH) {
      const int nb = min(BATCH, found - b0);
      for (int w = warp; w < nw; w += W) {  // the batch's chunks
        if (S.off[w + 1] <= b0 || S.off[w] >= b0 + BATCH) continue;
        const int s = word_cell(wb + w);
        const unsigned m = S.mask[w];
        const int slot = S.off[w] + __popc(m & lt) - b0;
        if (((m >> lane) & 1u) && slot >= 0 && slot < BATCH) {
          const int k = (wb + w - S.word0[s]) * 32 + lane;
          float rl[3], rh[3];
          chunk_box(s, k, rl, rh);
          S.bx[slot] = make_float2(rl[0], rh[0]);
          S.by[slot] = make_float2(rl[1], rh[1]);
          S.bz[slot] = make_float2(rl[2], rh[2]);
          const int a = S.cs[s] + NL_CH * k;
          S.first[slot] = a;
          S.meta[slot] = (unsigned short)(s | min(NL_CH, S.ce[s] - a) << 8);
        }
      }
      __syncthreads();
#pragma unroll 4
      for (int t = threadIdx.x; t < nb * NL_CH; t += BLOCK) {  // its atoms
        const int slot = t / NL_CH, u = t % NL_CH;
        const int meta = S.meta[slot];
        const double* const sh = S.shift[meta & 255];
        float4 v = make_float4(0.f, 0.f, 0.f, INFINITY);
        if (u < meta >> 8) {
          const int a = S.first[slot] + u;
          if (SPLIT) {
            v.x = (float)(x[a] + sh[0]);
            v.y = (float)(y[a] + sh[1]);
            v.z = (float)(z[a] + sh[2]);
          } else {
            const float4 r = T.rel[a], e = S.edge[meta & 255];
            v.x = r.x + e.x;
            v.y = r.y + e.y;
            v.z = r.z + e.z;
          }
          v.w = fmaf(v.x, v.x, fmaf(v.y, v.y, v.z * v.z));
        }
        S.atom[t] = v;
      }
      __syncthreads();
      if (i0 < ce) {
        unsigned short* const pick = S.pick[warp];
        int np = 0;
        for (int k0 = 0; k0 < nb; k0 += 32) {  // level 2
          const int k = min(k0 + lane, nb - 1);
          const float2 vx = S.bx[k], vy = S.by[k], vz = S.bz[k];
          const float rl[3] = {vx.x, vy.x, vz.x}, rh[3] = {vx.y, vy.y, vz.y};
          const bool near = (gap2(glo, ghi, rl, rh) < cut2_up) & (k0 + lane < nb);
          const unsigned m = __ballot_sync(0xffffffffu, near);
          if (near) pick[np + __popc(m & lt)] = (unsigned short)k;
          np += __popc(m);
        }
        if (lane < 8) pick[np + lane] = BATCH;  // pad with the empty chunk
        __syncwarp();
        const int u = lane % NL_CH;
        for (int t = 0; t < np; t += 32 / NL_CH) {
          const int ch = pick[t + lane / NL_CH];
          const float4 v = S.atom[ch * NL_CH + u];
          const int j = S.first[ch] + u;
          float d[NL_CH];
          bool in[NL_CH];
          // the warp's own chunk (its lanes meet themselves) and pairs in the
          // guard band are settled one by one
          bool odd = (unsigned)(j - i0) < (unsigned)NL_CH;
#pragma unroll
          for (int q = 0; q < NL_CH; ++q) {
            d[q] = fmaf(ax[q], v.x, fmaf(ay[q], v.y, fmaf(az[q], v.z, v.w)));
            in[q] = d[q] < lo_i[q];
            odd |= in[q] ^ (d[q] < hi_i[q]);
          }
          if (__any_sync(0xffffffffu, odd)) {
#pragma unroll
            for (int q = 0; q < NL_CH; ++q) {
              const int i = i0 + q;
              if (in[q] != (d[q] < hi_i[q]))  // the FP64 predicate decides
                in[q] = dist2_list(b, x[i], y[i], z[i], x[j], y[j], z[j]) < cut2;
              in[q] = in[q] && j != i;
            }
          }
#pragma unroll
          for (int q = 0; q < NL_CH; ++q) {
            if (SPLIT) {
              const bool bk = in[q] & (d[q] > near_i[q]);
              const unsigned mb = __ballot_sync(0xffffffffu, bk);
              const unsigned mf = __ballot_sync(0xffffffffu, in[q]) ^ mb;
              const int pos = (bk ? nback[q] : nfront[q]) + __popc((bk ? mb : mf) & lt);
              store_if(in[q] & (pos < cap), row + (q * cap + (bk ? cap - 1 - pos : pos)), j);
              nback[q] += __popc(mb);
              nfront[q] += __popc(mf);
            } else {
              const unsigned m = __ballot_sync(0xffffffffu, in[q]);
              const int pos = nfront[q] + __popc(m & lt);
              store_if(in[q] & (pos < cap), row + (q * cap + pos), j);
              nfront[q] += __popc(m);
            }
          }
        }
      }
      __syncthreads();  // the next batch overwrites this one
    }
  }
  int sum = 0;
#pragma unroll
  for (int q = 0; q < NL_CH; ++q) {
    const int n = nfront[q] + nback[q];
    if (i0 + q < ce && lane == q) {
      count[i0 + q] = n;
      if (SPLIT) far[i0 + q] = nback[q];
      if (n > cap) atomicOr(overflow, 1);
    }
    sum += n;
  }
  if (total && lane == 0 && i0 < ce) atomicAdd((unsigned long long*)total, (unsigned long long)sum);
}

// ---------------------------------------------------------------------------
// Candidate rows for boxes with fewer than three cells of edge cut_off + skin
// along some axis (edge between two and three times cut_off + skin): every
// atom j != i is tested with the reference's FP64 predicate (CaculateDistance:
// i minus j, single-shift minimum image, no FMA), so each pair is listed once.
// (The reference's cells have edge (cut_off + skin) / c, c = 1 for a Verlet
// list and ceil((cut_off + skin) / r_core) for RBL (linked_cell_locator.cpp:
// 26-40), and its (2c + 1)^3 stencil wraps onto the same cell more than once
// along an axis with fewer than 2c + 1 cells, WrapFullNeighborStencilIndex in
// full_neighbor_list_op.hip.cu:9-80, listing those pairs repeatedly.)
//
// Bound by latency and issue: n / 32 tests a lane of a warp, a few blocks an SM.
// A warp takes SL_C centre atoms; a block stages the fixed-point records of all
// atoms tile by tile.  Their wrapped differences are the minimum image, and
// |d|^2 in FP32 decides every pair outside a guard band (the RBL kernels'
// bound) around the cutoff and around r_near; the FP64 distance settles the
// rest.  Hits are appended in index order through a ballot prefix, far pairs (at
// least r_near, see FarSplit) to the back.  Measured, B200, 1,000 / 1,500 / 3,000
// atoms: 10.8 / 14.9 / 36.0 us; 16.5 / 23.6 / 43.0 us with a warp an atom and FP64
// distances.
// ---------------------------------------------------------------------------
constexpr int SL_WARPS = 8;
constexpr int SL_C = 2;       // centre atoms of a warp
constexpr int SL_TILE = 1024; // atoms staged at a time

struct SmallScreen {
  IntScreen cut, near;  // of the fixed-point |d|^2: list cutoff, near and far segment
  double cut2, near2;   // the same in FP64
  float cut_mid, cut_half, near_mid, near_half;  // intervals that contain the bands
  float w[3];           // L_d / L_max
};

template <bool SPLIT>
__global__ void __launch_bounds__(32 * SL_WARPS)
k_full_list_small(DBox b, SmallScreen sc, int n, const uint4* __restrict__ atoms,
                  const double* __restrict__ x, const double* __restrict__ y,
                  const double* __restrict__ z, int cap, int* __restrict__ count,
                  int* __restrict__ nbrs, int* __restrict__ overflow, int* __restrict__ far,
                  long long* __restrict__ total) {
  __shared__ uint4 s_u[SL_TILE];
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const unsigned lt = (1u << lane) - 1u;
  const int i0 = (blockIdx.x * SL_WARPS + warp) * SL_C;
  uint4 u[SL_C];
  int nf[SL_C], nb[SL_C];
#pragma unroll
  for (int q = 0; q < SL_C; ++q) {
    u[q] = atoms[min(i0 + q, n - 1)];
    nf[q] = nb[q] = 0;
  }
  int* const row = nbrs + (size_t)i0 * cap;
  for (int t0 = 0; t0 < n; t0 += SL_TILE) {
    const int tn = min(SL_TILE, n - t0);
    __syncthreads();  // the previous tile has been read
    for (int t = threadIdx.x; t < tn; t += 32 * SL_WARPS) s_u[t] = atoms[t0 + t];
    __syncthreads();
    if (i0 >= n) continue;
    for (int k0 = 0; k0 < tn; k0 += 32) {
      const int j = t0 + k0 + lane;
      const bool there = k0 + lane < tn;
      const uint4 v = s_u[min(k0 + lane, tn - 1)];
      float d2[SL_C];
      bool odd = false;
#pragma unroll
      for (int q = 0; q < SL_C; ++q) {
        const float dx = (float)(int)(v.x - u[q].x) * sc.w[0],
                    dy = (float)(int)(v.y - u[q].y) * sc.w[1],
                    dz = (float)(int)(v.z - u[q].z) * sc.w[2];
        d2[q] = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        // either guard band (written as two subtractions: fewer predicates)
        odd |= fabsf(d2[q] - sc.cut_mid) <= sc.cut_half;
        if (SPLIT) odd |= fabsf(d2[q] - sc.near_mid) <= sc.near_half;
      }
      const bool settle = __any_sync(0xffffffffu, odd & there);
#pragma unroll
      for (int q = 0; q < SL_C; ++q) {
        const int i = i0 + q;
        bool in = d2[q] < sc.cut.lo, bk = SPLIT & (d2[q] >= sc.near.hi);
        if (settle && there && i < n) {
          const bool c = d2[q] >= sc.cut.lo && d2[q] < sc.cut.hi,
                     f = SPLIT && d2[q] >= sc.near.lo && d2[q] < sc.near.hi;
          if (c || f) {
            const double r2 = dist2_list(b, x[i], y[i], z[i], x[j], y[j], z[j]);
            if (c) in = r2 < sc.cut2;
            if (f) bk = !(r2 < sc.near2);
          }
        }
        in = in & there & (j != i) & (i < n);
        bk = bk & in;
        const unsigned mb = SPLIT ? __ballot_sync(0xffffffffu, bk) : 0u;
        const unsigned mf = __ballot_sync(0xffffffffu, in) ^ mb;
        const int pos = (bk ? nb[q] : nf[q]) + __popc((bk ? mb : mf) & lt);
        store_if(in & (pos < cap), row + (q * cap + (bk ? cap - 1 - pos : pos)), j);
        nb[q] += __popc(mb);
        nf[q] += __popc(mf);
      }
    }
  }
  int sum = 0;
#pragma unroll
  for (int q = 0; q < SL_C; ++q) {
    if (i0 + q >= n) continue;
    sum += nf[q] + nb[q];
    if (lane == q) {
      count[i0 + q] = nf[q] + nb[q];
      if (SPLIT) far[i0 + q] = nb[q];
      if (nf[q] + nb[q] > cap) atomicOr(overflow, 1);
    }
  }
  if (total && lane == 0 && sum) atomicAdd((unsigned long long*)total, (unsigned long long)sum);
}

int launch_full_list_small(const DBox& b, double cutoff, int n, const uint4* atoms,
                           const double* x, const double* y, const double* z, int cap,
                           int* count, int* nbrs, int* overflow, cudaStream_t st,
                           const FarSplit* split, long long* total) {
  if (n <= 0) return RBX_OK;
  // the fixed-point screen's guard band in r^2 (see PairParams' screens):
  // quantisation below 6 s |d| and FP32 rounding below 2e-6 relative, several
  // times both
  double L = 0.0;
  for (int d = 0; d < 3; ++d) L = fmax(L, b.len[d]);
  const double qerr = 64.0 * (L / 4294967296.0) * (cutoff + 1.0);
  SmallScreen sc;
  sc.cut2 = cutoff * cutoff;
  sc.cut = make_screen(sc.cut2, L, 1e-4 + 8e-6 * sc.cut2 + qerr);
  // the near threshold is raised by 1e-9 relative: FP64 rounding never moves a
  // pair that could come within r_core before the next rebuild to the far segment
  sc.near2 = split ? split->r_near * split->r_near * (1.0 + 1e-9) : 0.0;
  sc.near = make_screen(sc.near2, L, 1e-4 + 8e-6 * sc.near2 + qerr);
  // a little wider than the bands, which decide
  auto around = [](const IntScreen& s, float* mid, float* half) {
    *mid = 0.5f * (s.lo + s.hi);
    *half = 0.5f * (s.hi - s.lo) + 1e-6f * s.hi;
  };
  around(sc.cut, &sc.cut_mid, &sc.cut_half);
  around(sc.near, &sc.near_mid, &sc.near_half);
  for (int d = 0; d < 3; ++d) sc.w[d] = (float)(b.len[d] / L);
  const int per_block = SL_WARPS * SL_C;
  const auto kern = split ? k_full_list_small<true> : k_full_list_small<false>;
  kern<<<(n + per_block - 1) / per_block, 32 * SL_WARPS, 0, st>>>(
      b, sc, n, atoms, x, y, z, cap, count, nbrs, overflow, split ? split->far : nullptr,
      total);
  count_launch();
  return check_launch("full_list_small");
}

// ---------------------------------------------------------------------------
// Gathers / scatters and integration.
// ---------------------------------------------------------------------------
__global__ void k_fill_i32(int n, int* __restrict__ p, int v) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = v;
}

// Zero the cell counts; with book (an engine rebuild), also its flags and
// candidate total, and count the rebuild.
__global__ void k_cells_reset(int ncell, int* __restrict__ counts, RebuildBook book) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ncell; i += gridDim.x * blockDim.x)
    counts[i] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (book.flags) book.flags[0] = book.flags[1] = 0;
    if (book.total) *book.total = 0;
    if (book.counter) *book.counter += 1;
  }
}

// One pass over a set of per-atom arrays: dst[a][i] = src[a][perm[i]] (perm
// null: a plain copy).  The set's pointers are kernel parameters, so one
// launch moves every array of the rebuild.
__global__ void k_move_set(int n, const int* __restrict__ perm, ArraySet s) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int p = perm ? perm[i] : i;
#pragma unroll
  for (int a = 0; a < ArraySet::kMaxF64; ++a)
    if (a < s.nf64) s.dst_f64[a][i] = s.src_f64[a][p];
#pragma unroll
  for (int a = 0; a < ArraySet::kMaxI32; ++a)
    if (a < s.ni32) s.dst_i32[a][i] = s.src_i32[a][p];
#pragma unroll
  for (int a = 0; a < ArraySet::kMaxU64; ++a)
    if (a < s.nu64) s.dst_u64[a][i] = s.src_u64[a][p];
}

// Per-step decision inside the step graph: advance the device epoch and take
// the rebuild branch when some atom moved more than skin / 2 since the last
// rebuild (max_d2 holds the bits of a non-negative double).
__global__ void k_step_decide(const unsigned long long* __restrict__ max_d2, double thr2,
                              int* __restrict__ epoch, cudaGraphConditionalHandle rebuild) {
  *epoch += 1;
  cudaGraphSetConditional(rebuild, __longlong_as_double((long long)*max_d2) > thr2 ? 1u : 0u);
}

__global__ void k_zero_u64(unsigned long long* __restrict__ p) { *p = 0ULL; }

__global__ void k_add_i32(int* __restrict__ p, int v) { *p += v; }

template <typename T>
__global__ void k_gather(int n, const int* __restrict__ perm, const T* __restrict__ src,
                         T* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[perm[i]];
}
template <typename T>
__global__ void k_scatter(int n, const int* __restrict__ idx, const T* __restrict__ src,
                          T* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[idx[i]] = src[i];
}

// UpdateVelocity (update_velocity_op.hip.cu:5-28), fmt2v folded into inv_mass.
__global__ void k_kick(int n, const double* __restrict__ fx, const double* __restrict__ fy,
                       const double* __restrict__ fz, const int* __restrict__ type,
                       const double* __restrict__ inv_mass, double half_dt,
                       double* __restrict__ vx, double* __restrict__ vy,
                       double* __restrict__ vz) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double s = inv_mass[type[i]] * half_dt;
  vx[i] += fx[i] * s;
  vy[i] += fy[i] * s;
  vz[i] += fz[i] * s;
}

// UpdatePositionFlag + ApplyPBC (update_position_op.hip.cu:22-46, box.h:133-169),
// fused with the skin check DisplacementSq (base_neighbor_list_builder.cpp:102-116)
// and, for the mixed form, the fixed-point record {ux, uy, uz, q_f32}.  With
// kick.fx the first half kick of the step comes first (k_kick's arithmetic).
// With decide.ctr (inside a step graph) the last block to finish takes the
// step's rebuild decision as k_step_decide does, then clears the maximum and
// the block counter for the next step.
struct DriftArgs {
  DBox b;
  int n;
  double dt;
  double *x, *y, *z, *vx, *vy, *vz;
  const double *x0, *y0, *z0;
  unsigned long long* max_d2;
  uint4* atoms;
  const double* q;
  ImageRefs img;
  Pos3 old;
  KickArgs kick;
  DecideArgs decide;
};

// Block bx of a grid of gx blocks.
__device__ __forceinline__ void drift_body(const DriftArgs& A, int bx, int gx) {
  const DBox& b = A.b;
  const int n = A.n;
  const double dt = A.dt;
  double* __restrict__ x = A.x;
  double* __restrict__ y = A.y;
  double* __restrict__ z = A.z;
  double* __restrict__ vx = A.vx;
  double* __restrict__ vy = A.vy;
  double* __restrict__ vz = A.vz;
  const double* __restrict__ x0 = A.x0;
  const double* __restrict__ y0 = A.y0;
  const double* __restrict__ z0 = A.z0;
  unsigned long long* __restrict__ max_d2 = A.max_d2;
  uint4* __restrict__ atoms = A.atoms;
  const double* __restrict__ q = A.q;
  const ImageRefs& img = A.img;
  const Pos3& old = A.old;
  const KickArgs& kick = A.kick;
  const DecideArgs& decide = A.decide;
  const int i = bx * blockDim.x + threadIdx.x;
  double d2 = 0.0;
  if (i < n) {
    if (old.x) {  // positions before the drift, for SHAKE
      old.x[i] = x[i];
      old.y[i] = y[i];
      old.z[i] = z[i];
    }
    double v[3] = {vx[i], vy[i], vz[i]};
    if (kick.fx) {
      const double s = kick.inv_mass[kick.type[i]] * kick.half_dt;
      v[0] += kick.fx[i] * s;
      v[1] += kick.fy[i] * s;
      v[2] += kick.fz[i] * s;
      vx[i] = v[0];
      vy[i] = v[1];
      vz[i] = v[2];
    }
    double p[3] = {x[i] + v[0] * dt, y[i] + v[1] * dt, z[i] + v[2] * dt};
    for (int d = 0; d < 3; ++d) {  // periodic wrap, counted in the image flags
      int w = 0;
      if (p[d] >= b.lo[d] + b.len[d]) {
        p[d] -= b.len[d];
        w = 1;
      }
      if (p[d] < b.lo[d]) {
        p[d] += b.len[d];
        w = -1;
      }
      if (w && img.c[d]) img.c[d][i] += w;
    }
    x[i] = p[0];
    y[i] = p[1];
    z[i] = p[2];
    if (max_d2) {
      const double ddx = min_image1(p[0] - x0[i], b.len[0], b.half[0]);
      const double ddy = min_image1(p[1] - y0[i], b.len[1], b.half[1]);
      const double ddz = min_image1(p[2] - z0[i], b.len[2], b.half[2]);
      d2 = ddx * ddx + ddy * ddy + ddz * ddz;
    }
    if (atoms) {
      uint4 a;
      a.x = to_fixed(p[0], b.lo[0], 4294967296.0 / b.len[0]);
      a.y = to_fixed(p[1], b.lo[1], 4294967296.0 / b.len[1]);
      a.z = to_fixed(p[2], b.lo[2], 4294967296.0 / b.len[2]);
      a.w = __float_as_uint((float)q[i]);
      atoms[i] = a;
    }
  }
  if (max_d2) {  // block maximum, then one atomic per block
    __shared__ unsigned long long s_max[32];
    unsigned long long bits = (unsigned long long)__double_as_longlong(d2);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long t = __shfl_xor_sync(0xffffffffu, bits, o);
      bits = t > bits ? t : bits;
    }
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = bits;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < (int)(blockDim.x >> 5); ++w) bits = s_max[w] > bits ? s_max[w] : bits;
      atomicMax(max_d2, bits);
    }
  }
  if (decide.ctr) {
    __syncthreads();  // the block's maximum is folded in (by thread 0, below)
    if (threadIdx.x == 0) {
      __threadfence();
      if (atomicAdd(decide.ctr, 1u) == (unsigned)gx - 1) {  // the last block
        __threadfence();
        const unsigned long long m = atomicAdd(max_d2, 0ULL);
        *decide.epoch += 1;
        cudaGraphSetConditional(decide.cond,
                                __longlong_as_double((long long)m) > decide.thr2 ? 1u : 0u);
        *max_d2 = 0ULL;
        *decide.ctr = 0u;
      }
    }
  }
}

__global__ void __launch_bounds__(256) k_drift(DriftArgs a) {
  drift_body(a, blockIdx.x, gridDim.x);
}

__global__ void __launch_bounds__(256)
k_drift_batch(const DriftArgs* __restrict__ a, const int* __restrict__ start, int nrep) {
  const int r = batch_replica(start, nrep, blockIdx.x);
  const int b0 = __ldg(start + r);
  drift_body(a[r], blockIdx.x - b0, __ldg(start + r + 1) - b0);
}

__global__ void k_to_fixed(DBox b, int n, const double* __restrict__ x,
                           const double* __restrict__ y, const double* __restrict__ z,
                           const double* __restrict__ q, uint4* __restrict__ atoms) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint4 a;
  a.x = to_fixed(x[i], b.lo[0], 4294967296.0 / b.len[0]);
  a.y = to_fixed(y[i], b.lo[1], 4294967296.0 / b.len[1]);
  a.z = to_fixed(z[i], b.lo[2], 4294967296.0 / b.len[2]);
  a.w = __float_as_uint((float)q[i]);
  atoms[i] = a;
}

__global__ void k_max_disp(DBox b, int n, const double* __restrict__ x,
                           const double* __restrict__ y, const double* __restrict__ z,
                           const double* __restrict__ x0, const double* __restrict__ y0,
                           const double* __restrict__ z0, unsigned long long* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double d2 = 0.0;
  if (i < n) {
    double dx = x[i] - x0[i], dy = y[i] - y0[i], dz = z[i] - z0[i];
    // MinImageDistance_while (box.h:75-97) as one bounded step: the nearest
    // image by rint, so a non-finite coordinate cannot spin the loop.
    dx -= b.len[0] * rint(dx / b.len[0]);
    dy -= b.len[1] * rint(dy / b.len[1]);
    dz -= b.len[2] * rint(dz / b.len[2]);
    d2 = dx * dx + dy * dy + dz * dz;
  }
  warp_max_atomic(d2, out);
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
size_t cells_scratch_bytes(int n, int ncell) {
  // counts[ncell] + fill[ncell] + cell[n] + sub[n] + tmp[n], 256-byte aligned pieces
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  return al(sizeof(int) * (size_t)ncell) * 2 + al(sizeof(int) * (size_t)n) * 3;
}

int launch_cells_sort(const DBox& b, const int dims[3], int n, const double* x, const double* y,
                      const double* z, int* perm, int* cell_of_sorted, int* cell_start,
                      void* scratch, int* status, cudaStream_t st, const RebuildBook* book) {
  const int ncell = dims[0] * dims[1] * dims[2];
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  char* p = (char*)scratch;
  int* counts = (int*)p;
  p += al(sizeof(int) * (size_t)ncell);
  int* fill = (int*)p;
  p += al(sizeof(int) * (size_t)ncell);
  int* cell = (int*)p;
  p += al(sizeof(int) * (size_t)n);
  unsigned* sub = (unsigned*)p;
  p += al(sizeof(int) * (size_t)n);
  unsigned* tmp = (unsigned*)p;
  k_cells_reset<<<grid_for(ncell, 256, sm_count() * 4), 256, 0, st>>>(
      ncell, counts, book ? *book : RebuildBook{nullptr, nullptr, nullptr});
  count_launch();
  if (n > 0) {
    CellGeom g;
    for (int d = 0; d < 3; ++d) {
      g.edge[d] = b.len[d] / dims[d];
      g.inv[d] = 1.0 / g.edge[d];
    }
    k_cell_assign<<<(n + 255) / 256, 256, 0, st>>>(b, g, dims[0], dims[1], dims[2], n, x, y, z,
                                                   cell, sub, counts);
    count_launch();
  }
  k_cell_scan<<<1, 1024, 0, st>>>(ncell, counts, cell_start, fill);
  count_launch();
  if (n > 0) {
    k_cell_scatter<<<(n + 255) / 256, 256, 0, st>>>(n, cell, sub, fill, tmp);
    count_launch();
  }
  k_cell_segsort<<<ncell, sort_block(n, ncell), 0, st>>>(
      ncell, n, cell_start, tmp, perm, cell_of_sorted, status);
  count_launch();
  return check_launch("cells_sort");
}

static size_t list_pieces(int n, int ncell, size_t piece[6]) {
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  piece[0] = al(sizeof(float4) * (size_t)n);
  piece[1] = piece[2] = al(sizeof(float4) * full_list_chunks(n, ncell));
  piece[3] = al(sizeof(int) * full_list_groups(n, ncell, ListShape<8>::GROUP));
  piece[4] = list_dilute(n, ncell)
                 ? al(sizeof(int) * full_list_groups(n, ncell, ListShape<1>::GROUP))
                 : 0;
  piece[5] = list_dilute(n, ncell) ? al(sizeof(int) * (1 + (size_t)list_many(n))) : 0;
  return piece[0] + piece[1] + piece[2] + piece[3] + piece[4] + piece[5];
}

size_t full_list_scratch_bytes(int n, int ncell) {
  size_t piece[6];
  return list_pieces(n, ncell, piece);
}

int launch_full_list(const DBox& b, const int dims[3], double cutoff, int n, const double* x,
                     const double* y, const double* z, const int* cell_start, int cap,
                     int* count, int* nbrs, int* overflow, void* scratch, cudaStream_t st,
                     const FarSplit* split, long long* total, const uint4* atoms) {
  const int ncell = dims[0] * dims[1] * dims[2];
  if (n <= 0) return RBX_OK;
  if (dims[0] < 3 || dims[1] < 3 || dims[2] < 3) {
    if (!atoms) {
      set_error("full_list: fewer than three cells along an axis need fixed-point records");
      return RBX_ERR_INVALID;
    }
    return launch_full_list_small(b, cutoff, n, atoms, x, y, z, cap, count, nbrs, overflow, st,
                                  split, total);
  }
  const double cut2 = cutoff * cutoff;
  double emax = 0.0;
  for (int d = 0; d < 3; ++d) emax = fmax(emax, b.len[d] / dims[d]);
  // FP32 screening error of |v|^2 - 2 u.v against C - |u|^2.  u (|u_d| <= e/2)
  // is rounded once relative to its cell's centre.  v (|v_d| <= 3e/2) is rounded
  // once relative to the same centre in split rows, where its value also places
  // the pair in the near or the far segment; in plain rows it is the FP32 sum
  // of the image's offset (e) and of the position relative to its own cell's
  // centre (e/2), read as one word an atom (200,000 atoms: 466 us, 485 with the
  // FP64 positions).  A coordinate of v - u is off by at most 2 or 3.5 e 2^-24,
  // which moves |d|^2 by at most 4 or 7 sqrt(3) r e 2^-24 (e = largest cell
  // edge, r = cutoff); the roundings of |v|^2, the three FMAs, |u|^2 and
  // C - |u|^2 add at most (60 e^2 + 3 r^2) 2^-24.  Pairs within twice that of
  // the cutoff take the FP64 path.
  const double err =
      ((split ? 4.0 : 7.0) * sqrt(3.0) * cutoff * emax + 60.0 * emax * emax + 3.0 * cut2) / 16777216.0;
  const double band = 2.0 * err;
  const float lo_band = (float)(cut2 - band), hi_band = (float)(cut2 + band);
  float cut2_up = (float)cut2;  // rounded up
  if ((double)cut2_up < cut2) cut2_up = nextafterf(cut2_up, INFINITY);
  size_t piece[6];
  list_pieces(n, ncell, piece);
  char* p = (char*)scratch;
  ListTables T;
  T.rel = split ? nullptr : (float4*)p;
  T.lo = (float4*)(p + piece[0]);
  T.hi = (float4*)(p + piece[0] + piece[1]);
  T.group_cell = (int*)(p + piece[0] + piece[1] + piece[2]);
  T.few_cell = piece[4] ? (int*)(p + piece[0] + piece[1] + piece[2] + piece[3]) : nullptr;
  T.many = T.few_cell ? (int*)((char*)T.few_cell + piece[4]) : nullptr;
  // a thread an atom: 32 threads a cell up to some 60 atoms (200,000 atoms of 1 / 16 /
  // 120 a cell: 103 / 9 / 7 us, 128 threads 190 / 15 / 5)
  k_chunk_boxes<<<ncell, n < 60LL * ncell ? 32 : 128, 0, st>>>(b, dims[0], dims[1], dims[2], x, y,
                                                              z, cell_start, T);
  count_launch();
  // far threshold in r^2, raised by the FP32 error of the test value
  const float near2 = split ? (float)(split->r_near * split->r_near + band) : INFINITY;
  const int many = (int)full_list_groups(n, ncell, ListShape<8>::GROUP);
  auto build = [&](auto kern, unsigned blocks, int warps, int smem) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
        cudaSuccess)
      return check_launch("full_list (shared memory)");
    kern<<<blocks, 32 * warps, smem, st>>>(
        b, dims[0], dims[1], dims[2], cut2, cut2_up, lo_band, hi_band, x, y, z, cell_start, T,
        cap, count, nbrs, overflow, near2, split ? split->far : nullptr, total);
    count_launch();
    return check_launch("full_list");
  };
  if (T.few_cell) {
    k_many_groups<<<(many + 255) / 256, 256, 0, st>>>(many, T);
    count_launch();
    const int rc = build(split ? k_full_list<true, 1> : k_full_list<false, 1>,
                         (unsigned)full_list_groups(n, ncell, ListShape<1>::GROUP), 1,
                         (int)sizeof(FullListSmem<1>));
    if (rc) return rc;
  }
  return build(split ? k_full_list<true, 8> : k_full_list<false, 8>,
               (unsigned)(T.few_cell ? std::min(many, list_many(n)) : many), 8,
               (int)sizeof(FullListSmem<8>));
}

// dst[a][idx[i]] = src[a][i] for every array of the set (one launch).
__global__ void k_scatter_set(int n, const int* __restrict__ idx, ArraySet s) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int p = idx[i];
#pragma unroll
  for (int a = 0; a < ArraySet::kMaxF64; ++a)
    if (a < s.nf64) s.dst_f64[a][p] = s.src_f64[a][i];
#pragma unroll
  for (int a = 0; a < ArraySet::kMaxI32; ++a)
    if (a < s.ni32) s.dst_i32[a][p] = s.src_i32[a][i];
#pragma unroll
  for (int a = 0; a < ArraySet::kMaxU64; ++a)
    if (a < s.nu64) s.dst_u64[a][p] = s.src_u64[a][i];
}

// dst[3 idx[i] + d] = column d at i.
__global__ void k_scatter_rows(int n, const int* __restrict__ idx, const double* __restrict__ a,
                               const double* __restrict__ b, const double* __restrict__ c,
                               double* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double* const p = dst + 3 * (size_t)idx[i];
  p[0] = a[i];
  p[1] = b[i];
  p[2] = c[i];
}

int launch_scatter_rows(int n, const int* idx, const double* a, const double* b, const double* c,
                        double* dst, cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_scatter_rows<<<(n + 255) / 256, 256, 0, st>>>(n, idx, a, b, c, dst);
  count_launch();
  return check_launch("scatter_rows");
}

int launch_scatter_set(int n, const int* idx, const ArraySet& set, cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_scatter_set<<<(n + 255) / 256, 256, 0, st>>>(n, idx, set);
  count_launch();
  return check_launch("scatter_set");
}

int launch_move_set(int n, const int* perm, const ArraySet& set, cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_move_set<<<(n + 255) / 256, 256, 0, st>>>(n, perm, set);
  count_launch();
  return check_launch("move_set");
}

int launch_fill_i32(int n, int* p, int v, cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_fill_i32<<<grid_for(n, 256, sm_count() * 4), 256, 0, st>>>(n, p, v);
  count_launch();
  return check_launch("fill_i32");
}

int launch_zero_u64(unsigned long long* p, cudaStream_t st) {
  k_zero_u64<<<1, 1, 0, st>>>(p);
  count_launch();
  return check_launch("zero_u64");
}

int launch_add_i32(int* p, int v, cudaStream_t st) {
  k_add_i32<<<1, 1, 0, st>>>(p, v);
  count_launch();
  return check_launch("add_i32");
}

int launch_step_decide(const unsigned long long* max_d2, double thr2, int* epoch,
                       cudaGraphConditionalHandle rebuild, cudaStream_t st) {
  k_step_decide<<<1, 1, 0, st>>>(max_d2, thr2, epoch, rebuild);
  count_launch();
  return check_launch("step_decide");
}

int launch_gather_f64(int n, const int* perm, const double* src, double* dst, cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_gather<double><<<(n + 255) / 256, 256, 0, st>>>(n, perm, src, dst);
  count_launch();
  return check_launch("gather_f64");
}
int launch_gather_i32(int n, const int* perm, const int* src, int* dst, cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_gather<int><<<(n + 255) / 256, 256, 0, st>>>(n, perm, src, dst);
  count_launch();
  return check_launch("gather_i32");
}
int launch_gather_u64(int n, const int* perm, const unsigned long long* src,
                      unsigned long long* dst, cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_gather<unsigned long long><<<(n + 255) / 256, 256, 0, st>>>(n, perm, src, dst);
  count_launch();
  return check_launch("gather_u64");
}
int launch_scatter_f64(int n, const int* idx, const double* src, double* dst, cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_scatter<double><<<(n + 255) / 256, 256, 0, st>>>(n, idx, src, dst);
  count_launch();
  return check_launch("scatter_f64");
}
int launch_scatter_i32(int n, const int* idx, const int* src, int* dst, cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_scatter<int><<<(n + 255) / 256, 256, 0, st>>>(n, idx, src, dst);
  count_launch();
  return check_launch("scatter_i32");
}

int launch_kick(int n, const double* fx, const double* fy, const double* fz, const int* type,
                const double* inv_mass, double half_dt, double* vx, double* vy, double* vz,
                cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_kick<<<(n + 255) / 256, 256, 0, st>>>(n, fx, fy, fz, type, inv_mass, half_dt, vx, vy, vz);
  count_launch();
  return check_launch("kick");
}

int launch_drift(const DBox& b, int n, double dt, double* x, double* y, double* z,
                 double* vx, double* vy, double* vz, const double* x0,
                 const double* y0, const double* z0, unsigned long long* max_d2_bits,
                 uint4* atoms, const double* q, ImageRefs img, Pos3 old, cudaStream_t st,
                 const KickArgs* kick, const DecideArgs* decide) {
  if (n <= 0) return RBX_OK;
  DriftArgs a;
  a.b = b;
  a.n = n;
  a.dt = dt;
  a.x = x;
  a.y = y;
  a.z = z;
  a.vx = vx;
  a.vy = vy;
  a.vz = vz;
  a.x0 = x0;
  a.y0 = y0;
  a.z0 = z0;
  a.max_d2 = max_d2_bits;
  a.atoms = atoms;
  a.q = q;
  a.img = img;
  a.old = old;
  a.kick = kick ? *kick : KickArgs{nullptr, nullptr, nullptr, nullptr, nullptr, 0.0};
  a.decide = decide ? *decide : DecideArgs{nullptr, 0.0, nullptr, {}};
  const int grid = (n + 255) / 256;
  if (batch_recorder()) return record_phase(PH_DRIFT, 0, grid, 256, 0, &a, sizeof a);
  k_drift<<<grid, 256, 0, st>>>(a);
  count_launch();
  return check_launch("drift");
}

int launch_drift_batch(const void* args, const int* start, int nrep, int total, cudaStream_t st) {
  k_drift_batch<<<total, 256, 0, st>>>(static_cast<const DriftArgs*>(args), start, nrep);
  count_launch();
  return check_launch("drift_batch");
}

int launch_to_fixed(const DBox& b, int n, const double* x, const double* y, const double* z,
                    const double* q, uint4* atoms, cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_to_fixed<<<(n + 255) / 256, 256, 0, st>>>(b, n, x, y, z, q, atoms);
  count_launch();
  return check_launch("to_fixed");
}

int launch_max_disp(const DBox& b, int n, const double* x, const double* y, const double* z,
                    const double* x0, const double* y0, const double* z0,
                    unsigned long long* max_d2_bits, cudaStream_t st) {
  if (n <= 0) return RBX_OK;
  k_max_disp<<<(n + 255) / 256, 256, 0, st>>>(b, n, x, y, z, x0, y0, z0, max_d2_bits);
  count_launch();
  return check_launch("max_disp");
}

}  // namespace rbx
