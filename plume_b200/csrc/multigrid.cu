// The pressure solve on the device (chadmv/plume src/plume/sim/pressure.py:124-141, multigrid.py:24-147):
// red-black Gauss-Seidel sweeps and multigrid V-cycles, with the reference's update order and arithmetic.
//
// Launch structure of one V-cycle:
//   - each colour of a sweep is one launch, in place (k_colour_rows4, or k_colour_cells for rows that are no multiple
//     of four cells; k_rb_split4 on a top level in colour-split storage);
//   - the residual, its restriction to the coarse level and the zeroing of the coarse pressure are one
//     launch (k_residual_restrict, k_residual_restrict_split);
//   - prolongation is one launch (k_prolong_rows4, k_prolong_add_split8 and k_prolong_add_split4);
//   - between levels of which one does not halve the other, these two are k_restrict_any and k_prolong_any;
//   - the small levels run in one launch (cluster_solve.cu): from the first of at most cluster_max_cells cells
//     down, in the shared memory of a 16-CTA thread-block cluster, the smallest of them (at most 512 cell pairs along z,
//     so up to 1024 cells) in one CTA of it. When that covers the whole hierarchy, all cycles are that one launch;
//   - levels of at least g_tiled_min_cells cells (by default none) sweep by k_rb_sweep instead, one launch a sweep: a tile
//     of 8x8x32 cells and a 2-cell halo in shared memory; red is updated on the tile and a 1-cell shell, then black on the
//     tile, so every value equals the one the two separate colour passes produce. Prolongation is folded into the first
//     such sweep (the tile loads q + prolong(coarse));
//   - the defect-correction solve's cycles, whose coarsest level is swept in double, run the levels of at most
//     2048 cells in one 1024-thread block instead (k_block_solve).
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "cluster_solve.cuh"
#include "stencil_table.cuh"

namespace plume {

constexpr int TILE_I = 8, TILE_J = 8, TILE_K = 32, HALO = 2;
constexpr int QI = TILE_I + 2 * HALO, QJ = TILE_J + 2 * HALO, QK = TILE_K + 2 * HALO;  // pressure region
constexpr int RI = TILE_I + 2, RJ = TILE_J + 2, RK = TILE_K + 2;                      // rhs region
constexpr int SWEEP_THREADS = 256;
constexpr int COARSEST_SWEEPS = 20;  // multigrid.py:24-33
constexpr int COARSEST_SWEEPS_PER_CELL = 4;
constexpr int BOTTOM_THREADS = 1024;
constexpr int BOTTOM_MAX_LEVELS = 8;
constexpr long SINGLE_MAX_CELLS = 1024;  // bottom kind 1: larger levels are spread over its 8 CTAs
constexpr int BOTTOM_WARP_PAIRS = 128;  // levels with at most this many cell pairs per colour run on one warp
// Per-level strategy (set by plume_tune_solver): levels of at least g_tiled_min_cells cells sweep in tiles,
// smaller ones one colour per launch; the first level of at most g_bottom_max_cells cells and everything
// below it runs in one launch (coarse_plan).
static long g_tiled_min_cells = 1L << 40;  // measured: per-colour sweeps win while the levels fit in L2
// The bottom: the first level of at most this many cells and all below it (plume_tune_solver's bottom_max_cells). Those of at
// most 512 cell pairs along z (cluster_solve_single) run in one CTA, larger ones in slabs.
static long g_bottom_max_cells = 2048;
// The top level runs in colour-split storage (given caller scratch) when it has at least this many cells
// (plume_tune_split): levels whose q and rhs do not fit in L2. Measured on B200 at 256x384x256, 4 V-cycles: the
// solve takes 3.14 ms split against 3.52 ms natural (colour pass 45.5 against 59.9 us, prolongation 91 against
// 109 us, residual and restriction about 110 against 107 us, plus 0.15 ms of layout conversions per solve); at
// 128x192x128, whose levels fit in L2, split is slower (0.97 against 0.78 ms).
static long g_split_min_cells = 1L << 23;
static int g_bottom_kind = 0;  // 0: levels above the bottom join its launch in a 16-CTA cluster; 1: an 8-CTA cluster from the bottom
// Levels above the bottom join its launch (bottom kind 0) up to this many cells. A colour pass of a level costs a launch
// of its own about 2 us in a graph, and in the cluster 0.6 us and 0.8 us more per 110 thousand cells; where the cluster
// starts below the top level, each cycle also loads and stores its first level (3 us). Measured on B200, 4 cycles, the
// solve with the level at stake in the cluster and as launches of its own:
//   the top level: 40x40x40 200 and 212 us, 48x48x48 228 and 226, 75x33x45 253 and 252; 52x52x52 254 and 236, 48x72x48
//   258 and 235;
//   below it: 32x48x32 275 and 279 us (64x96x64 grid), 500 and 504 (128x192x128); 36x40x36 305 and 296 (72x80x72), 38x38x38
//   684 and 679 (152x152x152), 36x48x36 336 and 322 (72x96x72), 40x60x40 960 and 938 (160x240x160);
//   below it, with overhanging cells: 35x45x39 379 and 354 us (69x90x77), 38x57x46 425 and 389 (75x113x91), 49x49x49 458
//   and 406 (97x97x97). Their limit dates from launched passes that branched on a cell's surroundings (482 us at 75x113x91,
//   455 in the cluster); against the present ones, 6 to 11% faster there, it lies too high.
// PLUME_CLUSTER_MAX_CELLS overrides both limits (for measurements).
static long cluster_max_cells(const PlumeGridInfo& info, bool top) {
  static const long set = [] {
    const char* v = getenv("PLUME_CLUSTER_MAX_CELLS");
    return v ? atol(v) : 0L;
  }();
  if (set) return set;
  const bool overhangs = info.fill_hi[0] != 1.0f || info.fill_hi[1] != 1.0f || info.fill_hi[2] != 1.0f;
  return top || overhangs ? 120000 : 60000;
}
constexpr size_t BOTTOM_MAX_SMEM = 200 * 1024;

// The solve's kernels are launched with programmatic dependent launch: each may be scheduled while the
// previous one drains and waits here, before touching memory, until that one has finished and its writes are
// visible (a no-op when launched without it). Measured on B200: 4% off the 4-cycle solve at 128x192x128
// (0.868 -> 0.833 ms). Triggering the successor early (griddepcontrol.launch_dependents) measured slower: the
// waiting blocks take SM slots from the running kernel.
__device__ __forceinline__ void wait_for_previous_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }


// One full red-black sweep of a tile; with PROLONG the tile first adds the coarse correction
// (prolong_add_kernel, multigrid.py:63-68) to every pressure it loads.
// The sweep reads `q_in` and writes `q_out` (different arrays): a tile's halo belongs to its neighbours, which
// may already have written their cells in the same launch.
template <bool PROLONG, bool UNIFORM>
__global__ void __launch_bounds__(SWEEP_THREADS)
    k_rb_sweep(PlumeGridInfo info, const float* __restrict__ q_in, float* __restrict__ q_out,
               const float* __restrict__ rhs, float relaxation, const float* __restrict__ coarse_q, Dims coarse) {
  wait_for_previous_grid();
  __shared__ float sq[QI * QJ * QK];
  __shared__ float sr[RI * RJ * RK];
  const int n0 = info.dims[0], n1 = info.dims[1], n2 = info.dims[2];
  const int i0 = blockIdx.z * TILE_I, j0 = blockIdx.y * TILE_J, k0 = blockIdx.x * TILE_K;
  const int t = threadIdx.x;
  for (int idx = t; idx < QI * QJ * QK; idx += SWEEP_THREADS) {
    const int a = idx / (QJ * QK), rem = idx - a * (QJ * QK), b = rem / QK, c = rem - b * QK;
    const int gi = i0 - HALO + a, gj = j0 - HALO + b, gk = k0 - HALO + c;
    float value = 0.0f;
    if (gi >= 0 && gi < n0 && gj >= 0 && gj < n1 && gk >= 0 && gk < n2) {
      value = __ldg(q_in + (gi * n1 + gj) * n2 + gk);
      if (PROLONG) value = value + sample_index_space(coarse_q, coarse, prolong_point(gi, gj, gk));
    }
    sq[idx] = value;
  }
  for (int idx = t; idx < RI * RJ * RK; idx += SWEEP_THREADS) {
    const int a = idx / (RJ * RK), rem = idx - a * (RJ * RK), b = rem / RK, c = rem - b * RK;
    const int gi = i0 - 1 + a, gj = j0 - 1 + b, gk = k0 - 1 + c;
    sr[idx] = (gi >= 0 && gi < n0 && gj >= 0 && gj < n1 && gk >= 0 && gk < n2) ? __ldg(rhs + (gi * n1 + gj) * n2 + gk)
                                                                              : 0.0f;
  }
  __syncthreads();
  auto qi = [&](int gi, int gj, int gk) { return ((gi - i0 + HALO) * QJ + (gj - j0 + HALO)) * QK + (gk - k0 + HALO); };
  auto load = [&](int gi, int gj, int gk) { return sq[qi(gi, gj, gk)]; };
  const float ghost = ghost_coupling(info);
  // red (colour 0: i + j + k even) on the tile and its 1-cell shell; one red cell per pair along k
  constexpr int RPK = RK / 2;
  for (int p = t; p < RI * RJ * RPK; p += SWEEP_THREADS) {
    const int a = p / (RJ * RPK), rem = p - a * (RJ * RPK), b = rem / RPK, kp = rem - b * RPK;
    const int gi = i0 - 1 + a, gj = j0 - 1 + b, kbase = k0 - 1 + 2 * kp;
    const int gk = kbase + ((gi + gj + kbase) & 1);
    if (gi < 0 || gi >= n0 || gj < 0 || gj >= n1 || gk < 0 || gk >= n2) continue;
    const int at_q = qi(gi, gj, gk);
    const float r = sr[((gi - i0 + 1) * RJ + (gj - j0 + 1)) * RK + (gk - k0 + 1)];
    float out;
    if (relax_cell(UNIFORM, info, ghost, gi, gj, gk, sq[at_q], r, relaxation, load, out)) sq[at_q] = out;
  }
  __syncthreads();
  // black (colour 1) on the tile
  constexpr int TPK = TILE_K / 2;
  for (int p = t; p < TILE_I * TILE_J * TPK; p += SWEEP_THREADS) {
    const int a = p / (TILE_J * TPK), rem = p - a * (TILE_J * TPK), b = rem / TPK, kp = rem - b * TPK;
    const int gi = i0 + a, gj = j0 + b, kbase = k0 + 2 * kp;
    const int gk = kbase + (((gi + gj + kbase) & 1) ^ 1);
    if (gi >= n0 || gj >= n1 || gk >= n2) continue;
    const int at_q = qi(gi, gj, gk);
    const float r = sr[((gi - i0 + 1) * RJ + (gj - j0 + 1)) * RK + (gk - k0 + 1)];
    float out;
    if (relax_cell(UNIFORM, info, ghost, gi, gj, gk, sq[at_q], r, relaxation, load, out)) sq[at_q] = out;
  }
  __syncthreads();
  for (int idx = t; idx < TILE_I * TILE_J * TILE_K; idx += SWEEP_THREADS) {
    const int a = idx / (TILE_J * TILE_K), rem = idx - a * (TILE_J * TILE_K), b = rem / TILE_K, c = rem - b * TILE_K;
    const int gi = i0 + a, gj = j0 + b, gk = k0 + c;
    if (gi < n0 && gj < n1 && gk < n2) q_out[(gi * n1 + gj) * n2 + gk] = sq[qi(gi, gj, gk)];
  }
}

// ---- levels swept by colour in the natural layout ----------------------------------------------------------------
// One colour of a sweep in place (red_black_sweep_kernel, pressure.py:80-92). A colour reads only the other colour, so
// the in-place update is race-free. The kernels below have no branch over code that does not run: a missing
// neighbour's load goes to the cell's own row and its value is replaced by the 0 that neighbor_sum adds, couplings come
// from the level's class table, quotients are products with double reciprocals.
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

__device__ __forceinline__ float coupled_sum(const ClassStencil& e, float xm, float xp, float ym, float yp, float zm, float zp) {
  return ((((e.c[0] * xm + e.c[1] * xp) + e.c[2] * ym) + e.c[3] * yp) + e.c[4] * zm) + e.c[5] * zp;
}
__device__ __forceinline__ float plain_sum(float xm, float xp, float ym, float yp, float zm, float zp) {
  return ((((xm + xp) + ym) + yp) + zm) + zp;
}

// One cell per thread, rows of any length.
template <bool UNIFORM>
__global__ void k_colour_cells(const __grid_constant__ LevelTable t, Dims d, float* q, const float* __restrict__ rhs,
                               int color, float relaxation) {
  wait_for_previous_grid();
  const int i = blockIdx.z, j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = 2 * (blockIdx.x * blockDim.x + threadIdx.x) + ((i + j + color) & 1);
  if (j >= d.n1 || k >= d.n2) return;
  const int plane = d.n1 * d.n2, at_c = at(d, i, j, k);
  const bool x0 = i > 0, x1 = i < d.n0 - 1, y0 = j > 0, y1 = j < d.n1 - 1, z0 = k > 0, z1 = k < d.n2 - 1;
  const float vxm = q[x0 ? at_c - plane : at_c], vxp = q[x1 ? at_c + plane : at_c];
  const float vym = q[y0 ? at_c - d.n2 : at_c], vyp = q[y1 ? at_c + d.n2 : at_c];
  const float vzm = q[z0 ? at_c - 1 : at_c], vzp = q[z1 ? at_c + 1 : at_c];
  const float xm = x0 ? vxm : 0.0f, xp = x1 ? vxp : 0.0f, ym = y0 ? vym : 0.0f, yp = y1 ? vyp : 0.0f;
  const float zm = z0 ? vzm : 0.0f, zp = z1 ? vzp : 0.0f;
  const float own = q[at_c], r = __ldg(rhs + at_c);
  const ClassStencil& e = t.e[16 * class_of(i, d.n0) + 4 * class_of(j, d.n1) + class_of(k, d.n2)];
  const float sq = UNIFORM ? plain_sum(xm, xp, ym, yp, zm, zp) : coupled_sum(e, xm, xp, ym, yp, zm, zp);
  const float value = own + relaxation * (quotient(sq - e.vc * r, e.inv) - own);
  q[at_c] = UNIFORM || e.sc != 0.0f ? value : own;  // a cell with no coupling at all (a level of one cell) is left alone
}

// Four consecutive cells of a row per thread, two of them of the colour: 16-byte loads of the row, of its four
// neighbouring rows and of rhs, and the one value beyond the four that the row's parity needs. The other colour's two
// values are stored back unchanged: this pass never writes them, so any thread reading them sees the same floats. Rows
// of a multiple of four cells, 16-byte-aligned arrays. Measured on B200 at 128x192x128, one pass cold: 7.8 us; with the
// row-interior and boundary cases as branches and the division by six behind a range test 9.9 us.
template <bool UNIFORM>
__global__ void k_colour_rows4(const __grid_constant__ LevelTable t, Dims d, float* __restrict__ q,
                               const float* __restrict__ rhs, int color, float relaxation) {
  wait_for_previous_grid();
  const int i = blockIdx.z, j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (j >= d.n1 || k0 >= d.n2) return;
  const bool odd = (i + j + color) & 1;  // this colour's cells: k0 + odd and k0 + odd + 2
  const int plane = d.n1 * d.n2, row = (i * d.n1 + j) * d.n2 + k0;
  const bool x0 = i > 0, x1 = i < d.n0 - 1, y0 = j > 0, y1 = j < d.n1 - 1;
  const float4 c = ld4(q + row), r = ldg4(rhs + row);
  const float4 xm = ld4(q + (x0 ? row - plane : row)), xp = ld4(q + (x1 ? row + plane : row));
  const float4 ym = ld4(q + (y0 ? row - d.n2 : row)), yp = ld4(q + (y1 ? row + d.n2 : row));
  const int beyond = odd ? k0 + 4 : k0 - 1;
  const bool has_far = beyond >= 0 && beyond < d.n2;
  const float far_value = q[row + (has_far ? beyond - k0 : 0)], far = has_far ? far_value : 0.0f;
  auto pick = [&](const float4& v, int n) { return n == 0 ? (odd ? v.y : v.x) : (odd ? v.w : v.z); };
  const float o0 = odd ? c.x : c.y, o1 = odd ? c.z : c.w;  // the other colour's two
  const ClassStencil* table = t.e + 16 * class_of(i, d.n0) + 4 * class_of(j, d.n1);
  float out[2];
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const int k = k0 + (odd ? 1 : 0) + 2 * n;
    const float a = x0 ? pick(xm, n) : 0.0f, b = x1 ? pick(xp, n) : 0.0f;
    const float e0 = y0 ? pick(ym, n) : 0.0f, e1 = y1 ? pick(yp, n) : 0.0f;
    const float zm = n == 0 ? (odd ? o0 : far) : (odd ? o1 : o0), zp = n == 0 ? (odd ? o1 : o0) : (odd ? far : o1);
    const ClassStencil& e = table[class_of(k, d.n2)];
    const float sq = UNIFORM ? plain_sum(a, b, e0, e1, zm, zp) : coupled_sum(e, a, b, e0, e1, zm, zp);
    const float own = pick(c, n);
    out[n] = own + relaxation * (quotient(sq - e.vc * pick(r, n), e.inv) - own);
  }
  *reinterpret_cast<float4*>(q + row) = odd ? make_float4(c.x, out[0], c.z, out[1]) : make_float4(out[0], c.y, out[1], c.w);
}

// Four consecutive cells k0 .. k0 + 3 of a row (p: the cell k0): one 16-byte load where rows hold a multiple of four
// cells and arrays are aligned (WIDE), else four 4-byte loads, with 0 beyond the row's end.
struct Quad {
  float v[4];
  __device__ __forceinline__ Quad() {}
  __device__ __forceinline__ Quad(float4 a) : v{a.x, a.y, a.z, a.w} {}
};

template <bool WIDE>
__device__ __forceinline__ Quad load_quad(const float* p, int k0, int n2) {
  if constexpr (WIDE) return Quad(ldg4(p));
  Quad r;
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const bool there = k0 + n < n2;
    const float value = __ldg(p + (there ? n : 0));
    r.v[n] = there ? value : 0.0f;
  }
  return r;
}

__device__ __forceinline__ Quad where(bool there, const Quad& a) {
  Quad r;
#pragma unroll
  for (int n = 0; n < 4; ++n) r.v[n] = there ? a.v[n] : 0.0f;
  return r;
}

// prolong_add_kernel (multigrid.py:63-68), four consecutive cells k0 .. k0 + 3 of a row per thread: they
// share the coarse sample's x and y axes, and along z they read the coarse columns m - 1 .. m + 2 (m = k0 / 2, clamped),
// each blended in x then y once. Cell k0 + n sits at coarse z = m - 0.25, m + 0.25, m + 0.75, m + 1.25: exact weights,
// except where the clamp gives the first or the last column the weight 1 (k = 0, and k = n2 - 1 of an even n2). Every
// operation is sample_index_space's. Measured on B200 at 128x192x128, cold: 8.3 us against 16.2 us with one cell per
// thread.
template <bool WIDE>
__global__ void k_prolong_rows4(Dims coarse, Dims fine, const float* __restrict__ cq, float* __restrict__ q) {
  wait_for_previous_grid();
  const int i = blockIdx.z, j = blockIdx.y * blockDim.y + threadIdx.y, k0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (j >= fine.n1 || k0 >= fine.n2) return;
  const F3 g = prolong_point(i, j, 0);
  const Axis1 x = axis_of(g[0], coarse.n0, coarse.n1 * coarse.n2), y = axis_of(g[1], coarse.n1, coarse.n2);
  const int m = k0 / 2, end = coarse.n2 - 1 - m;  // the last column, from column m
  const float* base = cq + (x.i0 * coarse.n1 + y.i0) * coarse.n2 + m;
  const float* rows[4] = {base, base + x.step, base + y.step, base + x.step + y.step};
  float* const row = q + at(fine, i, j, k0);
  Quad own;
  if constexpr (WIDE) {
    own = Quad(ld4(row));
  } else {
#pragma unroll
    for (int n = 0; n < 4; ++n) own.v[n] = row[k0 + n < fine.n2 ? n : 0];
  }
  float c[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    c[r][0] = __ldg(rows[r] + (k0 == 0 ? 0 : -1));
    if constexpr (WIDE) {
      const float2 mid = __ldg(reinterpret_cast<const float2*>(rows[r]));
      c[r][1] = mid.x;
      c[r][2] = mid.y;
    } else {
      c[r][1] = __ldg(rows[r]);
      c[r][2] = __ldg(rows[r] + imin_(1, end));
    }
    c[r][3] = __ldg(rows[r] + imin_(2, end));
  }
  float e[4];
#pragma unroll
  for (int o = 0; o < 4; ++o) e[o] = lerp_w(lerp_w(c[0][o], c[1][o], x), lerp_w(c[2][o], c[3][o], x), y);
  const bool front = k0 == 0;
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    // columns (n + 1) / 2 and (n + 1) / 2 + 1 of e, weights 0.25 and 0.75 or 0.75 and 0.25; at a clamp the first two
    // columns, or the last one twice, with weights 1 and 0
    const int lo = (n + 1) / 2;
    const bool first = n == 0 && front, last = (n & 1) && m + n / 2 >= coarse.n2 - 1, clamped = first || last;
    const float a = first ? e[1] : e[lo], b = first ? e[2] : (last ? e[lo] : e[lo + 1]);
    own.v[n] = own.v[n] + (a * (clamped ? 1.0f : (n & 1 ? 0.75f : 0.25f)) + b * (clamped ? 0.0f : (n & 1 ? 0.25f : 0.75f)));
  }
  if constexpr (WIDE) {
    *reinterpret_cast<float4*>(row) = make_float4(own.v[0], own.v[1], own.v[2], own.v[3]);
  } else {
#pragma unroll
    for (int n = 0; n < 4; ++n)
      if (k0 + n < fine.n2) row[n] = own.v[n];
  }
}

// residual_kernel + restrict_kernel (multigrid.py:36-60) + coarse.q.zero_() (:143): each coarse cell averages the
// residuals of its (up to 8) children, summed in the reference's child order. Two coarse cells per thread: the children
// are four consecutive cells k0 .. k0 + 3 of two rows in two planes, loaded as rows with the eight rows around them.
// Measured on B200 at 128x192x128, cold: 10.0 us against 17.7 us with one coarse cell per thread.
template <bool UNIFORM, bool WIDE>
__global__ void k_residual_restrict(const __grid_constant__ LevelTable t, Dims fd, const float* __restrict__ q,
                                    const float* __restrict__ rhs, Dims coarse, float* __restrict__ coarse_rhs,
                                    float* __restrict__ coarse_q) {
  wait_for_previous_grid();
  const int i = blockIdx.z, j = blockIdx.y * blockDim.y + threadIdx.y, k0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (j >= coarse.n1 || k0 >= fd.n2) return;
  const int plane = fd.n1 * fd.n2;
  const bool two_i = 2 * i + 1 < fd.n0, two_j = 2 * j + 1 < fd.n1, front = k0 == 0, back = k0 + 4 >= fd.n2;
  const int corner = at(fd, 2 * i, 2 * j, k0);
  int row[2][2];
  Quad own[2][2];
#pragma unroll
  for (int di = 0; di < 2; ++di)
#pragma unroll
    for (int dj = 0; dj < 2; ++dj) {  // a missing child row: the first one's, its value never used
      row[di][dj] = corner + (di && two_i ? plane : 0) + (dj && two_j ? fd.n2 : 0);
      own[di][dj] = load_quad<WIDE>(q + row[di][dj], k0, fd.n2);
    }
  float total[2] = {0.0f, 0.0f};
#pragma unroll
  for (int di = 0; di < 2; ++di)
#pragma unroll
    for (int dj = 0; dj < 2; ++dj) {
      const int fi = 2 * i + di, fj = 2 * j + dj, c = row[di][dj];
      const bool there = (di == 0 || two_i) && (dj == 0 || two_j);
      const bool x0 = fi > 0, x1 = fi < fd.n0 - 1, y0 = fj > 0, y1 = fj < fd.n1 - 1;
      const bool x_out = di == 0 ? x0 : x1, y_out = dj == 0 ? y0 : y1;  // the rows beyond the children's
      const int x_step = di == 0 ? -plane : plane, y_step = dj == 0 ? -fd.n2 : fd.n2;
      const Quad x_row = where(x_out, load_quad<WIDE>(q + (x_out ? c + x_step : c), k0, fd.n2));
      const Quad y_row = where(y_out, load_quad<WIDE>(q + (y_out ? c + y_step : c), k0, fd.n2));
      const Quad xm = di == 0 ? x_row : own[0][dj], xp = di == 0 ? where(x1, own[1][dj]) : x_row;
      const Quad ym = dj == 0 ? y_row : own[di][0], yp = dj == 0 ? where(y1, own[di][1]) : y_row;
      const float vl = __ldg(q + c + (front ? 0 : -1)), vr = __ldg(q + c + (back ? 0 : 4));
      const float left = front ? 0.0f : vl, right = back ? 0.0f : vr;
      const Quad r = load_quad<WIDE>(rhs + c, k0, fd.n2);
      const ClassStencil* table = t.e + 16 * class_of(imin_(fi, fd.n0 - 1), fd.n0) + 4 * class_of(imin_(fj, fd.n1 - 1), fd.n1);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const float* o = own[di][dj].v;
        const float zm = n == 0 ? left : o[n > 0 ? n - 1 : 0], zp = n == 3 ? right : o[n < 3 ? n + 1 : 3];
        const ClassStencil& e = table[class_of(k0 + n, fd.n2)];
        const float sq = UNIFORM ? plain_sum(xm.v[n], xp.v[n], ym.v[n], yp.v[n], zm, zp)
                                 : coupled_sum(e, xm.v[n], xp.v[n], ym.v[n], yp.v[n], zm, zp);
        const float sum = total[n / 2] + (r.v[n] - quotient(sq - e.sc * o[n], e.inv_vc));
        total[n / 2] = there && (WIDE || k0 + n < fd.n2) ? sum : total[n / 2];
      }
    }
  const float share = (two_i ? 0.5f : 1.0f) * (two_j ? 0.5f : 1.0f);
  const int out = at(coarse, i, j, k0 / 2);
  if constexpr (WIDE) {
    *reinterpret_cast<float2*>(coarse_rhs + out) = make_float2(total[0] * (0.5f * share), total[1] * (0.5f * share));
    *reinterpret_cast<float2*>(coarse_q + out) = make_float2(0.0f, 0.0f);
  } else {
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      if (k0 / 2 + n >= coarse.n2) break;
      coarse_rhs[out + n] = total[n] * (k0 + 2 * n + 1 < fd.n2 ? 0.5f * share : share);  // / 1, 2, 4 or 8: the same float
      coarse_q[out + n] = 0.0f;
    }
  }
}

// Between levels that do not halve (a caller's own hierarchy, such as one that rounds down): residual_kernel + restrict_kernel
// + coarse.q.zero_() and prolong_add_kernel with one cell per thread and every index held to its level, so for any two
// sets of dims. A coarse cell without children takes 0 / 0, as the reference's average does.
__global__ void k_restrict_any(const __grid_constant__ LevelTable t, Dims fd, const float* __restrict__ q,
                               const float* __restrict__ rhs, Dims coarse, float* __restrict__ coarse_rhs,
                               float* __restrict__ coarse_q) {
  wait_for_previous_grid();
  const int i = blockIdx.z, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= coarse.n1 || k >= coarse.n2) return;
  const int plane = fd.n1 * fd.n2;
  float total = 0.0f, count = 0.0f;
#pragma unroll 1
  for (int child = 0; child < 8; ++child) {  // in the reference's order (di, dj, dk)
    const int fi = 2 * i + (child >> 2), fj = 2 * j + (child >> 1 & 1), fk = 2 * k + (child & 1);
    if (fi >= fd.n0 || fj >= fd.n1 || fk >= fd.n2) continue;
    const int c = at(fd, fi, fj, fk);
    const float xm = fi > 0 ? __ldg(q + c - plane) : 0.0f, xp = fi < fd.n0 - 1 ? __ldg(q + c + plane) : 0.0f;
    const float ym = fj > 0 ? __ldg(q + c - fd.n2) : 0.0f, yp = fj < fd.n1 - 1 ? __ldg(q + c + fd.n2) : 0.0f;
    const float zm = fk > 0 ? __ldg(q + c - 1) : 0.0f, zp = fk < fd.n2 - 1 ? __ldg(q + c + 1) : 0.0f;
    const ClassStencil& e = t.e[16 * class_of(fi, fd.n0) + 4 * class_of(fj, fd.n1) + class_of(fk, fd.n2)];
    total = total + (__ldg(rhs + c) - quotient(coupled_sum(e, xm, xp, ym, yp, zm, zp) - e.sc * __ldg(q + c), e.inv_vc));
    count = count + 1.0f;
  }
  const int out = at(coarse, i, j, k);
  coarse_rhs[out] = total / count;
  coarse_q[out] = 0.0f;
}

__global__ void k_prolong_any(Dims coarse, Dims fine, const float* __restrict__ cq, float* __restrict__ q) {
  wait_for_previous_grid();
  const int i = blockIdx.z, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= fine.n1 || k >= fine.n2) return;
  const int c = at(fine, i, j, k);
  q[c] = q[c] + sample_index_space(cq, coarse, prolong_point(i, j, k));
}

// ---- the top level in colour-split storage -----------------------------------------------------------------
// A level larger than L2 is swept from two arrays per quantity, one per colour: cell (i, j, k) of colour
// c = (i + j + k) & 1 sits at ((c * nx + i) * ny + j) * H + (k >> 1), H = (nz + 1) / 2 rounded up to a multiple
// of four. A colour pass then reads and writes whole sectors of the cells it needs (its own q and rhs, the other
// colour's q) instead of sectors shared by both colours. A cell's six face neighbours all sit in the other
// colour's array: its x and y neighbours at the same half index m, one plane (ny * H) or one row (H) away; its
// z neighbours at m - 1 + p and m + p, p = k & 1. The split kernels load whole rows of four half indices and
// hand the natural-layout stencil functions (relax_cell, residual_cell) those values through a loader, so every
// value is the same as in the natural layout.
// natural -> split (to_split) or split -> natural: thread (i, j, m) moves the cells k = 2m and 2m + 1
template <bool TO_SPLIT>
__global__ void k_split_layout(Dims d, int H, const float* __restrict__ in, float* __restrict__ out) {
  wait_for_previous_grid();
  const int i = blockIdx.z, j = blockIdx.y * blockDim.y + threadIdx.y, m = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= d.n1 || m >= H) return;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int k = 2 * m + ((i + j + c) & 1);
    const long s = ((long)(c * d.n0 + i) * d.n1 + j) * H + m;
    if (k < d.n2) {
      const long n = ((long)i * d.n1 + j) * d.n2 + k;
      if (TO_SPLIT) out[s] = in[n];
      else out[n] = in[s];
    } else if (TO_SPLIT) {
      out[s] = 0.0f;  // the padding slot of an odd row
    }
  }
}

// One colour pass with four cells of a row per thread and 16-byte loads: the thread's own q and rhs, the other colour's
// rows one plane and one row away (x and y neighbours, at the same half indices), and the other colour's own row (z
// neighbours) plus the one value beyond the four that the row's parity needs. Rows are padded to a multiple of four; a
// padding slot stays 0, which is also what a missing z neighbour adds. Uniform levels. Measured on B200 at 256x384x256,
// one pass cold: 34.7 us; with separate row-interior and boundary code and the division by six behind a range test
// 36.8 us. Its 176 MB take 27 us at the copy rate.
__global__ void k_rb_split4(const __grid_constant__ LevelTable t, Dims d, int H, float* __restrict__ qs,
                            const float* __restrict__ rs, int color, float relaxation) {
  wait_for_previous_grid();
  const int i = blockIdx.z, j = blockIdx.y * blockDim.y + threadIdx.y;
  const int m0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (j >= d.n1 || m0 >= H) return;
  const bool odd = (i + j + color) & 1;  // cell k = 2 m + odd
  const long plane = (long)d.n1 * H;
  const long own = ((long)(color * d.n0 + i) * d.n1 + j) * H + m0;
  const long oth = ((long)((1 - color) * d.n0 + i) * d.n1 + j) * H + m0;  // not written by this pass
  const bool x0 = i > 0, x1 = i < d.n0 - 1, y0 = j > 0, y1 = j < d.n1 - 1;
  const float4 q4 = ld4(qs + own), r4 = ldg4(rs + own);
  const float4 xm = ldg4(qs + (x0 ? oth - plane : oth)), xp = ldg4(qs + (x1 ? oth + plane : oth));
  const float4 ym = ldg4(qs + (y0 ? oth - H : oth)), yp = ldg4(qs + (y1 ? oth + H : oth));
  const float4 zc = ldg4(qs + oth);
  const bool has_far = odd ? m0 + 4 < H : m0 > 0;
  const float far_value = __ldg(qs + oth + (has_far ? (odd ? 4 : -1) : 0)), far = has_far ? far_value : 0.0f;
  const float qv[4] = {q4.x, q4.y, q4.z, q4.w}, rv[4] = {r4.x, r4.y, r4.z, r4.w};
  const float xa[4] = {xm.x, xm.y, xm.z, xm.w}, xb[4] = {xp.x, xp.y, xp.z, xp.w};
  const float ya[4] = {ym.x, ym.y, ym.z, ym.w}, yb[4] = {yp.x, yp.y, yp.z, yp.w};
  const float zv[4] = {zc.x, zc.y, zc.z, zc.w};
  const ClassStencil* table = t.e + 16 * class_of(i, d.n0) + 4 * class_of(j, d.n1);
  const double inner = table[d.n2 >= 4 ? 1 : 2].inv, first = table[class_of(0, d.n2)].inv, last = table[3].inv;
  const float vc = t.e[0].vc;
  const int cells = (d.n2 + (odd ? 0 : 1)) / 2 - m0;          // how many of the four exist
  const int last_n = (d.n2 & 1) == (odd ? 0 : 1) ? cells - 1 : -1;  // the one at k = n2 - 1, if it has this parity
  float out[4];
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const float zm = odd ? zv[n] : (n == 0 ? far : zv[n > 0 ? n - 1 : 0]);
    const float zp = odd ? (n == 3 ? far : zv[n < 3 ? n + 1 : 3]) : zv[n];
    const float sq = plain_sum(x0 ? xa[n] : 0.0f, x1 ? xb[n] : 0.0f, y0 ? ya[n] : 0.0f, y1 ? yb[n] : 0.0f, zm, zp);
    const double inv = n == last_n ? last : (n == 0 && m0 == 0 && !odd ? first : inner);
    const float value = qv[n] + relaxation * (quotient(sq - vc * rv[n], inv) - qv[n]);
    out[n] = n < cells ? value : qv[n];
  }
  *reinterpret_cast<float4*>(qs + own) = make_float4(out[0], out[1], out[2], out[3]);
}

// k_residual_restrict with the fine level in split storage, four coarse cells kc0 .. kc0 + 3 per thread. The children of
// coarse cell kc sit at half index m = kc in both colours' rows (fk = 2 kc and 2 kc + 1 are one of each colour). The
// thread loads both colours' 16-byte rows of its two by two child rows once: they are each other's x, y and z
// neighbours; around them it loads the rows beyond in x and y and the value beyond the four that an end's z neighbour
// needs. Each coarse cell adds its children in the reference's order (di, dj, dk). Uniform levels. Bound by load latency,
// so by the warps in flight: measured on B200 at 256x384x256, the 4-cycle solve takes 2.223 ms at four blocks of 64
// registers per SM (a few spilled), 2.294 ms at three of 80, 2.298 ms at two; with two coarse cells per thread 2.269 ms
// at best.
__global__ void __launch_bounds__(256, 4)
    k_residual_restrict_split(const __grid_constant__ LevelTable t, Dims fd, int H, const float* __restrict__ qs,
                              const float* __restrict__ rs, Dims coarse, float* __restrict__ coarse_rhs,
                              float* __restrict__ coarse_q) {
  wait_for_previous_grid();
  const int i = blockIdx.z, j = blockIdx.y * blockDim.y + threadIdx.y;
  const int m0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (j >= coarse.n1 || m0 >= coarse.n2) return;
  const long plane = (long)fd.n1 * H, colour = (long)fd.n0 * plane;
  const bool two_i = 2 * i + 1 < fd.n0, two_j = 2 * j + 1 < fd.n1;
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const long corner = (2L * i * fd.n1 + 2 * j) * H + m0;
  // own[di][dj][p]: the child row's cells of parity p along z; (2 i + di + 2 j + dj) & 1 == (di + dj) & 1, so they have
  // the colour (di + dj + p) & 1
  long row[2][2];
  Quad own[2][2][2];
#pragma unroll
  for (int di = 0; di < 2; ++di)
#pragma unroll
    for (int dj = 0; dj < 2; ++dj) {  // a missing child row: the first one's, its value never used
      row[di][dj] = corner + (di && two_i ? plane : 0) + (dj && two_j ? H : 0);
#pragma unroll
      for (int p = 0; p < 2; ++p) own[di][dj][p] = Quad(ldg4(qs + ((di + dj + p) & 1) * colour + row[di][dj]));
    }
  float total[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  const double inv_vc = t.e[0].inv_vc;
  const int front = class_of(0, fd.n2), inner = fd.n2 >= 4 ? 1 : 2, last_m = (fd.n2 - 1) >> 1, last_p = (fd.n2 - 1) & 1;
#pragma unroll
  for (int di = 0; di < 2; ++di)
#pragma unroll
    for (int dj = 0; dj < 2; ++dj) {
      const int fi = 2 * i + di, fj = 2 * j + dj;
      const bool there = (di == 0 || two_i) && (dj == 0 || two_j);
      const bool x0 = fi > 0, x1 = fi < fd.n0 - 1, y0 = fj > 0, y1 = fj < fd.n1 - 1;
      const ClassStencil* table = t.e + 16 * class_of(imin_(fi, fd.n0 - 1), fd.n0) + 4 * class_of(imin_(fj, fd.n1 - 1), fd.n1);
      const float sc_inner = table[inner].sc, sc_front = table[front].sc, sc_last = table[3].sc;
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const long mine = ((di + dj + p) & 1) * colour + row[di][dj], c = ((di + dj + p + 1) & 1) * colour + row[di][dj];
        Quad xm, xp, ym, yp;
        if (di == 0) {
          const float4 v = ldg4(qs + (x0 ? c - plane : c));
          xm = Quad(x0 ? v : zero);
          xp = x1 ? own[1][dj][p] : Quad(zero);  // the same cells one plane on have the other colour
        } else {
          const float4 v = ldg4(qs + (x1 ? c + plane : c));
          xm = own[0][dj][p];
          xp = Quad(x1 ? v : zero);
        }
        if (dj == 0) {
          const float4 v = ldg4(qs + (y0 ? c - H : c));
          ym = Quad(y0 ? v : zero);
          yp = y1 ? own[di][1][p] : Quad(zero);
        } else {
          const float4 v = ldg4(qs + (y1 ? c + H : c));
          ym = own[di][0][p];
          yp = Quad(y1 ? v : zero);
        }
        // z neighbours at m - 1 and m (p = 0) or m and m + 1 (p = 1) of the other parity's row; padding slots hold 0
        const bool has_far = p == 0 ? m0 > 0 : m0 + 4 < H;
        const float far_value = __ldg(qs + c + (has_far ? (p == 0 ? -1 : 4) : 0)), far = has_far ? far_value : 0.0f;
        const Quad r(ldg4(rs + mine));
        const float* o = own[di][dj][1 - p].v;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const float zm = p == 0 ? (n == 0 ? far : o[n > 0 ? n - 1 : 0]) : o[n];
          const float zp = p == 0 ? o[n] : (n == 3 ? far : o[n < 3 ? n + 1 : 3]);
          const float sc = p == last_p && m0 + n == last_m ? sc_last : (p == 0 && n == 0 && m0 == 0 ? sc_front : sc_inner);
          const float sq = plain_sum(xm.v[n], xp.v[n], ym.v[n], yp.v[n], zm, zp);
          const float sum = total[n] + (r.v[n] - quotient(sq - sc * own[di][dj][p].v[n], inv_vc));
          total[n] = there && 2 * (m0 + n) + p < fd.n2 ? sum : total[n];
        }
      }
    }
  const float share = (two_i ? 0.5f : 1.0f) * (two_j ? 0.5f : 1.0f);
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    if (m0 + n >= coarse.n2) break;
    const int out = at(coarse, i, j, m0 + n);
    coarse_rhs[out] = total[n] * (2 * (m0 + n) + 1 < fd.n2 ? 0.5f * share : share);  // / 1, 2, 4 or 8: the same float
    coarse_q[out] = 0.0f;
  }
}

// k_prolong_rows4 with the fine level in split storage, four cells of a row per thread: thread (c, i, j, m0)
// adds to its cells m0 .. m0 + 3 of colour c. The four share the coarse sample's x and y axes; along z they
// read six consecutive coarse columns (m0 - 1 + p .. m0 + 4 + p, clamped), each blended in x then y once
// (sample_index_space's first lerps, which run per column in that order), and each cell blends its two
// columns in z: the same float operations as sample_index_space at prolong_point, with fewer loads and less
// index arithmetic.
__global__ void k_prolong_add_split4(Dims coarse, Dims fine, int H, const float* __restrict__ cq,
                                     float* __restrict__ qs) {
  wait_for_previous_grid();
  const int c = blockIdx.z / fine.n0, i = blockIdx.z - c * fine.n0;
  const int j = blockIdx.y * blockDim.y + threadIdx.y, m0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (j >= fine.n1 || m0 >= H) return;
  const int p = (i + j + c) & 1;  // cell k = 2 m + p
  const F3 g = prolong_point(i, j, 2 * m0 + p);
  const Axis1 x = axis_of(g[0], coarse.n0, coarse.n1 * coarse.n2), y = axis_of(g[1], coarse.n1, coarse.n2);
  const float* base = cq + (x.i0 * coarse.n1 + y.i0) * coarse.n2;
  const int zbase = m0 - 1 + p;
  float e[6];
#pragma unroll
  for (int o = 0; o < 6; ++o) {
    const float* col = base + imin_(imax_(zbase + o, 0), coarse.n2 - 1);
    e[o] = lerp_w(lerp_w(__ldg(col), __ldg(col + x.step), x), lerp_w(__ldg(col + y.step), __ldg(col + x.step + y.step), x),
                  y);
  }
  const long own = ((long)(c * fine.n0 + i) * fine.n1 + j) * H + m0;
  const float4 q4 = ld4(qs + own);
  float out[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const int k = 2 * (m0 + n) + p;
    if (k >= fine.n2) continue;
    const F3 gk = prolong_point(i, j, k);
    const Axis1 z = axis_of(gk[2], coarse.n2, 1);
    const int off = z.i0 - zbase;  // n, or n + 1 where the lower clamp holds the first cell at column 0
    float value;
    if (off == n || off == n + 1) {
      const float lo = off == n ? e[n] : e[n + 1];
      const float hi = z.step == 0 ? lo : (off == n ? e[n + 1] : e[n + 2]);
      value = lerp_w(lo, hi, z);
    } else {
      value = sample_index_space(cq, coarse, gk);
    }
    out[n] = out[n] + value;
  }
  *reinterpret_cast<float4*>(qs + own) = make_float4(out[0], out[1], out[2], out[3]);
}

// k_prolong_add_split4 for both colours of four half indices m0 .. m0 + 3 of a row per thread (eight fine cells
// k = 2 m0 .. 2 m0 + 7), on a coarse level whose rows hold a multiple of four cells. The eight share the coarse
// sample's x and y axes, and along z they read the seven coarse columns m0 - 1 .. m0 + 5 (clamped), fetched
// from each of the four (x, y) rows as one 16-byte load, one 8-byte load and one 4-byte load. Each column is
// blended in x then y once, and each cell blends its two columns in z: sample_index_space's operations at
// prolong_point, as in k_prolong_add_split4.
__device__ __forceinline__ float pick7(const float* e, int o) {
  return o == 0 ? e[0] : o == 1 ? e[1] : o == 2 ? e[2] : o == 3 ? e[3] : o == 4 ? e[4] : o == 5 ? e[5] : e[6];
}

// The z blend of k_prolong_add_split8 for the four cells k = 2 (m0 + n) + P of a row. Cell m of parity P sits at
// coarse z = m - 0.25 (P = 0: columns m - 1 and m, weight 0.75 on m) or m + 0.25 (P = 1: columns m and m + 1,
// weight 0.25 on m + 1); axis_of forms exactly those indices and weights (t = 0.75 or 0.25, 1 - t = 0.25 or
// 0.75, all exact) except where a clamp holds: cell m = 0 of parity 0 and cell m = n2 - 1 of parity 1, which
// take the general blend.
template <int P>
__device__ __forceinline__ void prolong_row(const float* e, float* out, int i, int j, int m0, const Dims& coarse,
                                            const Dims& fine, const float* __restrict__ cq) {
  constexpr float t = P == 0 ? 0.75f : 0.25f, u = P == 0 ? 0.25f : 0.75f;
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const int m = m0 + n, k = 2 * m + P;
    if (k >= fine.n2) continue;
    float value = e[n + P] * u + e[n + P + 1] * t;  // lerp_w(column m - 1 + P, column m + P, z)
    if ((P == 0 && m == 0) || (P == 1 && m == coarse.n2 - 1)) {
      const F3 gk = prolong_point(i, j, k);
      const Axis1 z = axis_of(gk[2], coarse.n2, 1);
      const int off = z.i0 - (m0 - 1);  // the clamped cell's column in e
      if (off >= 0 && off <= 5) {
        const float lo = pick7(e, off);
        value = lerp_w(lo, z.step == 0 ? lo : pick7(e, off + 1), z);
      } else {
        value = sample_index_space(cq, coarse, gk);
      }
    }
    out[n] = out[n] + value;
  }
}

__global__ void k_prolong_add_split8(Dims coarse, Dims fine, int H, const float* __restrict__ cq,
                                     float* __restrict__ qs) {
  wait_for_previous_grid();
  const int i = blockIdx.z, j = blockIdx.y * blockDim.y + threadIdx.y, m0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (j >= fine.n1 || m0 >= H) return;
  const F3 g = prolong_point(i, j, 0);
  const Axis1 x = axis_of(g[0], coarse.n0, coarse.n1 * coarse.n2), y = axis_of(g[1], coarse.n1, coarse.n2);
  const float* base = cq + (x.i0 * coarse.n1 + y.i0) * coarse.n2;
  const float* rows[4] = {base, base + x.step, base + y.step, base + x.step + y.step};
  float c[4][7];  // row r's columns m0 - 1 .. m0 + 5, clamped into the row
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const float4 mid = ldg4(rows[r] + m0);
    const float lo = m0 > 0 ? __ldg(rows[r] + m0 - 1) : mid.x;
    float2 hi;
    if (m0 + 4 < coarse.n2) hi = __ldg(reinterpret_cast<const float2*>(rows[r] + m0 + 4));
    else hi = make_float2(mid.w, mid.w);
    c[r][0] = lo, c[r][1] = mid.x, c[r][2] = mid.y, c[r][3] = mid.z, c[r][4] = mid.w, c[r][5] = hi.x, c[r][6] = hi.y;
  }
  float e[7];
#pragma unroll
  for (int o = 0; o < 7; ++o) e[o] = lerp_w(lerp_w(c[0][o], c[1][o], x), lerp_w(c[2][o], c[3][o], x), y);
#pragma unroll
  for (int col = 0; col < 2; ++col) {
    const int p = (i + j + col) & 1;  // cell k = 2 m + p
    const long own = ((long)(col * fine.n0 + i) * fine.n1 + j) * H + m0;
    const float4 q4 = ld4(qs + own);
    float out[4] = {q4.x, q4.y, q4.z, q4.w};
    if (p == 0) prolong_row<0>(e, out, i, j, m0, coarse, fine, cq);
    else prolong_row<1>(e, out, i, j, m0, coarse, fine, cq);
    *reinterpret_cast<float4*>(qs + own) = make_float4(out[0], out[1], out[2], out[3]);
  }
}

// ---- the one-block coarse solve with the coarsest level in double (the defect-correction solve's cycles) ----

struct BlockArgs {
  int count;
  int sweeps;
  PlumeLevel lv[BOTTOM_MAX_LEVELS];
  int offset[BOTTOM_MAX_LEVELS];
  int coef_offset[BOTTOM_MAX_LEVELS];  // a level with overhanging cells: its CellCoef table's float offset (else -1)
  int f64_offset;  // the coarsest level's double copy, from this float offset
};

// The stencil of one cell of a level with overhanging cells (fill_hi < 1), as neighbor_sum and relaxed compute
// it: the six couplings in neighbor_sum's order (x-, x+, y-, y+, z-, z+; a ghost's coupling, or 0 for a closed
// face, where the neighbour is outside the level), their sum sc added in that order, and the source scale
// vc = (cell_volume * cell_m) * cell_m. The one-block solve builds these once per launch for its non-uniform
// levels, so each sweep's update is loads, products and sums, without neighbor_sum's seven divisions.
struct CellCoef {
  float c[6];
  float sc, vc;
};

__device__ __forceinline__ CellCoef cell_coef(const PlumeGridInfo& info, int i, int j, int k) {
  const int c[3] = {i, j, k};
  CellCoef out;
  float sc = 0.0f;
#pragma unroll
  for (int axis = 0; axis < 3; ++axis) {
    float area = 1.0f;
#pragma unroll
    for (int other = 0; other < 3; ++other)
      if (other != axis) area = area * cell_fill(info, other, c[other]);
    const float own = cell_fill(info, axis, c[axis]);
    float tc[2];
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const int step = side == 0 ? -1 : 1;
      const int n = c[axis] + step;
      if (n >= 0 && n < info.dims[axis]) tc[side] = area / (0.5f * (own + cell_fill(info, axis, n)));
      else if ((step < 0 && info.open_lo[axis] == 1) || (step > 0 && info.open_hi[axis] == 1))
        tc[side] = area / (0.5f * own + info.ghost_gap);
      else tc[side] = 0.0f;
      out.c[2 * axis + side] = tc[side];
    }
    sc = (sc + tc[0]) + tc[1];
  }
  out.sc = sc;
  out.vc = cell_volume(info, i, j, k) * info.cell_m * info.cell_m;
  return out;
}

// neighbor_sum's sq from a cell's table entry: the in-level neighbours' coupling * pressure, 0 for the rest,
// added in its order.
__device__ __forceinline__ float coef_sum(const CellCoef& e, const float* q, const Dims& d, int i, int j, int k) {
  const int c[3] = {i, j, k}, n[3] = {d.n0, d.n1, d.n2}, stride[3] = {d.n1 * d.n2, d.n2, 1};
  const int own = at(d, i, j, k);
  float sq = 0.0f;
#pragma unroll
  for (int axis = 0; axis < 3; ++axis) {
    const float t0 = c[axis] > 0 ? e.c[2 * axis] * q[own - stride[axis]] : 0.0f;
    const float t1 = c[axis] < n[axis] - 1 ? e.c[2 * axis + 1] * q[own + stride[axis]] : 0.0f;
    sq = (sq + t0) + t1;
  }
  return sq;
}

// The coarsest level's sweeps in double (the defect-correction solve's correction cycles; no reference
// counterpart): q and rhs widened into `dq`/`drhs`, the red-black sweeps of relaxed_f64 over the whole block,
// q rounded back to float.
__device__ __forceinline__ void coarsest_f64(const PlumeGridInfo& info, float* q, const float* rhs, int sweeps,
                                             double relaxation, double* dq, double* drhs) {
  const Dims d = dims_of(info);
  const int n = d.n0 * d.n1 * d.n2;
  for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
    dq[idx] = q[idx];
    drhs[idx] = rhs[idx];
  }
  __syncthreads();
  auto load = [&](int a, int b, int c) { return dq[at(d, a, b, c)]; };
  for (int s = 0; s < sweeps; ++s)
    for (int color = 0; color < 2; ++color) {
      for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
        const int i = idx / (d.n1 * d.n2), r = idx - i * d.n1 * d.n2, j = r / d.n2, k = r - j * d.n2;
        if (((i + j + k) & 1) != color) continue;
        double out;
        if (relaxed_f64(info, i, j, k, dq[idx], drhs[idx], relaxation, load, out)) dq[idx] = out;
      }
      __syncthreads();
    }
  for (int idx = threadIdx.x; idx < n; idx += blockDim.x) q[idx] = (float)dq[idx];
  __syncthreads();
}

// The coarsest level in double when it is not inside the one-block solve: one block, arrays in global memory.
__global__ void __launch_bounds__(BOTTOM_THREADS) k_coarsest_f64(PlumeGridInfo info, float* q, const float* rhs,
                                                                 int sweeps) {
  wait_for_previous_grid();
  extern __shared__ double staged[];
  const int n = info.dims[0] * info.dims[1] * info.dims[2];
  coarsest_f64(info, q, rhs, sweeps, 1.5, staged, staged + n);
}

// Visits the index triples (i, j, c) of p = start, start + stride, ... in an (n0, n1, nc) box without a
// division per step: one division at the start, then the stride's own (di, dj, dc) added with carries.
struct Walk {
  int i, j, c, di, dj, dc, n1, nc;
  __device__ Walk(int start, int stride, int n1_, int nc_) : n1(n1_), nc(nc_) {
    const int plane = n1 * nc;
    i = start / plane;
    int r = start - i * plane;
    j = r / nc;
    c = r - j * nc;
    di = stride / plane;
    r = stride - di * plane;
    dj = r / nc;
    dc = r - dj * nc;
  }
  __device__ __forceinline__ void next() {
    c += dc;
    if (c >= nc) {
      c -= nc;
      ++j;
    }
    j += dj;
    if (j >= n1) {
      j -= n1;
      ++i;
    }
    i += di;
  }
};

// The cells of one colour that a thread updates in the one-block solve, with everything about them that stays
// fixed through a smoothing call held in registers: the cell's and its six neighbours' shared-memory indices
// (16 bits each, 0xffff for a neighbour outside the level), and the coupling total sc and the source term
// (cell_m * cell_m) * rhs of relaxed_uniform. A sweep pass is then seven shared loads, the sums and the update: the same float operations as relaxed_uniform, with
// an interior cell's sum (((((a + b) + c) + d) + e) + f) taken as ((((((0 + a) + b) + c) + d) + e) + f), equal
// in value (0 + a == a up to the sign of a zero).
constexpr int STENCIL_SLOTS = 2;
constexpr unsigned NO_CELL = 0xffffu;

struct StencilSlot {
  unsigned own_and_x0, x1_y0, y1_z0, z1;  // pairs of 16-bit indices
  float sc, source;
};

__device__ __forceinline__ unsigned pack16(unsigned lo, unsigned hi) { return (lo & 0xffffu) | (hi << 16); }

__device__ __forceinline__ StencilSlot stencil_slot(const PlumeGridInfo& info, const Dims& d, float ghost, const float* q,
                                                    const float* rhs, int p, int pairs_k, int color) {
  StencilSlot slot;
  slot.own_and_x0 = NO_CELL;
  const int i = p / (d.n1 * pairs_k), r = p - i * (d.n1 * pairs_k);
  const int j = r / pairs_k, k = 2 * (r - j * pairs_k) + ((i + j + color) & 1);
  if (k >= d.n2) return slot;
  const int c[3] = {i, j, k};
  const int stride[3] = {d.n1 * d.n2, d.n2, 1};
  const int own = at(d, i, j, k);
  unsigned nb[6];
  float sc = 0.0f;
#pragma unroll
  for (int axis = 0; axis < 3; ++axis) {  // neighbor_sum_uniform's couplings, in its order
    float tc0 = 0.0f, tc1 = 0.0f;
    nb[2 * axis] = nb[2 * axis + 1] = NO_CELL;
    if (c[axis] > 0) {
      nb[2 * axis] = own - stride[axis];
      tc0 = 1.0f;
    } else if (info.open_lo[axis] == 1) {
      tc0 = ghost;
    }
    if (c[axis] < info.dims[axis] - 1) {
      nb[2 * axis + 1] = own + stride[axis];
      tc1 = 1.0f;
    } else if (info.open_hi[axis] == 1) {
      tc1 = ghost;
    }
    sc = (sc + tc0) + tc1;
  }
  if (sc == 0.0f) return slot;  // no coupling at all: relaxed_uniform leaves the cell alone
  slot.own_and_x0 = pack16(own, nb[0]);
  slot.x1_y0 = pack16(nb[1], nb[2]);
  slot.y1_z0 = pack16(nb[3], nb[4]);
  slot.z1 = nb[5];
  slot.sc = sc;
  slot.source = info.cell_m * info.cell_m * rhs[own];
  return slot;
}

__device__ __forceinline__ float neighbour16(const float* q, unsigned index) { return index == NO_CELL ? 0.0f : q[index]; }

__device__ __forceinline__ void relax_slot(float* q, const StencilSlot& slot, float relaxation) {
  if ((slot.own_and_x0 & 0xffffu) == NO_CELL) return;
  const float a = neighbour16(q, slot.own_and_x0 >> 16), b = neighbour16(q, slot.x1_y0 & 0xffffu);
  const float c = neighbour16(q, slot.x1_y0 >> 16), e = neighbour16(q, slot.y1_z0 & 0xffffu);
  const float f = neighbour16(q, slot.y1_z0 >> 16), g = neighbour16(q, slot.z1);
  const float sq = (((((0.0f + a) + b) + c) + e) + f) + g;
  const float target = (sq - slot.source) / slot.sc;
  float* own = q + (slot.own_and_x0 & 0xffffu);
  *own = *own + relaxation * (target - *own);
}

// `sweeps` red-black sweeps of a uniform level from register-held stencils: `lanes` threads (one warp or the
// whole block) with at most STENCIL_SLOTS cells of each colour each. Returns false, having done nothing, when
// the level does not fit that.
__device__ __forceinline__ bool stencil_smooth(const PlumeGridInfo& info, float* q, const float* rhs, int sweeps, float relaxation) {
  const Dims d = dims_of(info);
  const int pairs_k = (d.n2 + 1) / 2;
  const int pairs = d.n0 * d.n1 * pairs_k;
  const bool one_warp = pairs <= 32 * STENCIL_SLOTS;
  const int lanes = one_warp ? 32 : BOTTOM_THREADS;
  if (!is_uniform(info) || pairs > lanes * STENCIL_SLOTS || d.n0 * d.n1 * d.n2 >= (int)NO_CELL) return false;
  if (!one_warp || threadIdx.x < 32) {
    const float ghost = ghost_coupling(info);
    StencilSlot slot[2][STENCIL_SLOTS];
#pragma unroll
    for (int color = 0; color < 2; ++color)
#pragma unroll
      for (int n = 0; n < STENCIL_SLOTS; ++n) {
        const int p = threadIdx.x + n * lanes;
        if (p < pairs) slot[color][n] = stencil_slot(info, d, ghost, q, rhs, p, pairs_k, color);
        else slot[color][n].own_and_x0 = NO_CELL;
      }
    for (int s = 0; s < sweeps; ++s)
#pragma unroll
      for (int color = 0; color < 2; ++color) {
#pragma unroll
        for (int n = 0; n < STENCIL_SLOTS; ++n) relax_slot(q, slot[color][n], relaxation);
        if (one_warp) __syncwarp();
        else __syncthreads();
      }
  }
  __syncthreads();
  return true;
}

// block_smooth of a level with overhanging cells from its CellCoef table: relaxed's operations, the couplings
// read from the table. Out of line, so that the uniform levels' register stencils keep their registers.
__device__ __noinline__ void table_smooth(Dims d, float* q, const float* rhs, int sweeps, float relaxation,
                                          const CellCoef* coef) {
  const int pairs_k = (d.n2 + 1) / 2;
  const int pairs = d.n0 * d.n1 * pairs_k;
  const bool one_warp = pairs <= BOTTOM_WARP_PAIRS;
  if (!one_warp || threadIdx.x < 32) {
    for (int s = 0; s < sweeps; ++s)
      for (int color = 0; color < 2; ++color) {
        const int stride = one_warp ? 32 : BOTTOM_THREADS;
        Walk w((int)threadIdx.x, stride, d.n1, pairs_k);
        for (int p = threadIdx.x; p < pairs; p += stride, w.next()) {
          const int i = w.i, j = w.j;
          const int k = 2 * w.c + ((i + j + color) & 1);
          if (k >= d.n2) continue;
          const int idx = at(d, i, j, k);
          const CellCoef& e = coef[idx];
          if (e.sc == 0.0f) continue;
          const float sq = coef_sum(e, q, d, i, j, k);
          const float source = e.vc * rhs[idx];
          const float target = (sq - source) / e.sc;
          q[idx] = q[idx] + relaxation * (target - q[idx]);
        }
        if (one_warp) __syncwarp();
        else __syncthreads();
      }
  }
  __syncthreads();
}

// residual_at of a level with overhanging cells from its CellCoef table.
__device__ __noinline__ float table_residual(const CellCoef* coef, const float* q, const float* rhs, Dims d, int i, int j,
                                             int k) {
  const int f = at(d, i, j, k);
  const CellCoef& e = coef[f];
  return rhs[f] - divide(coef_sum(e, q, d, i, j, k) - e.sc * q[f], divisor(e.vc));
}

__device__ __forceinline__ void block_smooth(const PlumeGridInfo& info, float* q, const float* rhs, int sweeps, float relaxation,
                                             const CellCoef* coef = nullptr) {
  if (coef) return table_smooth(dims_of(info), q, rhs, sweeps, relaxation, coef);
  if (stencil_smooth(info, q, rhs, sweeps, relaxation)) return;
  const Dims d = dims_of(info);
  const int pairs_k = (d.n2 + 1) / 2;
  const int pairs = d.n0 * d.n1 * pairs_k;
  auto load = [&](int a, int b, int c) { return q[at(d, a, b, c)]; };
  const bool uniform = is_uniform(info);
  const float ghost = ghost_coupling(info);
  const bool one_warp = pairs <= BOTTOM_WARP_PAIRS;
  if (!one_warp || threadIdx.x < 32) {
    for (int s = 0; s < sweeps; ++s)
      for (int color = 0; color < 2; ++color) {
        const int stride = one_warp ? 32 : BOTTOM_THREADS;
        Walk w((int)threadIdx.x, stride, d.n1, pairs_k);
        for (int p = threadIdx.x; p < pairs; p += stride, w.next()) {
          const int i = w.i, j = w.j;
          const int k = 2 * w.c + ((i + j + color) & 1);
          if (k >= d.n2) continue;
          const int idx = at(d, i, j, k);
          float out;
          if (relax_cell(uniform, info, ghost, i, j, k, q[idx], rhs[idx], relaxation, load, out)) q[idx] = out;
        }
        if (one_warp) __syncwarp();
        else __syncthreads();
      }
  }
  __syncthreads();
}

// TABLES: some level has overhanging cells (CellCoef tables in b.coef_offset); without, the uniform levels'
// code is compiled alone.
template <bool TABLES>
__global__ void __launch_bounds__(BOTTOM_THREADS) k_block_solve(BlockArgs b) {
  wait_for_previous_grid();
  extern __shared__ float smem[];
  const int t = threadIdx.x;
  {
    const Dims d = dims_of(b.lv[0].info);
    const int n = d.n0 * d.n1 * d.n2;
    float* q = smem + b.offset[0];
    for (int idx = t; idx < n; idx += BOTTOM_THREADS) {
      q[idx] = b.lv[0].q[idx];
      q[n + idx] = b.lv[0].rhs[idx];
    }
  }
  auto coef_of = [&](int l) -> CellCoef* {
    if constexpr (TABLES) return b.coef_offset[l] >= 0 ? reinterpret_cast<CellCoef*>(smem + b.coef_offset[l]) : nullptr;
    else return nullptr;
  };
  for (int l = 0; TABLES && l < b.count; ++l) {
    CellCoef* table = coef_of(l);
    if (!table) continue;
    const Dims d = dims_of(b.lv[l].info);
    Walk w(t, BOTTOM_THREADS, d.n1, d.n2);
    for (int idx = t; idx < d.n0 * d.n1 * d.n2; idx += BOTTOM_THREADS, w.next())
      table[idx] = cell_coef(b.lv[l].info, w.i, w.j, w.c);
  }
  __syncthreads();
  for (int l = 0; l + 1 < b.count; ++l) {
    const PlumeGridInfo& info = b.lv[l].info;
    const Dims fd = dims_of(info), cd = dims_of(b.lv[l + 1].info);
    float* q = smem + b.offset[l];
    float* rhs = q + fd.n0 * fd.n1 * fd.n2;
    float* cq = smem + b.offset[l + 1];
    float* crhs = cq + cd.n0 * cd.n1 * cd.n2;
    const CellCoef* table = coef_of(l);
    block_smooth(info, q, rhs, b.sweeps, 1.0f, table);
    auto load = [&](int a, int bb, int c) { return q[at(fd, a, bb, c)]; };
    const bool uniform = is_uniform(info);
    const float ghost = ghost_coupling(info);
    const int coarse_cells = cd.n0 * cd.n1 * cd.n2;
    Walk w(t, BOTTOM_THREADS, cd.n1, cd.n2);
    for (int idx = t; idx < coarse_cells; idx += BOTTOM_THREADS, w.next()) {
      const int i = w.i, j = w.j, k = w.c;
      float total = 0.0f, count = 0.0f;
      for (int di = 0; di < 2; ++di)
        for (int dj = 0; dj < 2; ++dj)
          for (int dk = 0; dk < 2; ++dk) {
            const int fi = 2 * i + di, fj = 2 * j + dj, fk = 2 * k + dk;
            if (fi < fd.n0 && fj < fd.n1 && fk < fd.n2) {
              const int f = at(fd, fi, fj, fk);
              if (table) {
                total = total + table_residual(table, q, rhs, fd, fi, fj, fk);
              } else {
                total = total + residual_cell(uniform, info, ghost, fi, fj, fk, q[f], rhs[f], load);
              }
              count = count + 1.0f;
            }
          }
      crhs[idx] = total / count;
      cq[idx] = 0.0f;
    }
    __syncthreads();
  }
  {
    const PlumeGridInfo& info = b.lv[b.count - 1].info;
    const Dims d = dims_of(info);
    float* q = smem + b.offset[b.count - 1];
    const int longest = imax_(d.n0, imax_(d.n1, d.n2));
    const int n = d.n0 * d.n1 * d.n2;
    const int sweeps = imax_(COARSEST_SWEEPS, COARSEST_SWEEPS_PER_CELL * longest);
    double* staged = reinterpret_cast<double*>(smem + b.f64_offset);
    coarsest_f64(info, q, q + n, sweeps, 1.5, staged, staged + n);
  }
  for (int l = b.count - 2; l >= 0; --l) {
    const PlumeGridInfo& info = b.lv[l].info;
    const Dims fd = dims_of(info), cd = dims_of(b.lv[l + 1].info);
    float* q = smem + b.offset[l];
    const float* cq = smem + b.offset[l + 1];
    const int n = fd.n0 * fd.n1 * fd.n2;
    Walk w(t, BOTTOM_THREADS, fd.n1, fd.n2);
    for (int idx = t; idx < n; idx += BOTTOM_THREADS, w.next())
      q[idx] = q[idx] + sample_plain(cq, cd, prolong_point(w.i, w.j, w.c));
    __syncthreads();
    block_smooth(info, q, q + n, b.sweeps, 1.0f, coef_of(l));
  }
  for (int l = 0; l < b.count; ++l) {
    const Dims d = dims_of(b.lv[l].info);
    const int n = d.n0 * d.n1 * d.n2;
    const float* q = smem + b.offset[l];
    for (int idx = t; idx < n; idx += BOTTOM_THREADS) {
      b.lv[l].q[idx] = q[idx];
      if (l > 0) b.lv[l].rhs[idx] = q[n + idx];
    }
  }
}

// ---- host side --------------------------------------------------------------------------------------------

static long cells_of(const PlumeGridInfo& info) { return (long)info.dims[0] * info.dims[1] * info.dims[2]; }

static dim3 tile_grid(const PlumeGridInfo& info) {
  return dim3((info.dims[2] + TILE_K - 1) / TILE_K, (info.dims[1] + TILE_J - 1) / TILE_J,
              (info.dims[0] + TILE_I - 1) / TILE_I);
}

static bool pdl_enabled() {
  static const bool enabled = std::getenv("PLUME_B200_NO_PDL") == nullptr;
  return enabled;
}

// Launches a solve kernel, with programmatic dependent launch unless PLUME_B200_NO_PDL is set.
template <class... Params, class... Args>
static int launch_solve_kernel(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                               const char* what, Args... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = st;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = pdl_enabled() ? 1 : 0;
  int status = runtime_status(what, cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...));
  if (status != PLUME_OK) return status;
  return launch_status(what);
}

// A level's pressure lives in two arrays: sweeps alternate between them. `cur` holds the current values.
struct Pressure {
  float* cur;
  float* other;
  void flip() { std::swap(cur, other); }
};

static bool uniform_level(const PlumeGridInfo& info) {
  return info.fill_hi[0] == 1.0f && info.fill_hi[1] == 1.0f && info.fill_hi[2] == 1.0f;
}

template <bool PROLONG>
static void launch_tiled(const PlumeGridInfo& info, Pressure& q, const float* rhs, float relaxation,
                         const float* coarse_q, Dims cd, cudaStream_t st) {
  if (uniform_level(info))
    k_rb_sweep<PROLONG, true><<<tile_grid(info), SWEEP_THREADS, 0, st>>>(info, q.cur, q.other, rhs, relaxation, coarse_q, cd);
  else
    k_rb_sweep<PROLONG, false><<<tile_grid(info), SWEEP_THREADS, 0, st>>>(info, q.cur, q.other, rhs, relaxation, coarse_q, cd);
}

static bool rows4(const Dims& d, const void* a, const void* b) {
  return d.n2 % 4 == 0 && (((uintptr_t)a | (uintptr_t)b) & 15) == 0;
}

static int colour_sweep(const PlumeGridInfo& info, const LevelTable& table, float* q, const float* rhs, float relaxation,
                        cudaStream_t st) {
  const Dims d = dims_of(info);
  const bool uniform = uniform_level(info) && cells_of(info) > 1, wide = rows4(d, q, rhs);
  const dim3 grid(((wide ? d.n2 / 4 : (d.n2 + 1) / 2) + TZ - 1) / TZ, (d.n1 + TY - 1) / TY, d.n0);
  auto kernel = wide ? (uniform ? k_colour_rows4<true> : k_colour_rows4<false>)
                     : (uniform ? k_colour_cells<true> : k_colour_cells<false>);
  for (int color = 0; color < 2; ++color) {
    int status = launch_solve_kernel(kernel, grid, cell_block(), 0, st, "red-black colour", table, d, q, rhs, color, relaxation);
    if (status != PLUME_OK) return status;
  }
  return PLUME_OK;
}

static int launch_restrict(const PlumeGridInfo& info, const LevelTable& table, const float* q, const float* rhs,
                           const PlumeLevel& coarse, cudaStream_t st) {
  const Dims d = dims_of(info), cd = dims_of(coarse.info);
  if (!halves(info, coarse.info))
    return launch_solve_kernel(k_restrict_any, cell_grid(cd.n0, cd.n1, cd.n2), cell_block(), 0, st, "residual and restriction",
                               table, d, q, rhs, cd, coarse.rhs, coarse.q);
  const bool uniform = uniform_level(info);
  const bool wide = rows4(d, q, rhs) && (((uintptr_t)coarse.rhs | (uintptr_t)coarse.q) & 7) == 0;
  const dim3 grid(((d.n2 + 3) / 4 + TZ - 1) / TZ, (cd.n1 + TY - 1) / TY, cd.n0);
  auto kernel = wide ? (uniform ? k_residual_restrict<true, true> : k_residual_restrict<false, true>)
                     : (uniform ? k_residual_restrict<true, false> : k_residual_restrict<false, false>);
  return launch_solve_kernel(kernel, grid, cell_block(), 0, st, "residual and restriction", table, d, q, rhs, cd, coarse.rhs,
                             coarse.q);
}

static int launch_prolong(const PlumeGridInfo& info, float* q, const float* coarse_q, const PlumeGridInfo& coarse,
                          cudaStream_t st) {
  const Dims d = dims_of(info), cd = dims_of(coarse);
  if (!halves(info, coarse))
    return launch_solve_kernel(k_prolong_any, cell_grid(d.n0, d.n1, d.n2), cell_block(), 0, st, "prolong", cd, d, coarse_q, q);
  const bool wide = rows4(d, q, q) && ((uintptr_t)coarse_q & 7) == 0;
  const dim3 grid(((d.n2 + 3) / 4 + TZ - 1) / TZ, (d.n1 + TY - 1) / TY, d.n0);
  return launch_solve_kernel(wide ? k_prolong_rows4<true> : k_prolong_rows4<false>, grid, cell_block(), 0, st, "prolong", cd, d, coarse_q, q);
}

// The split top level's prolongation takes both colours of a row's four half indices per thread when the
// coarse rows hold a multiple of four cells (k_prolong_add_split8); PLUME_PROLONG8=0 keeps k_prolong_add_split4.
// Measured on B200 at 256x384x256, 4 V-cycles: the solve 3.094 -> 3.020 ms, every value unchanged.
static const bool g_prolong8 = [] {
  const char* v = getenv("PLUME_PROLONG8");
  return !(v && v[0] == '0');
}();

// The top level's split arrays: q then rhs, each 2 * nx * ny * H floats.
struct SplitTop {
  float* q;
  float* rhs;
  int H;
};

// Half-row length of the split arrays: (nz + 1) / 2 cells, padded to a multiple of four for 16-byte loads.
static int split_H(const PlumeGridInfo& info) { return ((info.dims[2] + 1) / 2 + 3) / 4 * 4; }

static long split_floats(const PlumeGridInfo& info) {
  return 2L * info.dims[0] * info.dims[1] * split_H(info);
}

static int split_sweeps(const PlumeGridInfo& info, const SplitTop& sp, int sweeps, const float* coarse_q,
                        const PlumeGridInfo* coarse, cudaStream_t st) {
  const Dims d = dims_of(info);
  if (coarse) {
    const Dims cd = dims_of(*coarse);
    const bool rows4 = g_prolong8 && cd.n2 % 4 == 0 && ((uintptr_t)coarse_q & 15) == 0;
    int status = rows4 ? launch_solve_kernel(k_prolong_add_split8, dim3((sp.H / 4 + TZ - 1) / TZ, (d.n1 + TY - 1) / TY, d.n0),
                                             cell_block(), 0, st, "prolong (split)", cd, d, sp.H, coarse_q, sp.q)
                       : launch_solve_kernel(k_prolong_add_split4, dim3((sp.H / 4 + TZ - 1) / TZ, (d.n1 + TY - 1) / TY, 2 * d.n0),
                                             cell_block(), 0, st, "prolong (split)", cd, d, sp.H, coarse_q, sp.q);
    if (status != PLUME_OK) return status;
  }
  const dim3 grid((sp.H / 4 + TZ - 1) / TZ, (d.n1 + TY - 1) / TY, d.n0);
  const LevelTable table = level_table(info);
  for (int s = 0; s < sweeps; ++s)
    for (int color = 0; color < 2; ++color) {
      int status = launch_solve_kernel(k_rb_split4, grid, cell_block(), 0, st, "red-black colour (split)", table, d, sp.H,
                                       sp.q, (const float*)sp.rhs, color, 1.0f);
      if (status != PLUME_OK) return status;
    }
  return PLUME_OK;
}

// `sweeps` full sweeps; when `coarse` is given its correction is prolonged first (folded into the first tiled
// sweep on large levels).
static int sweeps_with_prolong(const PlumeGridInfo& info, Pressure& q, const float* rhs, int sweeps, float relaxation,
                               const float* coarse_q, const PlumeGridInfo* coarse, cudaStream_t st) {
  int s = 0;
  const bool tiled = cells_of(info) >= g_tiled_min_cells;
  const LevelTable table = level_table(info);
  if (coarse) {
    const Dims cd = dims_of(*coarse);
    if (sweeps == 0 || !tiled) {
      int status = launch_prolong(info, q.cur, coarse_q, *coarse, st);
      if (status != PLUME_OK) return status;
    } else {
      launch_tiled<true>(info, q, rhs, relaxation, coarse_q, cd, st);
      int status = launch_status("red-black sweep with prolongation");
      if (status != PLUME_OK) return status;
      q.flip();
      s = 1;
    }
  }
  for (; s < sweeps; ++s) {
    if (tiled) {
      launch_tiled<false>(info, q, rhs, relaxation, nullptr, Dims{1, 1, 1}, st);
      int status = launch_status("red-black sweep");
      if (status != PLUME_OK) return status;
      q.flip();
    } else {
      int status = colour_sweep(info, table, q.cur, rhs, relaxation, st);
      if (status != PLUME_OK) return status;
    }
  }
  return PLUME_OK;
}

static int prepare_bottom();

// Sweeps on `q` with `scratch` as the second array; the result always ends in `q`.
int red_black_sweeps(const PlumeGridInfo& info, float* q, float* scratch, const float* rhs, int sweeps,
                     float relaxation, cudaStream_t st) {
  int status = PLUME_OK;
  if (g_bottom_kind == 0 && g_bottom_max_cells > 0 && cells_of(info) <= cluster_max_cells(info, true) &&
      cells_of(info) < g_tiled_min_cells) {  // every sweep in one launch, the level in shared memory
    if ((status = prepare_bottom()) != PLUME_OK) return status;
    const PlumeLevel level{info, q, const_cast<float*>(rhs), scratch};
    const bool single = cells_of(info) <= g_bottom_max_cells && cluster_solve_single(info);
    const ClusterSolve solve{&level, 1, single ? 0 : 1, single ? 1 : 16, 1, 0, false, false, sweeps, relaxation};
    if (cluster_solve_runs(solve)) return launch_cluster_solve(solve, pdl_enabled(), st);
  }
  Pressure p{q, scratch};
  status = sweeps_with_prolong(info, p, rhs, sweeps, relaxation, nullptr, nullptr, st);
  if (status != PLUME_OK || p.cur == q) return status;
  return runtime_status("pressure copy-back", cudaMemcpyAsync(q, p.cur, sizeof(float) * (size_t)cells_of(info),
                                                              cudaMemcpyDeviceToDevice, st));
}

static size_t f64_staging_offset(size_t float_bytes) { return (float_bytes + 7) / 8 * 8; }

static bool overhangs(const PlumeGridInfo& info) {
  return info.fill_hi[0] != 1.0f || info.fill_hi[1] != 1.0f || info.fill_hi[2] != 1.0f;
}

// The one-block solve's shared memory after its q and rhs arrays (`bytes`): a CellCoef table per level with
// overhanging cells, each from a 16-byte boundary. With `offsets`, the tables' float offsets (-1: none).
static size_t coef_bytes(const PlumeLevel* levels, int count, size_t bytes, int* offsets = nullptr) {
  for (int l = 0; l < count; ++l) {
    if (offsets) offsets[l] = -1;
    if (!overhangs(levels[l].info)) continue;
    bytes = (bytes + 15) / 16 * 16;
    if (offsets) offsets[l] = (int)(bytes / sizeof(float));
    bytes += sizeof(CellCoef) * (size_t)cells_of(levels[l].info);
  }
  return bytes;
}

// Which levels of a hierarchy run in one launch: from `start` down (count: none), those from `single_from` on in one
// CTA, with `ctas` CTAs for the levels between, or (coarse_f64) in one block of k_block_solve with `smem` bytes.
struct CoarsePlan {
  int start, single_from, ctas;
  size_t smem;
  bool store_all = true;  // this cycle is the solve's last: the coarser levels' arrays are left as it has them
};

static int coarsest_sweeps(const PlumeGridInfo& info) {
  const int longest = std::max(info.dims[0], std::max(info.dims[1], info.dims[2]));
  return std::max(COARSEST_SWEEPS, COARSEST_SWEEPS_PER_CELL * longest);
}

static ClusterSolve cluster_solve(const PlumeLevel* levels, int count, const CoarsePlan& plan, int cycles, int sweeps,
                                  bool store_all) {
  return ClusterSolve{levels + plan.start, count - plan.start, plan.single_from - plan.start, plan.ctas,
                      cycles, sweeps, plan.start > 0, store_all, coarsest_sweeps(levels[count - 1].info), 1.5f};
}

// `first_level`: the levels before it are not to be part of the launch.
static CoarsePlan coarse_plan(const PlumeLevel* levels, int count, int coarse_f64, int first_level) {
  CoarsePlan plan{count, count, 1, 0};
  for (int first = first_level; first < count && plan.start == count; ++first) {
    if (count - first > BOTTOM_MAX_LEVELS || cells_of(levels[first].info) > g_bottom_max_cells) continue;
    if (coarse_f64) {
      size_t bytes = 0;
      for (int l = first; l < count; ++l) bytes += 2 * sizeof(float) * (size_t)cells_of(levels[l].info);
      bytes = f64_staging_offset(coef_bytes(levels + first, count - first, bytes)) +
              2 * sizeof(double) * (size_t)cells_of(levels[count - 1].info);
      if (bytes <= BOTTOM_MAX_SMEM) plan = CoarsePlan{first, first, 1, bytes};
      continue;
    }
    // the first level of one CTA, the rest above it in slabs; then (kind 0) levels above the bottom join the launch
    const long single_cells = g_bottom_kind == 1 ? std::min(g_bottom_max_cells, SINGLE_MAX_CELLS) : g_bottom_max_cells;
    int single = first;
    while (single < count && (cells_of(levels[single].info) > single_cells || !cluster_solve_single(levels[single].info)))
      ++single;
    for (int top = g_bottom_kind == 1 ? first : first_level; top <= first && plan.start == count; ++top) {
      if (top < first && (cells_of(levels[top].info) > cluster_max_cells(levels[top].info, top == 0) || cells_of(levels[top].info) >= g_tiled_min_cells))
        continue;
      for (int ctas : {16, 8}) {
        const CoarsePlan here{top, single, top >= single ? 1 : (g_bottom_kind == 1 ? 8 : ctas), 0};
        if (plan.start == count && cluster_solve_runs(cluster_solve(levels, count, here, 1, 0, true))) plan = here;
      }
    }
  }
  return plan;
}

// Lets the one-launch solves use their shared memory and cluster size (once per device, outside any capture).
static int prepare_bottom() {
  static std::mutex mutex;
  static bool configured[64] = {};
  int device = 0;
  int status = prepare_cluster_solve();
  if (status != PLUME_OK) return status;
  if ((status = runtime_status("current device", cudaGetDevice(&device))) != PLUME_OK) return status;
  std::lock_guard<std::mutex> lock(mutex);
  if (device >= 0 && device < 64 && !configured[device]) {
    for (auto kernel : {k_block_solve<false>, k_block_solve<true>})
      if (status == PLUME_OK)
        status = runtime_status("coarse solve shared memory",
                                cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     (int)BOTTOM_MAX_SMEM));
    if (status == PLUME_OK)
      status = runtime_status("coarse solve shared memory",
                              cudaFuncSetAttribute(k_coarsest_f64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)BOTTOM_MAX_SMEM));
    if (status != PLUME_OK) return status;
    configured[device] = true;
  }
  return PLUME_OK;
}

static int launch_block_solve(const PlumeLevel* levels, int count, int sweeps, size_t smem, cudaStream_t st) {
  BlockArgs b{};
  b.count = count;
  b.sweeps = sweeps;
  int offset = 0;
  for (int l = 0; l < count; ++l) {
    b.lv[l] = levels[l];
    b.offset[l] = offset;
    offset += 2 * (int)cells_of(levels[l].info);
  }
  const size_t table_end = coef_bytes(levels, count, sizeof(float) * (size_t)offset, b.coef_offset);
  b.f64_offset = (int)(f64_staging_offset(table_end) / sizeof(float));
  bool tables = false;
  for (int l = 0; l < count; ++l) tables = tables || b.coef_offset[l] >= 0;
  return launch_solve_kernel(tables ? k_block_solve<true> : k_block_solve<false>, dim3(1), dim3(BOTTOM_THREADS), smem, st,
                             "coarse-level block solve", b);
}

// One V-cycle below `index` (multigrid.py:130-147). Every level keeps its pressure in q and uses its residual
// array as the sweeps' second array; the residual itself is never stored (k_residual_restrict).
static int v_cycle(const PlumeLevel* levels, int count, int index, Pressure& q, const CoarsePlan& plan, int sweeps,
                   cudaStream_t st, int coarse_f64, const SplitTop* split = nullptr) {
  const PlumeLevel& lv = levels[index];
  if (index == 0 && split) {  // the top level in split storage (never the bottom or the coarsest level)
    int status = split_sweeps(lv.info, *split, sweeps, nullptr, nullptr, st);
    if (status != PLUME_OK) return status;
    const PlumeLevel& coarse = levels[1];
    const Dims cd = dims_of(coarse.info);
    const dim3 grid(((cd.n2 + 3) / 4 + TZ - 1) / TZ, (cd.n1 + TY - 1) / TY, cd.n0);
    status = launch_solve_kernel(k_residual_restrict_split, grid, cell_block(), 0, st, "residual and restriction (split)",
                                 level_table(lv.info), dims_of(lv.info), split->H, (const float*)split->q,
                                 (const float*)split->rhs, cd, coarse.rhs, coarse.q);
    if (status != PLUME_OK) return status;
    Pressure coarse_q{coarse.q, coarse.residual};
    if ((status = v_cycle(levels, count, 1, coarse_q, plan, sweeps, st, coarse_f64)) != PLUME_OK) return status;
    if (coarse_q.cur != coarse.q) {
      status = runtime_status("coarse pressure copy",
                              cudaMemcpyAsync(coarse.q, coarse_q.cur, sizeof(float) * cd.n0 * cd.n1 * cd.n2,
                                              cudaMemcpyDeviceToDevice, st));
      if (status != PLUME_OK) return status;
    }
    return split_sweeps(lv.info, *split, sweeps, coarse.q, &coarse.info, st);
  }
  if (index == plan.start) {
    if (coarse_f64) return launch_block_solve(levels + index, count - index, sweeps, plan.smem, st);
    return launch_cluster_solve(cluster_solve(levels, count, plan, 1, sweeps, plan.store_all), pdl_enabled(), st);
  }
  if (index == count - 1) {
    if (coarse_f64) {
      const size_t bytes = 2 * sizeof(double) * (size_t)cells_of(lv.info);
      if (bytes > BOTTOM_MAX_SMEM) return fail(PLUME_ERR_INVALID, "coarsest level too large for the double solve");
      int status = prepare_bottom();
      if (status != PLUME_OK) return status;
      return launch_solve_kernel(k_coarsest_f64, dim3(1), dim3(BOTTOM_THREADS), bytes, st, "coarsest double solve",
                                 lv.info, q.cur, lv.rhs, coarsest_sweeps(lv.info));
    }
    return sweeps_with_prolong(lv.info, q, lv.rhs, coarsest_sweeps(lv.info), 1.5f, nullptr, nullptr, st);
  }
  int status = sweeps_with_prolong(lv.info, q, lv.rhs, sweeps, 1.0f, nullptr, nullptr, st);
  if (status != PLUME_OK) return status;
  const PlumeLevel& coarse = levels[index + 1];
  const Dims cd = dims_of(coarse.info);
  if ((status = launch_restrict(lv.info, level_table(lv.info), q.cur, lv.rhs, coarse, st)) != PLUME_OK) return status;
  Pressure coarse_q{coarse.q, coarse.residual};
  if ((status = v_cycle(levels, count, index + 1, coarse_q, plan, sweeps, st, coarse_f64)) != PLUME_OK)
    return status;
  if (coarse_q.cur != coarse.q) {  // an odd number of coarsest sweeps left the result in the second array
    status = runtime_status("coarse pressure copy", cudaMemcpyAsync(coarse.q, coarse_q.cur, sizeof(float) * cd.n0 * cd.n1 * cd.n2,
                                                                    cudaMemcpyDeviceToDevice, st));
    if (status != PLUME_OK) return status;
  }
  return sweeps_with_prolong(lv.info, q, lv.rhs, sweeps, 1.0f, coarse.q, &coarse.info, st);
}

// Whether the top level runs split: scratch given, at least two levels with level 0 above the bottom (a level of
// at most g_bottom_max_cells) and halved by level 1, uniform couplings, swept by colour (not tiled) and at least g_split_min_cells cells.
static bool use_split(const PlumeLevel* levels, int count, int coarse_f64, const float* scratch) {
  const PlumeGridInfo& info = levels[0].info;
  return scratch && ((uintptr_t)scratch & 15) == 0 && count >= 2 && uniform_level(info) && halves(info, levels[1].info) &&
         cells_of(info) >= g_split_min_cells && cells_of(info) < g_tiled_min_cells &&
         coarse_plan(levels, count, coarse_f64, 0).single_from > 0;
}

static int multigrid_direct(const PlumeLevel* levels, int count, int cycles, int sweeps, cudaStream_t st,
                            int coarse_f64, float* split_scratch = nullptr) {
  const bool split = use_split(levels, count, coarse_f64, split_scratch);
  CoarsePlan plan = coarse_plan(levels, count, coarse_f64, split ? 1 : 0);
  if (split) {
    const PlumeGridInfo& info = levels[0].info;
    const Dims d = dims_of(info);
    SplitTop sp{split_scratch, split_scratch + split_floats(info), split_H(info)};
    const dim3 grid((sp.H + TZ - 1) / TZ, (d.n1 + TY - 1) / TY, d.n0);
    int status = launch_solve_kernel(k_split_layout<true>, grid, cell_block(), 0, st, "pressure to split storage", d,
                                     sp.H, (const float*)levels[0].q, sp.q);
    if (status != PLUME_OK) return status;
    if ((status = launch_solve_kernel(k_split_layout<true>, grid, cell_block(), 0, st, "divergence to split storage",
                                      d, sp.H, (const float*)levels[0].rhs, sp.rhs)) != PLUME_OK)
      return status;
    Pressure unused{levels[0].q, levels[0].residual};
    for (int c = 0; c < cycles; ++c) {
      plan.store_all = c == cycles - 1;
      if ((status = v_cycle(levels, count, 0, unused, plan, sweeps, st, coarse_f64, &sp)) != PLUME_OK)
        return status;
    }
    return launch_solve_kernel(k_split_layout<false>, grid, cell_block(), 0, st, "pressure from split storage", d,
                               sp.H, (const float*)sp.q, levels[0].q);
  }
  if (plan.start == 0 && !coarse_f64 && cycles > 0)
    return launch_cluster_solve(cluster_solve(levels, count, plan, cycles, sweeps, true), pdl_enabled(), st);
  Pressure q{levels[0].q, levels[0].residual};
  for (int c = 0; c < cycles; ++c) {
    plan.store_all = c == cycles - 1;
    int status = v_cycle(levels, count, 0, q, plan, sweeps, st, coarse_f64);
    if (status != PLUME_OK) return status;
  }
  if (q.cur == levels[0].q) return PLUME_OK;
  return runtime_status("pressure copy-back", cudaMemcpyAsync(levels[0].q, q.cur, sizeof(float) * (size_t)cells_of(levels[0].info),
                                                              cudaMemcpyDeviceToDevice, st));
}

}  // namespace plume

namespace plume {

// ---- replaying the solve as a CUDA graph -----------------------------------------------------------------
// The launch sequence of a solve depends only on the levels (geometry and arrays), the cycle and sweep
// counts and the strategy, so it is captured once into a graph (on a private stream: capture records and
// runs nothing) and replayed on the caller's stream, which saves the per-launch cost of its ~30 launches per
// V-cycle, most of them short.
struct GraphKey {
  int device;
  int count, cycles, sweeps, kind, coarse_f64;
  long tiled, bottom, split_min;
  float* split;
  PlumeLevel levels[16];
  bool operator==(const GraphKey& o) const { return std::memcmp(this, &o, sizeof(GraphKey)) == 0; }
};

struct GraphEntry {
  GraphKey key;
  uint64_t hash;
  cudaGraphExec_t exec;
  size_t kernels;  // kernel nodes in the graph
};

static uint64_t key_hash(const GraphKey& key) {  // FNV-1a over the key's bytes
  uint64_t h = 1469598103934665603ull;
  const unsigned char* bytes = reinterpret_cast<const unsigned char*>(&key);
  for (size_t i = 0; i < sizeof(GraphKey); ++i) h = (h ^ bytes[i]) * 1099511628211ull;
  return h;
}

static std::mutex g_graph_mutex;
static std::vector<GraphEntry> g_graphs;
static cudaStream_t g_capture_stream[64] = {};
static bool g_use_graphs = true;
constexpr size_t MAX_GRAPHS = 1024;  // one per live level hierarchy (batched runs hold many)

static int graph_for(const GraphKey& key, const PlumeLevel* levels, cudaGraphExec_t* out, size_t* kernels) {
  const uint64_t hash = key_hash(key);
  for (const GraphEntry& e : g_graphs)
    if (e.hash == hash && e.key == key) {
      *out = e.exec;
      *kernels = e.kernels;
      return PLUME_OK;
    }
  cudaStream_t& cap = g_capture_stream[key.device];
  int status = PLUME_OK;
  if (!cap) status = runtime_status("capture stream", cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
  if (status != PLUME_OK) return status;
  // one-time function attributes are set outside the capture: run the smallest possible warm-up first
  status = runtime_status("begin capture", cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
  if (status != PLUME_OK) return status;
  set_launch_counting(false);
  const int run = multigrid_direct(levels, key.count, key.cycles, key.sweeps, cap, key.coarse_f64, key.split);
  set_launch_counting(true);
  cudaGraph_t graph = nullptr;
  status = runtime_status("end capture", cudaStreamEndCapture(cap, &graph));
  if (run != PLUME_OK || status != PLUME_OK) {
    if (graph) cudaGraphDestroy(graph);
    return run != PLUME_OK ? run : status;
  }
  size_t nodes = 0, kernel_nodes = 0;
  if (cudaGraphGetNodes(graph, nullptr, &nodes) == cudaSuccess && nodes > 0) {
    std::vector<cudaGraphNode_t> list(nodes);
    if (cudaGraphGetNodes(graph, list.data(), &nodes) == cudaSuccess)
      for (cudaGraphNode_t node : list) {
        cudaGraphNodeType type;
        if (cudaGraphNodeGetType(node, &type) == cudaSuccess && type == cudaGraphNodeTypeKernel) ++kernel_nodes;
      }
  }
  cudaGraphExec_t exec = nullptr;
  status = runtime_status("instantiate graph", cudaGraphInstantiate(&exec, graph, 0));
  cudaGraphDestroy(graph);
  if (status != PLUME_OK) return status;
  if (g_graphs.size() >= MAX_GRAPHS) {
    cudaGraphExecDestroy(g_graphs.front().exec);
    g_graphs.erase(g_graphs.begin());
  }
  g_graphs.push_back(GraphEntry{key, hash, exec, kernel_nodes});
  *out = exec;
  *kernels = kernel_nodes;
  return PLUME_OK;
}

int multigrid_cycles(const PlumeLevel* levels, int count, int cycles, int sweeps, cudaStream_t st, int coarse_f64,
                     float* split_scratch) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  int device = 0;
  int prepared = prepare_bottom();
  if (prepared != PLUME_OK) return prepared;
  if (!g_use_graphs || count > 16 || cudaStreamIsCapturing(st, &capturing) != cudaSuccess ||
      capturing != cudaStreamCaptureStatusNone || cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64)
    return multigrid_direct(levels, count, cycles, sweeps, st, coarse_f64, split_scratch);
  GraphKey key;
  std::memset(&key, 0, sizeof(key));
  key.device = device;
  key.count = count;
  key.cycles = cycles;
  key.sweeps = sweeps;
  key.kind = g_bottom_kind;
  key.coarse_f64 = coarse_f64;
  key.tiled = g_tiled_min_cells;
  key.bottom = g_bottom_max_cells;
  key.split_min = g_split_min_cells;
  key.split = split_scratch;
  std::memcpy(key.levels, levels, sizeof(PlumeLevel) * count);
  std::lock_guard<std::mutex> lock(g_graph_mutex);
  cudaGraphExec_t exec = nullptr;
  size_t kernels = 0;
  int status = graph_for(key, levels, &exec, &kernels);
  if (status != PLUME_OK) return status;
  status = runtime_status("graph launch", cudaGraphLaunch(exec, st));
  if (status == PLUME_OK) count_launches(kernels);
  return status;
}

}  // namespace plume

extern "C" int plume_use_graphs(int32_t enable) {
  plume::g_use_graphs = enable != 0;
  return PLUME_OK;
}

extern "C" int plume_tune_solver(long long tiled_min_cells, long long bottom_max_cells, int32_t bottom_kind) {
  if (tiled_min_cells < 1 || bottom_max_cells < 0 || bottom_kind < 0 || bottom_kind > 1)
    return plume::fail(PLUME_ERR_INVALID, "tune_solver: thresholds must be positive, bottom_kind 0 or 1");
  plume::g_tiled_min_cells = (long)tiled_min_cells;
  plume::g_bottom_max_cells = (long)bottom_max_cells;
  plume::g_bottom_kind = bottom_kind;
  return PLUME_OK;
}

extern "C" int plume_tune_split(long long min_cells) {
  if (min_cells < 1) return plume::fail(PLUME_ERR_INVALID, "tune_split: min_cells must be positive");
  plume::g_split_min_cells = (long)min_cells;
  return PLUME_OK;
}

extern "C" long long plume_split_min_cells(void) { return plume::g_split_min_cells; }

extern "C" long long plume_split_scratch_floats(const PlumeGridInfo* info) {
  if (!info || info->dims[0] < 1 || info->dims[1] < 1 || info->dims[2] < 1)
    return plume::fail(PLUME_ERR_INVALID, "split_scratch_floats: bad dims");
  return 2 * plume::split_floats(*info);
}

extern "C" int plume_solver_tuning(long long* tiled_min_cells, long long* bottom_max_cells, int32_t* bottom_kind) {
  if (!tiled_min_cells || !bottom_max_cells || !bottom_kind)
    return plume::fail(PLUME_ERR_INVALID, "solver_tuning: null output");
  *tiled_min_cells = plume::g_tiled_min_cells;
  *bottom_max_cells = plume::g_bottom_max_cells;
  *bottom_kind = plume::g_bottom_kind;
  return PLUME_OK;
}
