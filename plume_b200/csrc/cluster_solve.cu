// Multigrid V-cycles over the small levels of the pressure solve in one launch of one thread-block cluster
// (chadmv/plume src/plume/sim/pressure.py:39-92, multigrid.py:36-68, :124-147), with the reference's update
// order and arithmetic: every float equals the one the launches of multigrid.cu produce.
//
// What bounds these levels is latency, not work: a colour pass of 50 thousand cells is a third of a microsecond
// of arithmetic on a few SMs but costs a whole launch (2 to 5 us in a graph) as a kernel of its own, and a V-cycle
// over four such levels is about forty dependent passes. So the levels' arrays stay in the shared memory of up to
// 16 SMs and a pass ends in a cluster barrier (500 to 700 cycles) instead of a launch. Measured on B200 when it was made,
// the solve against the per-colour launches of then with the levels of at most 2048 cells in one block: 38x48x38 (2
// cycles) 107 against 195 us, 48x48x48 (4 cycles) 207 against 413, 64x96x64 270 against 380, 75x113x91 455 against 750,
// 128x192x128 610 against 729. The launched passes have since become as fast a level: with only the levels of at most
// 2048 cells in the cluster, against the rule of multigrid.cu, 64x96x64 takes 290 and 275 us, 128x192x128 511 and 496,
// 48x48x48 238 and 241, 38x48x38 131 and 141.
//
// What a pass then waits for is instruction fetch and dependent arithmetic: two to four warps a scheduler run
// each phase once through and go on to the next. So the hot phases are free of branches over code that does not
// run (missing neighbours read a float that stays 0, stores without a receiver go to floats nothing reads,
// quotients have no slow path), loops are kept rolled, and index divisions are multiplications (Divider).
// At 128 registers a thread it spills 40 bytes.
// Rejected: 1024 threads with one cell each (more barrier time); one mbarrier arrival per neighbour and pass instead
// of the cluster barrier (1.95 against 1.3 thousand cycles a pass over 6 thousand cells); a block's larger levels with
// two cells of a colour per thread in one CTA instead of slabs.
//
// Layout. A level before `single_from` is cut into slabs of whole x-planes, one per CTA, in colour-split storage:
// q[colour][plane][j][m] with one halo plane on each side, rhs[colour][plane][j][m], cell (i, j, k) of colour
// (i + j + k) & 1 at m = k >> 1. Lanes walk m, so neighbouring lanes read neighbouring words (the natural layout's
// stride of two cells would put two lanes in each bank). A CTA stores its boundary planes' new values straight
// into its neighbours' halo planes through distributed shared memory, so the passes themselves read local memory
// only. Halo planes outside the level and the padding slot of an odd row hold 0, which is what neighbor_sum adds
// for a missing neighbour. Levels from `single_from` on sit in CTA 0 in natural layout.
//
// Stencils come from a table per level by cell class (stencil_table.cuh), built once per launch with the reference's
// operations. The quotient (sq - source) / sc is the product with the table's double reciprocal of sc.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "cluster_solve.cuh"
#include "stencil_table.cuh"

namespace plume {

namespace cg = cooperative_groups;

constexpr int CS_THREADS = 512;
constexpr size_t CS_MAX_SMEM = 220 * 1024;

constexpr int STENCIL_FLOATS = sizeof(ClassStencil) / sizeof(float);

// x / d and x % d for 0 <= x < 65536, d < 65536 by one multiplication: inverse = ceil(2^32 / d), 0 for d = 1.
struct Divider {
  int d;
  unsigned inverse;
  __device__ __forceinline__ int quotient(int x) const { return inverse ? (int)__umulhi((unsigned)x, inverse) : x; }
};

struct ClusterLevel {
  PlumeGridInfo info;
  float* q;
  float* rhs;
  int planes;      // x-planes per CTA; 0 when the level lives in CTA 0
  int H;           // floats per row of a colour: (n2 + 1) / 2 cells, padded to a multiple of four
  int q_at, rhs_at, table_at;  // float offsets in shared memory
  int uniform;     // no overhanging cells: every inner coupling is 1
  Divider by_planes, by_n1, by_n2, by_half, by_quads;  // planes, the axes, (n2 + 1) / 2 and H / 4
};

struct ClusterArgs {
  int count, single_from, cycles, sweeps, last_sweeps;
  int from_zero;  // the first level's pressure starts at 0 (its array is not read)
  float last_relaxation;
  int buffer_at;  // the coarse planes a CTA's prolongation reads (natural layout)
  int zero_at;    // four floats that stay 0 (missing neighbours), then four that nothing reads
  int floats;     // shared memory in use
  int store_all;  // the coarser levels' arrays are wanted too, not only the first level's pressure
  ClusterLevel lv[CLUSTER_MAX_LEVELS];
};

extern __shared__ __align__(16) float smem[];

// 1 / d for quotient(): two Newton steps in double from the approximate float reciprocal (relative error 2^-23, then
// 2^-46, then the double's rounding), without a division's branch. For divisors the approximate one holds for
// (spacing_in_range).
__device__ __forceinline__ double reciprocal(float d) {
  const double x = (double)d;
  double y = (double)__fdividef(1.0f, d);
  y = __fma_rn(y, __fma_rn(-x, y, 1.0), y);
  return __fma_rn(y, __fma_rn(-x, y, 1.0), y);
}

// The stencil of cell (i, j, k), written to `out`: neighbor_sum's couplings (poisson.cuh) in its order. Rolled up: it
// runs once per launch, when each of its instructions is fetched for the first time.
__device__ __forceinline__ void write_stencil(const PlumeGridInfo& info, int i, int j, int k, ClassStencil* out) {
  const float fill[3] = {cell_fill(info, 0, i), cell_fill(info, 1, j), cell_fill(info, 2, k)};
  float sc = 0.0f;
#pragma unroll 1
  for (int face = 0; face < 6; ++face) {
    const int axis = face >> 1, step = face & 1 ? 1 : -1;
    const int index = axis == 0 ? i : (axis == 1 ? j : k);
    const float own = axis == 0 ? fill[0] : (axis == 1 ? fill[1] : fill[2]);
    const float area = (axis == 0 ? fill[1] : fill[0]) * (axis == 2 ? fill[1] : fill[2]);
    const int n = index + step;
    const bool inside = n >= 0 && n < info.dims[axis], open = step < 0 ? info.open_lo[axis] == 1 : info.open_hi[axis] == 1;
    const float apart = inside ? 0.5f * (own + cell_fill(info, axis, n)) : 0.5f * own + info.ghost_gap;
    const float coupling = inside || open ? quotient(area, reciprocal(apart)) : 0.0f;
    out->c[face] = coupling;
    sc = sc + coupling;
  }
  const float vc = fill[0] * fill[1] * fill[2] * info.cell_m * info.cell_m;
  out->sc = sc;
  out->vc = vc;
  out->inv = reciprocal(sc);  // unused when sc is 0
  out->inv_vc = reciprocal(vc);
}

struct Cta {
  cg::cluster_group cluster;
  int rank;
  int ctas;
  __device__ __forceinline__ void sync() const {
    if (ctas > 1) cluster.sync();
    else __syncthreads();
  }
  // a float of shared memory of another CTA
  __device__ __forceinline__ float* remote(int at, int other) const { return cluster.map_shared_rank(smem + at, other); }
};

// The index triple (i, j, c) of x = (i * n1 + j) * nc + c.
struct Triple {
  int i, j, c;
  __device__ __forceinline__ Triple(int x, const Divider& by_n1, const Divider& by_nc) {
    const int row = by_nc.quotient(x);
    c = x - row * by_nc.d;
    i = by_n1.quotient(row);
    j = row - i * by_n1.d;
  }
};

// The CTA holding x-plane i of a level (0 for a level in one CTA).
__device__ __forceinline__ int owner_of(const ClusterLevel& L, int i) { return L.planes ? L.by_planes.quotient(i) : 0; }

// The float offset of cell (i, j, k)'s right-hand side (or, with `halo` 1, pressure) from its array's start in its
// owner's shared memory.
__device__ __forceinline__ int cell_at(const ClusterLevel& L, int owner, int i, int j, int k, int halo) {
  const int n1 = L.info.dims[1];
  const int slab = ((((i + j + k) & 1) * (L.planes + 2 * halo) + i - owner * L.planes + halo) * n1 + j) * L.H + (k >> 1);
  return L.planes ? slab : (i * n1 + j) * L.info.dims[2] + k;
}

// The slab of a level this CTA holds, and where its arrays are.
struct Slab {
  int lo, planes;       // first x-plane and how many (0 when the level has fewer slabs than the cluster has CTAs)
  int P, n0, n1, n2, H, plane;  // plane = n1 * H
  int q_at, rhs_at;
  __device__ __forceinline__ Slab(const ClusterLevel& L, const Cta& c) {
    P = L.planes;
    n0 = L.info.dims[0];
    n1 = L.info.dims[1];
    n2 = L.info.dims[2];
    H = L.H;
    plane = n1 * H;
    lo = imin_(c.rank * P, n0);
    planes = imin_(lo + P, n0) - lo;
    q_at = L.q_at;
    rhs_at = L.rhs_at;
  }
  // float offsets of the row (colour, local plane -1 .. P, j)
  __device__ __forceinline__ int q_row(int colour, int pl, int j) const { return q_at + (colour * (P + 2) + pl + 1) * plane + j * H; }
  __device__ __forceinline__ int rhs_row(int colour, int pl, int j) const { return rhs_at + (colour * P + pl) * plane + j * H; }
};

__device__ __forceinline__ float4 at4(int at) { return *reinterpret_cast<const float4*>(smem + at); }

struct Four {
  float v[4];
  __device__ __forceinline__ Four(float4 a) : v{a.x, a.y, a.z, a.w} {}
};

// The float holding the z neighbour beyond a thread's four cells m0 .. m0 + 3 of parity p, in the other colour's row
// at `oth`: below the first for even cells, above the last for odd ones.
__device__ __forceinline__ int far_z(int oth, int m0, int p, int H, int zero) {
  const int at = p == 0 ? oth - 1 : oth + 4;
  return (p == 0 ? m0 > 0 : m0 + 4 < H) ? at : zero;
}

// Stores four new values of the local plane pl, and into the halo plane of the neighbouring CTA when pl is a
// boundary plane. The addresses are chosen instead of the stores being branched over: without a neighbour they go
// to four floats that nothing reads (zero + 4).
struct Push {
  float *below, *above;  // shared memory of the neighbouring CTAs, or null
  int sink;
  __device__ __forceinline__ Push(const Slab& s, const Cta& c, int zero) {
    below = s.planes > 0 && s.lo > 0 ? c.remote(0, c.rank - 1) : nullptr;
    above = s.planes > 0 && s.lo + s.planes < s.n0 ? c.remote(0, c.rank + 1) : nullptr;
    sink = zero + 4;
  }
  __device__ __forceinline__ void store(const Slab& s, int own, int pl, float4 value) const {
    *reinterpret_cast<float4*>(smem + own) = value;
    float* const b = pl == 0 && below ? below + own + s.P * s.plane : smem + sink;
    float* const a = pl == s.planes - 1 && above ? above + own - (pl + 1) * s.plane : smem + sink;
    *reinterpret_cast<float4*>(b) = value;
    *reinterpret_cast<float4*>(a) = value;
  }
};

// A row's classes along z: k = 0, the inner cells and k = n2 - 1 (on a level without overhanging cells the last
// cell but one is an inner cell).
__device__ __forceinline__ int inner_class(int n) { return n >= 4 ? 1 : 2; }

// `sweeps` red-black sweeps of a slab level (red_black_sweep_kernel, pressure.py:80-92). A thread takes four cells
// of a row (the half indices m0 .. m0 + 3) and walks the slab's planes with them, so that the other colour's
// values at m0 .. m0 + 3 serve as x+ neighbours, then z neighbours, then x- neighbours from one 16-byte load. The
// body is kept short and free of branches: with two to four warps a scheduler, instruction fetch and latency are
// what a pass waits for.
template <bool UNIFORM>
__device__ __forceinline__ void slab_smooth(const ClusterLevel& L, const Cta& c, int zero, int sweeps, float relaxation) {
  const Slab s(L, c);
  const int quads = s.H / 4, columns = s.planes > 0 ? s.n1 * quads : 0;
  const ClassStencil* table = reinterpret_cast<const ClassStencil*>(smem + L.table_at);
  const float h2 = L.info.cell_m * L.info.cell_m;
  const int inner = inner_class(s.n2), front = class_of(0, s.n2), last_m = (s.n2 - 1) >> 1, last_p = (s.n2 - 1) & 1;
  const Push push(s, c, zero);
#pragma unroll 1
  for (int pass = 0; pass < 2 * sweeps; ++pass) {
    const int colour = pass & 1;
#pragma unroll 1
    for (int column = threadIdx.x; column < columns; column += CS_THREADS) {
      const int j = L.by_quads.quotient(column), m0 = 4 * (column - j * quads), last_n = last_m - m0;
      const ClassStencil* rows = table + 4 * class_of(j, s.n1);
      int oth = s.q_row(1 - colour, 0, j) + m0, own = s.q_row(colour, 0, j) + m0, rhs = s.rhs_row(colour, 0, j) + m0;
      float4 low = at4(oth - s.plane), mid = at4(oth);
#pragma unroll 1
      for (int pl = 0; pl < s.planes; ++pl, oth += s.plane, own += s.plane, rhs += s.plane) {
        const int i = s.lo + pl, p = (i + j + colour) & 1;  // cell k = 2 m + p
        const float4 high = at4(oth + s.plane);
        const Four xm(low), xp(high), zc(mid), q(at4(own)), r(at4(rhs));
        const Four ym(at4(j > 0 ? oth - s.H : zero)), yp(at4(j < s.n1 - 1 ? oth + s.H : zero));
        const float far = smem[far_z(oth, m0, p, s.H, zero)];
        const ClassStencil* row = rows + 16 * class_of(i, s.n0);
        float x[4], out[4];
        double inv[4];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const float zm = p == 0 ? (n == 0 ? far : zc.v[n > 0 ? n - 1 : 0]) : zc.v[n];
          const float zp = p == 0 ? zc.v[n] : (n == 3 ? far : zc.v[n < 3 ? n + 1 : 3]);
          if (UNIFORM) {
            x[n] = (((((xm.v[n] + xp.v[n]) + ym.v[n]) + yp.v[n]) + zm) + zp) - h2 * r.v[n];
            inv[n] = row[p == last_p && n == last_n ? 3 : (n == 0 && m0 == 0 && p == 0 ? front : inner)].inv;
          } else {
            const ClassStencil& e = row[class_of(2 * (m0 + n) + p, s.n2)];
            x[n] = (((((e.c[0] * xm.v[n] + e.c[1] * xp.v[n]) + e.c[2] * ym.v[n]) + e.c[3] * yp.v[n]) + e.c[4] * zm) +
                    e.c[5] * zp) - e.vc * r.v[n];
            inv[n] = e.inv;
          }
        }
        const int cells = (s.n2 - p + 1) / 2 - m0;  // how many of the four exist; a padding slot stays 0
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const float value = q.v[n] + relaxation * (quotient(x[n], inv[n]) - q.v[n]);
          out[n] = n < cells ? value : q.v[n];
        }
        const float4 result = make_float4(out[0], out[1], out[2], out[3]);
        push.store(s, own, pl, result);
        low = mid;
        mid = high;
      }
    }
    c.sync();
  }
}

__device__ __forceinline__ float stencil_residual(const ClassStencil& e, float q, float rhs, float xm, float xp, float ym,
                                                  float yp, float zm, float zp) {  // residual_at from a class stencil
  const float sq = ((((e.c[0] * xm + e.c[1] * xp) + e.c[2] * ym) + e.c[3] * yp) + e.c[4] * zm) + e.c[5] * zp;
  return rhs - quotient(sq - e.sc * q, e.inv_vc);
}

// residual_kernel + restrict_kernel + coarse.q.zero_() (multigrid.py:36-60, :143) from slab level F into C. The
// CTA holding the first child plane of a coarse plane forms its cells, four of a row per thread: the children of
// coarse cell kc sit at half index m = kc in both colours' rows. The second child plane and the one beyond may be
// the next CTAs' (read through distributed shared memory).
template <bool UNIFORM>
__device__ __forceinline__ void slab_restrict(const ClusterLevel& F, const ClusterLevel& C, const Cta& c, int zero) {
  const Slab s(F, c);
  const int c1 = C.info.dims[1], c2 = C.info.dims[2], quads = s.H / 4;
  const ClassStencil* table = reinterpret_cast<const ClassStencil*>(smem + F.table_at);
  const int inner = inner_class(s.n2), front = class_of(0, s.n2), last_m = (s.n2 - 1) >> 1, last_p = (s.n2 - 1) & 1;
  {  // the coarse pressure starts at 0 (halo planes included)
    const int floats = C.planes ? 2 * (C.planes + 2) * c1 * C.H : (c.rank == 0 ? C.info.dims[0] * c1 * c2 : 0);
#pragma unroll 1
    for (int n = threadIdx.x; n < floats; n += CS_THREADS) smem[C.q_at + n] = 0.0f;
  }
  const int first = (s.lo + 1) / 2, planes = s.planes > 0 ? (s.lo + s.planes + 1) / 2 - first : 0;
  // the planes beyond this CTA's halo: the pressure of local plane P + 1, the right-hand side of local plane P
  const bool next = s.planes > 0 && s.lo + s.planes < s.n0, beyond = s.planes > 0 && s.lo + s.P + 1 < s.n0;
  const float* const next_rhs = next ? c.remote(s.rhs_at, c.rank + 1) : smem;
  const float* const beyond_q =
      beyond ? (s.P == 1 ? c.remote(s.q_at, c.rank + 2) + s.plane : c.remote(s.q_at, c.rank + 1) + 2 * s.plane) : smem;
  const double inv_h2 = table[0].inv_vc;  // UNIFORM: the same for every cell
#pragma unroll 1
  for (int at = threadIdx.x; at < planes * c1 * quads; at += CS_THREADS) {
    const Triple w(at, C.by_n1, F.by_quads);
    const int ci = first + w.i, cj = w.j, m0 = 4 * w.c;
    float total[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
    for (int child = 0; child < 4; ++child) {  // in the reference's order (di, dj, then dk)
      const bool there = 2 * ci + (child >> 1) < s.n0 && 2 * cj + (child & 1) < s.n1;
      const int fi = there ? 2 * ci + (child >> 1) : 2 * ci, fj = there ? 2 * cj + (child & 1) : 2 * cj;
      const int pl = fi - s.lo, in_plane = fj * s.H + m0, colour_q = (s.P + 2) * s.plane, colour_rhs = s.P * s.plane;
      const ClassStencil* row = table + 4 * (4 * class_of(fi, s.n0) + class_of(fj, s.n1));
      // cells of parity p have colour c0 ^ p; `rows[p]`: their row of this plane
      const int c0 = (fi + fj) & 1, at_q = s.q_row(0, pl, fj) + m0;
      const int rows[2] = {at_q + c0 * colour_q, at_q + (1 - c0) * colour_q};
      const float* high = smem + (fi < s.n0 - 1 ? at_q + s.plane : zero);
      high = pl == s.P && beyond ? beyond_q + in_plane : high;
      const int high_step = fi < s.n0 - 1 ? colour_q : 0;
      const float* right = pl == s.P ? next_rhs + in_plane : smem + s.rhs_row(0, pl, fj) + m0;
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int own = rows[p], oth = rows[1 - p], c_own = c0 ^ p, c_oth = 1 - c_own;
        const Four xm(at4(oth - s.plane)), zc(at4(oth)), q(at4(own));
        const Four xp(*reinterpret_cast<const float4*>(high + c_oth * high_step));
        const Four r(*reinterpret_cast<const float4*>(right + c_own * colour_rhs));
        const Four ym(at4(fj > 0 ? oth - s.H : zero)), yp(at4(fj < s.n1 - 1 ? oth + s.H : zero));
        const float far = smem[far_z(oth, m0, p, s.H, zero)];
        const int cells = (s.n2 - p + 1) / 2 - m0;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const float zm = p == 0 ? (n == 0 ? far : zc.v[n > 0 ? n - 1 : 0]) : zc.v[n];
          const float zp = p == 0 ? zc.v[n] : (n == 3 ? far : zc.v[n < 3 ? n + 1 : 3]);
          float residual;
          if (UNIFORM) {
            const float sc = row[p == last_p && m0 + n == last_m ? 3 : (n == 0 && m0 == 0 && p == 0 ? front : inner)].sc;
            const float sq = ((((xm.v[n] + xp.v[n]) + ym.v[n]) + yp.v[n]) + zm) + zp;
            residual = r.v[n] - quotient(sq - sc * q.v[n], inv_h2);
          } else {
            residual = stencil_residual(row[class_of(2 * (m0 + n) + p, s.n2)], q.v[n], r.v[n], xm.v[n], xp.v[n], ym.v[n],
                                        yp.v[n], zm, zp);
          }
          const float sum = total[n] + residual;
          total[n] = there && n < cells ? sum : total[n];
        }
      }
    }
    const float xy = (2 * ci + 1 < s.n0 ? 0.5f : 1.0f) * (2 * cj + 1 < s.n1 ? 0.5f : 1.0f);
    const int owner = owner_of(C, ci);
    float* out = owner == c.rank ? smem : c.remote(0, owner);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int ck = m0 + n;
      if (ck < c2) out[C.rhs_at + cell_at(C, owner, ci, cj, ck, 0)] = total[n] * (xy * (2 * ck + 1 < s.n2 ? 0.5f : 1.0f));  // / 1, 2, 4 or 8: the same float
    }
  }
}

// prolong_add_kernel (multigrid.py:63-68) from C into slab level F: the coarse planes this CTA's cells sample are
// copied to its buffer first, from whichever CTAs hold them. A thread takes the eight cells at half indices
// m0 .. m0 + 3 of a row: they share the coarse sample's x and y axes, along z they read the six coarse columns
// m0 - 1 .. m0 + 4 (clamped), each blended in x then y once, and cell m of parity p blends columns m - 1 + p and
// m + p with the exact weights 0.75 and 0.25, except where the clamp holds (k = 0, and k = n2 - 1 of an even n2).
// Every operation is sample_index_space's (common.cuh).
__device__ __forceinline__ void slab_prolong(const ClusterLevel& F, const ClusterLevel& C, const Cta& c, int buffer_at,
                                             int zero) {
  const Slab s(F, c);
  const Dims cd{C.info.dims[0], C.info.dims[1], C.info.dims[2]};
  if (s.planes == 0) return;
  const int hi = s.lo + s.planes;
  const int first = imax_((s.lo - 1) >> 1, 0), last = imin_(hi >> 1, cd.n0 - 1);
  {
    const int cells = (last - first + 1) * cd.n1 * cd.n2;
#pragma unroll 1
    for (int base = threadIdx.x; base < cells; base += 2 * CS_THREADS) {  // two loads in flight per thread
      float value[2];
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const Triple w(imin_(base + n * CS_THREADS, cells - 1), C.by_n1, C.by_n2);
        const int ci = first + w.i, owner = owner_of(C, ci), at = C.q_at + cell_at(C, owner, ci, w.j, w.c, 1);
        value[n] = *(owner == c.rank ? smem + at : c.remote(at, owner));
      }
      smem[buffer_at + base] = value[0];
      if (base + CS_THREADS < cells) smem[buffer_at + base + CS_THREADS] = value[1];
    }
  }
  __syncthreads();
  const Push push(s, c, zero);
  const int quads = s.H / 4;
#pragma unroll 1
  for (int n = threadIdx.x; n < s.planes * s.n1 * quads; n += CS_THREADS) {
    const Triple w(n, F.by_n1, F.by_quads);
    const int pl = w.i, j = w.j, m0 = 4 * w.c, i = s.lo + pl;
    const F3 g = prolong_point(i, j, 0);
    const Axis1 x = axis_of(g[0], cd.n0, cd.n1 * cd.n2), y = axis_of(g[1], cd.n1, cd.n2);
    const float* base = smem + buffer_at + ((x.i0 - first) * cd.n1 + y.i0) * cd.n2;
    float e[6];
#pragma unroll
    for (int o = 0; o < 6; ++o) {
      const float* f = base + imin_(imax_(m0 - 1 + o, 0), cd.n2 - 1);
      e[o] = lerp_w(lerp_w(f[0], f[x.step], x), lerp_w(f[y.step], f[x.step + y.step], x), y);
    }
#pragma unroll 1
    for (int p = 0; p < 2; ++p) {
      const int own = s.q_row((i + j + p) & 1, pl, j) + m0, cells = (s.n2 - p + 1) / 2 - m0;
      const Four q(at4(own));
      const float t = p == 0 ? 0.75f : 0.25f, u = p == 0 ? 0.25f : 0.75f;
      float out[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float lo = p == 0 ? e[k] : e[k + 1], up = p == 0 ? e[k + 1] : e[k + 2];
        // at a clamp: column 0 and 1, or the last column twice, with weights 1 and 0
        const bool front = p == 0 && m0 + k == 0, back = p == 1 && m0 + k >= cd.n2 - 1;
        const float value = (front ? e[1] : lo) * (front || back ? 1.0f : u) +
                            (front ? e[2] : (back ? lo : up)) * (front || back ? 0.0f : t);
        out[k] = k < cells ? q.v[k] + value : q.v[k];
      }
      const float4 result = make_float4(out[0], out[1], out[2], out[3]);
      push.store(s, own, pl, result);
    }
  }
}

// ---- levels in CTA 0 ------------------------------------------------------------------------------------------
// A cell one thread updates in every sweep of a smoothing call: the shared-memory float offsets of itself and its
// neighbours (a missing neighbour: a float that stays 0), its couplings and source term. A slot without a cell, or
// with a cell that couples to nothing (which the reference leaves alone), holds the 0 float as its cell and zero
// couplings: its update stores that 0 again.
struct CellSlot {
  int own;
  int nb[6];
  float c[6];
  float source;
  double inv;
};

// The red (colour 0) and black cell of pair x = (i * n1 + j) * half + (k >> 1).
struct SlotPair {
  CellSlot slot[2];
  int odd;  // the red cell's parity along z
};

__device__ __forceinline__ SlotPair slot_pair(const ClusterLevel& L, int x, int zero) {
  const int n0 = L.info.dims[0], n1 = L.info.dims[1], n2 = L.info.dims[2];
  const Triple w(x, L.by_n1, L.by_half);
  const int i = imin_(w.i, n0 - 1), j = w.j;
  SlotPair pair;
  pair.odd = (w.i + j) & 1;
  const ClassStencil* row = reinterpret_cast<const ClassStencil*>(smem + L.table_at) + 4 * (4 * class_of(i, n0) + class_of(j, n1));
#pragma unroll
  for (int colour = 0; colour < 2; ++colour) {
    const int at_k = 2 * w.c + (pair.odd ^ colour), k = imin_(at_k, n2 - 1);
    const int index = (i * n1 + j) * n2 + k, own = L.q_at + index;
    const ClassStencil& e = row[class_of(k, n2)];
    const bool cell = w.i < n0 && at_k < n2 && e.sc != 0.0f;
    const bool there[6] = {i > 0, i < n0 - 1, j > 0, j < n1 - 1, k > 0, k < n2 - 1};
    const int step[6] = {-n1 * n2, n1 * n2, -n2, n2, -1, 1};
    CellSlot& slot = pair.slot[colour];
    slot.own = cell ? own : zero;
#pragma unroll
    for (int n = 0; n < 6; ++n) {
      slot.nb[n] = cell && there[n] ? own + step[n] : zero;
      slot.c[n] = cell ? e.c[n] : 0.0f;
    }
    slot.inv = cell ? e.inv : 0.0;
    slot.source = cell ? e.vc * smem[L.rhs_at + index] : 0.0f;
  }
  return pair;
}

__device__ __forceinline__ float relaxed_slot(const CellSlot& slot, float own, const float* nb, float relaxation) {
  const float sq = ((((slot.c[0] * nb[0] + slot.c[1] * nb[1]) + slot.c[2] * nb[2]) + slot.c[3] * nb[3]) +
                    slot.c[4] * nb[4]) + slot.c[5] * nb[5];
  return own + relaxation * (quotient(sq - slot.source, slot.inv) - own);
}

// `sweeps` red-black sweeps of a level of at most CS_THREADS cells of a colour, one of each per thread.
__device__ __forceinline__ void block_sweeps(const ClusterLevel& L, const SlotPair& pair, int threads, int sweeps,
                                             float relaxation) {
#pragma unroll 1
  for (int s = 0; s < sweeps; ++s) {
#pragma unroll
    for (int colour = 0; colour < 2; ++colour) {
      const CellSlot& slot = pair.slot[colour];
      float nb[6];
#pragma unroll
      for (int n = 0; n < 6; ++n) nb[n] = smem[slot.nb[n]];
      smem[slot.own] = relaxed_slot(slot, smem[slot.own], nb, relaxation);
      asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");  // the warps that hold cells meet alone
    }
  }
}

// The same on one warp (at most 32 cells of a colour): each lane keeps its red and black cell in registers and takes
// their neighbours (all of the other colour) from the lanes that hold them.
__device__ __forceinline__ void warp_sweeps(const ClusterLevel& L, const SlotPair& pair, int zero, int sweeps,
                                            float relaxation) {
  const int half = L.by_half.d, per_plane = L.info.dims[1] * half, lane = threadIdx.x;
  float red = smem[pair.slot[0].own], black = smem[pair.slot[1].own];
  // a cell of parity p has its z neighbours in the other colour at half indices m - 1 + p and m + p
  auto update = [&](const CellSlot& slot, float own, float other, int p) {
    const int from[6] = {lane - per_plane, lane + per_plane, lane - half, lane + half, lane - 1 + p, lane + p};
    float nb[6];
#pragma unroll
    for (int n = 0; n < 6; ++n) {
      const float value = __shfl_sync(0xffffffffu, other, from[n]);
      nb[n] = slot.nb[n] != zero ? value : 0.0f;
    }
    return relaxed_slot(slot, own, nb, relaxation);
  };
#pragma unroll 1
  for (int s = 0; s < sweeps; ++s) {
    red = update(pair.slot[0], red, black, pair.odd);
    black = update(pair.slot[1], black, red, 1 - pair.odd);
  }
  smem[pair.slot[0].own] = red;
  smem[pair.slot[1].own] = black;
}

__device__ __forceinline__ void single_smooth(const ClusterLevel& L, int zero, int sweeps, float relaxation) {
  const int pairs = L.info.dims[0] * L.info.dims[1] * L.by_half.d, threads = (pairs + 31) & ~31;
  if ((int)threadIdx.x < threads) {
    const SlotPair pair = slot_pair(L, threadIdx.x, zero);
    if (threads == 32) warp_sweeps(L, pair, zero, sweeps, relaxation);
    else block_sweeps(L, pair, threads, sweeps, relaxation);
  }
  __syncthreads();
}

// residual_kernel + restrict_kernel + coarse.q.zero_() from level F into C, one coarse cell per thread, its children
// in the reference's order.
__device__ __forceinline__ void single_restrict(const ClusterLevel& F, const ClusterLevel& C, int zero) {
  const Dims fd = dims_of(F.info), cd = dims_of(C.info);
  const ClassStencil* table = reinterpret_cast<const ClassStencil*>(smem + F.table_at);
  const int cells = cd.n0 * cd.n1 * cd.n2, sx = fd.n1 * fd.n2, sy = fd.n2;
#pragma unroll 1
  for (int n = threadIdx.x; n < cells; n += CS_THREADS) {
    const Triple w(n, C.by_n1, C.by_n2);
    float total = 0.0f;
#pragma unroll 1
    for (int child = 0; child < 4; ++child) {
#pragma unroll
      for (int dk = 0; dk < 2; ++dk) {
        const int ti = 2 * w.i + (child >> 1), tj = 2 * w.j + (child & 1), tk = 2 * w.c + dk;
        const bool there = ti < fd.n0 && tj < fd.n1 && tk < fd.n2;
        const int i = imin_(ti, fd.n0 - 1), j = imin_(tj, fd.n1 - 1), k = imin_(tk, fd.n2 - 1);
        const int f = at(fd, i, j, k), q = F.q_at + f;
        const ClassStencil& e = table[4 * (4 * class_of(i, fd.n0) + class_of(j, fd.n1)) + class_of(k, fd.n2)];
        const float sum = total + stencil_residual(e, smem[q], smem[F.rhs_at + f], smem[i > 0 ? q - sx : zero],
                                                   smem[i < fd.n0 - 1 ? q + sx : zero], smem[j > 0 ? q - sy : zero],
                                                   smem[j < fd.n1 - 1 ? q + sy : zero], smem[k > 0 ? q - 1 : zero],
                                                   smem[k < fd.n2 - 1 ? q + 1 : zero]);
        total = there ? sum : total;
      }
    }
    const float share = (2 * w.i + 1 < fd.n0 ? 0.5f : 1.0f) * (2 * w.j + 1 < fd.n1 ? 0.5f : 1.0f) * (2 * w.c + 1 < fd.n2 ? 0.5f : 1.0f);
    smem[C.rhs_at + n] = total * share;  // / 1, 2, 4 or 8: the same float
    smem[C.q_at + n] = 0.0f;
  }
  __syncthreads();
}

__device__ __forceinline__ void single_prolong(const ClusterLevel& F, const ClusterLevel& C) {
  const Dims fd = dims_of(F.info), cd = dims_of(C.info);
#pragma unroll 1
  for (int n = threadIdx.x; n < fd.n0 * fd.n1 * fd.n2; n += CS_THREADS) {
    const Triple w(n, F.by_n1, F.by_n2);
    smem[F.q_at + n] = smem[F.q_at + n] + sample_plain(smem + C.q_at, cd, prolong_point(w.i, w.j, w.c));
  }
  __syncthreads();
}

// ---- the kernel -------------------------------------------------------------------------------------------------
// Level L's pressure (unless it starts at 0) and right-hand side from global memory, copied asynchronously: this CTA's
// planes, and the halo planes' pressure as well.
__device__ __forceinline__ void copy_in(int at, const float* from) {
  const unsigned to = (unsigned)__cvta_generic_to_shared(smem + at);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(to), "l"(__cvta_generic_to_global(from)) : "memory");
}

__device__ __forceinline__ void load_level(const ClusterLevel& L, const Cta& c, bool from_zero) {
  const int n0 = L.info.dims[0], n1 = L.info.dims[1], n2 = L.info.dims[2], P = L.planes;
  const int lo = imin_(c.rank * P, n0), hi = P ? imin_(lo + P, n0) : (c.rank == 0 ? n0 : 0);
  const bool halo = P && lo < hi && !from_zero;
  const int from = halo ? imax_(lo - 1, 0) : lo, to = halo ? imin_(hi + 1, n0) : hi;
  const float* q = L.q + (long)from * n1 * n2;
  const float* rhs = L.rhs + (long)from * n1 * n2;
#pragma unroll 1
  for (int n = threadIdx.x; n < (to - from) * n1 * n2; n += CS_THREADS) {
    const Triple w(n, L.by_n1, L.by_n2);
    const int i = from + w.i;
    if (!from_zero) copy_in(L.q_at + cell_at(L, c.rank, i, w.j, w.c, 1), q + n);
    if (i >= lo && i < hi) copy_in(L.rhs_at + cell_at(L, c.rank, i, w.j, w.c, 0), rhs + n);
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// This CTA's part of level L's pressure, and of its right-hand side, to global memory.
__device__ __forceinline__ void store_level(const ClusterLevel& L, const Cta& c, bool with_rhs) {
  const int n0 = L.info.dims[0], n1 = L.info.dims[1], n2 = L.info.dims[2], P = L.planes;
  const int lo = imin_(c.rank * P, n0), hi = P ? imin_(lo + P, n0) : (c.rank == 0 ? n0 : 0);
  const long base = (long)lo * n1 * n2;
#pragma unroll 1
  for (int n = threadIdx.x; n < (hi - lo) * n1 * n2; n += CS_THREADS) {
    const Triple w(n, L.by_n1, L.by_n2);
    L.q[base + n] = smem[L.q_at + cell_at(L, c.rank, lo + w.i, w.j, w.c, 1)];
    if (with_rhs) L.rhs[base + n] = smem[L.rhs_at + cell_at(L, c.rank, lo + w.i, w.j, w.c, 0)];
  }
}

__global__ void __launch_bounds__(CS_THREADS, 1) k_cluster_solve(const __grid_constant__ ClusterArgs b) {
  const cg::cluster_group cluster = cg::this_cluster();
  const Cta c{cluster, (int)cluster.block_rank(), (int)cluster.num_blocks()};
  // shared memory starts at 0 (halo planes, padding slots, the zero word); the stencil tables need no input
#pragma unroll 1
  for (int n = 4 * threadIdx.x; n < b.floats; n += 4 * CS_THREADS)
    *reinterpret_cast<float4*>(smem + n) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  __syncthreads();
#pragma unroll 1
  for (int n = threadIdx.x; n < 64 * b.count; n += CS_THREADS) {
    const ClusterLevel& L = b.lv[n / 64];
    const int e = n % 64, i = class_index(e / 16, L.info.dims[0]), j = class_index(e / 4 % 4, L.info.dims[1]);
    write_stencil(L.info, i, j, class_index(e % 4, L.info.dims[2]), reinterpret_cast<ClassStencil*>(smem + L.table_at) + e);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the previous kernel's writes are visible from here on
  load_level(b.lv[0], c, b.from_zero != 0);
  c.sync();
  const int last = b.count - 1, zero = b.zero_at;
#pragma unroll 1
  for (int cycle = 0; cycle < b.cycles; ++cycle) {
#pragma unroll 1
    for (int visit = 0; visit <= 2 * last; ++visit) {  // down to the coarsest level and up again
      const bool down = visit < last, up = visit > last;
      const int l = up ? 2 * last - visit : visit;
      const ClusterLevel& L = b.lv[l];
      const int sweeps = l == last ? b.last_sweeps : b.sweeps;
      const float relaxation = l == last ? b.last_relaxation : 1.0f;
      if (l < b.single_from) {
        if (up) {
          if (l == b.single_from - 1) c.sync();  // CTA 0's part is done
          slab_prolong(L, b.lv[l + 1], c, b.buffer_at, zero);
          c.sync();
        }
        if (L.uniform) slab_smooth<true>(L, c, zero, sweeps, relaxation);
        else slab_smooth<false>(L, c, zero, sweeps, relaxation);
        if (down) {
          if (L.uniform) slab_restrict<true>(L, b.lv[l + 1], c, zero);
          else slab_restrict<false>(L, b.lv[l + 1], c, zero);
          c.sync();
        }
      } else if (c.rank == 0) {
        if (up) single_prolong(L, b.lv[l + 1]);
        single_smooth(L, zero, sweeps, relaxation);
        if (down) single_restrict(L, b.lv[l + 1], zero);
      }
    }
  }
#pragma unroll 1
  for (int l = 0; l < (b.store_all ? b.count : 1); ++l) store_level(b.lv[l], c, l > 0);
  c.sync();  // no CTA leaves while another may still read its shared memory
}

// ---- host side --------------------------------------------------------------------------------------------------
static int padded4(int n) { return (n + 3) / 4 * 4; }  // arrays start at 16-byte boundaries

static Divider divider(int d) { return Divider{d, d == 1 ? 0u : (unsigned)((0x100000000ull + d - 1) / d)}; }

static ClusterArgs cluster_args(const ClusterSolve& s) {
  ClusterArgs b{};
  b.count = s.count;
  b.single_from = s.single_from;
  b.from_zero = s.from_zero;
  b.store_all = s.store_all;
  b.cycles = s.cycles;
  b.sweeps = s.sweeps;
  b.last_sweeps = s.last_sweeps;
  b.last_relaxation = s.last_relaxation;
  int at = 0, buffer = 0;
  for (int l = 0; l < s.count; ++l) {  // tables first: 16-byte aligned
    b.lv[l].table_at = at;
    at += 64 * STENCIL_FLOATS;
  }
  for (int l = 0; l < s.count; ++l) {
    ClusterLevel& L = b.lv[l];
    L.info = s.levels[l].info;
    L.q = s.levels[l].q;
    L.rhs = s.levels[l].rhs;
    const int n0 = L.info.dims[0], n1 = L.info.dims[1], n2 = L.info.dims[2];
    L.H = ((n2 + 1) / 2 + 3) / 4 * 4;
    L.uniform = L.info.fill_hi[0] == 1.0f && L.info.fill_hi[1] == 1.0f && L.info.fill_hi[2] == 1.0f;
    L.planes = l < s.single_from ? (n0 + s.ctas - 1) / s.ctas : 0;
    L.by_planes = divider(std::max(L.planes, 1));
    L.by_n1 = divider(n1);
    L.by_n2 = divider(n2);
    L.by_half = divider((n2 + 1) / 2);
    L.by_quads = divider(L.H / 4);
    L.q_at = at;
    at += padded4(L.planes ? 2 * (L.planes + 2) * n1 * L.H : n0 * n1 * n2);
    L.rhs_at = at;
    at += padded4(L.planes ? 2 * L.planes * n1 * L.H : n0 * n1 * n2);
    if (L.planes && l + 1 < s.count) {
      const int32_t* cd = s.levels[l + 1].info.dims;
      buffer = std::max(buffer, std::min(cd[0], L.planes / 2 + 3) * cd[1] * cd[2]);
    }
  }
  b.buffer_at = at;
  b.zero_at = at + padded4(buffer);
  b.floats = b.zero_at + 8;
  return b;
}

bool cluster_solve_single(const PlumeGridInfo& info) {
  return (long)info.dims[0] * info.dims[1] * ((info.dims[2] + 1) / 2) <= CS_THREADS;
}

size_t cluster_solve_bytes(const ClusterSolve& s) {
  size_t floats = 0;  // the same sums as cluster_args, in 64 bits
  for (int l = 0; l < s.count; ++l) {
    const int32_t* d = s.levels[l].info.dims;
    const size_t H = ((d[2] + 1) / 2 + 3) / 4 * 4, planes = l < s.single_from ? (d[0] + s.ctas - 1) / s.ctas : 0;
    floats += planes ? 2 * (2 * planes + 2) * d[1] * H : 2 * (size_t)d[0] * d[1] * d[2];
    floats += 64 * STENCIL_FLOATS;
    if (floats > CS_MAX_SMEM) return (size_t)1 << 40;
  }
  return floats > CS_MAX_SMEM ? (size_t)1 << 40 : sizeof(float) * (size_t)cluster_args(s).floats;
}

static std::mutex g_cluster_mutex;
static bool g_cluster_ready[64] = {};
static bool g_cluster_16[64] = {};  // the device schedules clusters of 16

int prepare_cluster_solve() {
  int device = 0;
  int status = runtime_status("current device", cudaGetDevice(&device));
  if (status != PLUME_OK) return status;
  std::lock_guard<std::mutex> lock(g_cluster_mutex);
  if (device < 0 || device >= 64 || g_cluster_ready[device]) return PLUME_OK;
  status = runtime_status("cluster solve shared memory",
                          cudaFuncSetAttribute(k_cluster_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CS_MAX_SMEM));
  if (status != PLUME_OK) return status;
  if (cudaFuncSetAttribute(k_cluster_solve, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(16);
    config.blockDim = dim3(CS_THREADS);
    config.dynamicSmemBytes = CS_MAX_SMEM;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = 16;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    int clusters = 0;
    g_cluster_16[device] =
        cudaOccupancyMaxActiveClusters(&clusters, k_cluster_solve, &config) == cudaSuccess && clusters >= 1;
  }
  cudaGetLastError();  // a refused attribute or query only means clusters of 8
  g_cluster_ready[device] = true;
  return PLUME_OK;
}

// Whether reciprocal() holds for a level: the approximate division it starts from does for divisors of 2^-126 to 2^126,
// which the coupling sums are in always, cell_volume * cell_m * cell_m for spacings of about 1e-19 to 9e18 m.
static bool spacing_in_range(const PlumeGridInfo& info) {
  const float h2 = info.cell_m * info.cell_m;
  return h2 <= 0x1p126f && info.fill_hi[0] * info.fill_hi[1] * info.fill_hi[2] * info.cell_m * info.cell_m >= 0x1p-126f;
}

bool cluster_solve_runs(const ClusterSolve& s) {
  int device = 0;
  if (s.count < 1 || s.count > CLUSTER_MAX_LEVELS || cluster_solve_bytes(s) > CS_MAX_SMEM) return false;
  for (int l = 0; l < s.count; ++l)
    if (!spacing_in_range(s.levels[l].info) || (l > 0 && !halves(s.levels[l - 1].info, s.levels[l].info))) return false;
  if (s.single_from < s.count && !cluster_solve_single(s.levels[s.single_from].info)) return false;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return false;
  return s.ctas <= 8 || g_cluster_16[device];
}

int launch_cluster_solve(const ClusterSolve& s, bool dependent, cudaStream_t st) {
  const ClusterArgs b = cluster_args(s);
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(s.ctas);
  config.blockDim = dim3(CS_THREADS);
  config.dynamicSmemBytes = sizeof(float) * (size_t)b.floats;
  config.stream = st;
  cudaLaunchAttribute attribute[2];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = s.ctas;
  attribute[0].val.clusterDim.y = 1;
  attribute[0].val.clusterDim.z = 1;
  attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = dependent ? 2 : 1;
  int status = runtime_status("cluster solve", cudaLaunchKernelEx(&config, k_cluster_solve, b));
  if (status != PLUME_OK) return status;
  return launch_status("cluster solve");
}

}  // namespace plume
