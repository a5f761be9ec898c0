// Fused clamped-MacCormack advection for sm_100a: forward trace, backward trace and limiter in one pass.
//
// Reference: advect_maccormack and its kernels (src/plume/sim/advect.py:16-68) with the sampling functions of
// src/plume/sim/sample.py:10-82. The reference makes three full-grid passes per field (semi-Lagrangian into
// `hat`, semi-Lagrangian of `hat` backward into `back`, then the clamped correction) and re-reads the
// velocity for every trace. Here one kernel does all three for the three velocity components, and another for
// smoke and temperature together:
//
// - A block owns a tile of TY x TZ elements in (y, z) and marches along x over a segment of planes. The
//   velocity components (and, for the scalars, smoke and temperature) of the planes the traces can reach are
//   staged in shared memory: a ring of planes, each plane the tile plus two cells on every side, with indices
//   clamped at the array edges (edge replication). Every trilinear sample then reads 8 shared-memory words at
//   fixed offsets from one index.
// - `hat` (the forward semi-Lagrangian value) is computed for the tile plus a one-cell ring in (y, z), one
//   plane ahead of the correction, into a ring of hat planes in shared memory; it never goes to HBM. The
//   correction traces backward and samples that ring, so HBM sees each input read once and `next` written once.
// - A trace is only taken from shared memory when it stays inside the staged planes: |v| dt / dx < REACH at
//   the element and at the midpoint. Otherwise that element's hat, or its backward sample, is evaluated from
//   global memory with the same arithmetic (clamped indices), so results do not depend on which path ran.
//
// Arithmetic: positions, traces and the limiter keep the reference's float operations and their order. The
// trilinear blends use lerp(a, b, t) = fma(t, b - a, a) (one rounding fewer than a*(1-t) + b*t); values agree
// with the reference to about an ulp. With edge replication the lower clamp of each coordinate is the only
// clamp needed: a coordinate above n-1 blends two equal values, which the fma form returns exactly, and the
// min/max range covers the same corner values as range_index_space (sample.py:33-50), whose corners are
// those of the coordinate clamped into [0, n-1].
//
// The smoke budget's line totals (reduce.py:12-25) come out of the scalar march: each thread walks its
// (y, z) line along x and adds data, hat and next in float, per segment; k_segment_lines adds the segments of
// each line in order and the lines in double. Temperature's dissipation (dissipate.py:10-15) is applied as
// it is stored.
#include <algorithm>
#include <cstdlib>

#include "advect.cuh"
#include "march_plan.cuh"
#include "once_per_device.cuh"

namespace plume {
namespace mac {

// Tile height of the scalar march, and rows of threads of the velocity march: 8 (256 threads).
#ifndef PLUME_MAC_TY
#define PLUME_MAC_TY 8
#endif
constexpr int TY = PLUME_MAC_TY, TZ = 32, NT = TY * TZ;   // tile of one block: TY x 32 elements per plane
constexpr int BLOCKS_PER_SM = 1024 / NT;                // 512 threads: 2 blocks per SM, 256: 4
// Plane strides are padded to a multiple of 32 floats, so that samples in neighbouring planes of the same row
// and column fall in the same bank only for the same lane position (planes 720 floats apart would put lanes 16
// columns apart in one bank).
constexpr int pad32(int n) { return (n + 31) / 32 * 32; }
constexpr int RZ = TZ + 4, RY = TY + 4, RP = pad32(RY * RZ);  // staged plane: rows j0-2..j0+TY+1, cols k0-2..k0+TZ+1
constexpr int HZ = TZ + 2, HY = TY + 2, HP = pad32(HY * HZ);  // hat plane: rows j0-1..j0+TY, cols k0-1..k0+TZ
constexpr int HALO = HY * HZ - NT;                        // the hat plane's one-cell ring (84 elements at TY 8)
constexpr int VR = 8;                                     // velocity ring: planes i-1..i+2 in use, i+3 landing
constexpr int SR = 4;                                     // smoke/temperature ring: planes i..i+2, i+3 landing
constexpr int HR = 4;                                     // hat ring: planes i-1..i+1 read, i+2 written next
constexpr float REACH = 0.98f;                            // trace reach (cells) served from shared memory
// Floats after the last hat plane: where a coordinate's rounding step is a sixteenth of a cell or more (axes of 2^19), a
// trace just under REACH ends a whole cell away, and the upper corner, of weight 0, lies one row further.
constexpr int SLACK = HZ + 1;
constexpr int RPN = RY * RZ;                              // staged elements per plane
constexpr int STAGE_PER_THREAD = (RPN + NT - 1) / NT;
// The velocity march's tile: EPT elements per thread, in rows TY apart.
template <int EPT>
struct March {
  static constexpr int tile = EPT * TY, rows = tile + 4, staged = rows * RZ, plane = pad32(staged);  // staged plane
  static constexpr int hat_rows = tile + 2, hat_plane = pad32(hat_rows * HZ), halo = hat_rows * HZ - EPT * NT;
  static constexpr int per_thread = (staged + NT - 1) / NT;
  static constexpr size_t smem = sizeof(float) * (3 * VR * plane + HR * hat_plane + SLACK);
};

__device__ __forceinline__ float lerpm(float a, float b, float t) { return __fmaf_rn(t, b - a, a); }

// One axis of a sample: the coordinate clamped below at 0 (as sample.py's clamp), its floor and fraction.
struct Ax {
  int i;
  float t;
};
__device__ __forceinline__ Ax split(float g) {
  const float x = fmaxf(g, 0.0f);
  const float f = floorf(x);
  return Ax{(int)f, x - f};
}

// The 8 corners in the order a[dx + 2 dy + 4 dz].
__device__ __forceinline__ float blend8(const float* a, float tx, float ty, float tz) {
  const float c00 = lerpm(a[0], a[1], tx), c10 = lerpm(a[2], a[3], tx);
  const float c01 = lerpm(a[4], a[5], tx), c11 = lerpm(a[6], a[7], tx);
  return lerpm(lerpm(c00, c10, ty), lerpm(c01, c11, ty), tz);
}

__device__ __forceinline__ void range8(const float* a, float& lo, float& hi) {
  lo = fminf(fminf(fminf(a[0], a[1]), fminf(a[2], a[3])), fminf(fminf(a[4], a[5]), fminf(a[6], a[7])));
  hi = fmaxf(fmaxf(fmaxf(a[0], a[1]), fmaxf(a[2], a[3])), fmaxf(fmaxf(a[4], a[5]), fmaxf(a[6], a[7])));
}

// Corners from a ring of R staged planes; `inplane` = y * RZ + z - rowbase (the staged row and column).
template <int R, int S>
__device__ __forceinline__ void ring_corners(const float* ring, int x, int inplane, float* a) {
  const float* p0 = ring + (x & (R - 1)) * S + inplane;
  const float* p1 = ring + ((x + 1) & (R - 1)) * S + inplane;
  a[0] = p0[0];
  a[1] = p1[0];
  a[2] = p0[RZ];
  a[3] = p1[RZ];
  a[4] = p0[1];
  a[5] = p1[1];
  a[6] = p0[RZ + 1];
  a[7] = p1[RZ + 1];
}

// Corners from global memory, indices clamped to the array as sample.py does.
template <class T>
__device__ __forceinline__ void global_corners(const T* __restrict__ f, const Dims& d, int x, int y, int z, float* a) {
  // clamped before the step up: a coordinate beyond the int range has the largest int as its floor
  const int x0 = imin_(x, d.n0 - 1), x1 = imin_(x0 + 1, d.n0 - 1);
  const int y0 = imin_(y, d.n1 - 1), y1 = imin_(y0 + 1, d.n1 - 1);
  const int z0 = imin_(z, d.n2 - 1), z1 = imin_(z0 + 1, d.n2 - 1);
  a[0] = ldg_f(f + at(d, x0, y0, z0));
  a[1] = ldg_f(f + at(d, x1, y0, z0));
  a[2] = ldg_f(f + at(d, x0, y1, z0));
  a[3] = ldg_f(f + at(d, x1, y1, z0));
  a[4] = ldg_f(f + at(d, x0, y0, z1));
  a[5] = ldg_f(f + at(d, x1, y0, z1));
  a[6] = ldg_f(f + at(d, x0, y1, z1));
  a[7] = ldg_f(f + at(d, x1, y1, z1));
}

template <class T>
struct Args {
  PlumeGridInfo info;
  const T* vel[3];      // u, v, w: the velocity the traces follow (and, for G < 3, the advected field)
  const T* field[2];    // smoke, temperature (the scalar march)
  T* next[3];           // u, v, w next (velocity march) or smoke, temperature next (scalar march)
  float outside[2];     // the scalars' values beyond open faces
  int uses_outside;
  float dt;             // dt / cell_m
  int seg_len;          // planes per block along x
  int segs[4];          // segments per group (u, v, w; or the cells)
  float* partials;      // scalar march: float line sums [3][segs][ny * nz] (data, hat, next of smoke)
  int dissipate;        // scalar march: temperature = ambient + (T - ambient) * heat_keep on store
  float heat_keep, ambient;
};

// Position offset of group G's elements (u, v, w faces; 3 = cell centres).
template <int G>
__device__ __forceinline__ F3 offset_of() {
  return f3(G == 0 ? 0.0f : 0.5f, G == 1 ? 0.0f : 0.5f, G == 2 ? 0.0f : 0.5f);
}

__device__ __forceinline__ Dims group_dims(const PlumeGridInfo& info, int g) {
  return Dims{info.dims[0] + (g == 0), info.dims[1] + (g == 1), info.dims[2] + (g == 2)};
}

// Whether a trace by this velocity stays inside the staged planes: every component, each compared by itself, so that one
// that is no number does not (a maximum would pass over it, and its coordinate's index would leave the ring).
__device__ __forceinline__ bool within_reach(F3 v, float dt) {
  return fabsf(v[0]) * dt < REACH && fabsf(v[1]) * dt < REACH && fabsf(v[2]) * dt < REACH;
}

// ---- velocity at a point (sample.py:74-82), from the staged ring or from global memory --------------------
// The three components' axes are split once: x of v and w, y of u and w, z of u and v are the same
// coordinate minus 1/2.
template <int S>
__device__ __forceinline__ F3 ring_velocity(const float* vring, int rowbase, F3 m) {
  const Ax x0 = split(m[0]), x1 = split(m[0] - 0.5f);
  const Ax y0 = split(m[1]), y1 = split(m[1] - 0.5f);
  const Ax z0 = split(m[2]), z1 = split(m[2] - 0.5f);
  float a[8];
  ring_corners<VR, S>(vring, x0.i, y1.i * RZ + z1.i - rowbase, a);
  const float u = blend8(a, x0.t, y1.t, z1.t);
  ring_corners<VR, S>(vring + VR * S, x1.i, y0.i * RZ + z1.i - rowbase, a);
  const float v = blend8(a, x1.t, y0.t, z1.t);
  ring_corners<VR, S>(vring + 2 * VR * S, x1.i, y1.i * RZ + z0.i - rowbase, a);
  const float w = blend8(a, x1.t, y1.t, z0.t);
  return f3(u, v, w);
}

template <class T>
__device__ __forceinline__ F3 global_velocity(const Args<T>& A, F3 m) {
  const int nx = A.info.dims[0], ny = A.info.dims[1], nz = A.info.dims[2];
  const Ax x0 = split(m[0]), x1 = split(m[0] - 0.5f);
  const Ax y0 = split(m[1]), y1 = split(m[1] - 0.5f);
  const Ax z0 = split(m[2]), z1 = split(m[2] - 0.5f);
  float a[8];
  global_corners(A.vel[0], Dims{nx + 1, ny, nz}, x0.i, y1.i, z1.i, a);
  const float u = blend8(a, x0.t, y1.t, z1.t);
  global_corners(A.vel[1], Dims{nx, ny + 1, nz}, x1.i, y0.i, z1.i, a);
  const float v = blend8(a, x1.t, y0.t, z1.t);
  global_corners(A.vel[2], Dims{nx, ny, nz + 1}, x1.i, y1.i, z0.i, a);
  const float w = blend8(a, x1.t, y1.t, z0.t);
  return f3(u, v, w);
}

// ---- velocity at an element's own position (velocity_at at p = index + offset) ----------------------------
// Each component's trilinear weights there are 0 or 1/2: the component sampled on its own faces is read
// directly; for the others, the axis of the component sits half a cell above (corners c, c+1) and the axis of
// the element's group half a cell below (corners c-1, c), blended at 1/2 in the reference's axis order.
// Cells: each component sits half a cell above along its own axis. At the walls the clamp of sample.py keeps
// one corner; the staged ring's edge replication and the global path's clamped indices both give that value.
template <int G, int C>
struct Node {
  // direction of the half-cell shift of component C's sample along each axis: +1 above, -1 below, 0 none
  static constexpr int shift(int axis) {
    return G == 3 ? (axis == C ? 1 : 0) : (G == C ? 0 : (axis == C ? 1 : (axis == G ? -1 : 0)));
  }
  static constexpr int sx = shift(0), sy = shift(1), sz = shift(2);
};

// blend of one component at the element from a corner accessor load(dx, dy, dz)
template <int G, int C, class Load>
__device__ __forceinline__ float node_component(Load load) {
  using N = Node<G, C>;
  constexpr int ax0 = N::sx < 0 ? -1 : 0, ax1 = N::sx > 0 ? 1 : 0;
  constexpr int ay0 = N::sy < 0 ? -1 : 0, ay1 = N::sy > 0 ? 1 : 0;
  constexpr int az0 = N::sz < 0 ? -1 : 0, az1 = N::sz > 0 ? 1 : 0;
  auto along_x = [&](int dy, int dz) {
    const float a = load(ax0, dy, dz);
    if constexpr (N::sx == 0) return a;
    else return lerpm(a, load(ax1, dy, dz), 0.5f);
  };
  auto along_y = [&](int dz) {
    const float c0 = along_x(ay0, dz);
    if constexpr (N::sy == 0) return c0;
    else return lerpm(c0, along_x(ay1, dz), 0.5f);
  };
  const float y0 = along_y(az0);
  if constexpr (N::sz == 0) return y0;
  else return lerpm(y0, along_y(az1), 0.5f);
}

// The velocity ring's plane stride: padded to a multiple of 32 floats in the velocity march; the scalar march
// keeps it unpadded so that two blocks still fit in one SM's shared memory.
template <int G>
struct Stride {
  static constexpr int value = G == 3 ? RPN : RP;
};

template <int G, int S = Stride<G>::value>
__device__ __forceinline__ F3 ring_node(const float* vring, int x, int inplane) {
  auto ring = [&](const float* r) {
    return [=](int dx, int dy, int dz) { return r[((x + dx) & (VR - 1)) * S + inplane + dy * RZ + dz]; };
  };
  return f3(node_component<G, 0>(ring(vring)), node_component<G, 1>(ring(vring + VR * S)),
            node_component<G, 2>(ring(vring + 2 * VR * S)));
}

template <int G, class T>
__device__ __forceinline__ F3 global_node(const Args<T>& A, int x, int y, int z) {
  const int nx = A.info.dims[0], ny = A.info.dims[1], nz = A.info.dims[2];
  auto global = [&](const T* f, Dims d) {
    return [=](int dx, int dy, int dz) {
      const int a = imin_(imax_(x + dx, 0), d.n0 - 1), b = imin_(imax_(y + dy, 0), d.n1 - 1);
      const int c = imin_(imax_(z + dz, 0), d.n2 - 1);
      return ldg_f(f + at(d, a, b, c));
    };
  };
  return f3(node_component<G, 0>(global(A.vel[0], Dims{nx + 1, ny, nz})),
            node_component<G, 1>(global(A.vel[1], Dims{nx, ny + 1, nz})),
            node_component<G, 2>(global(A.vel[2], Dims{nx, ny, nz + 1})));
}

// ---- the forward (semi-Lagrangian) value and its clamp range at one element --------------------------------
template <int G>
struct Fields {
  static constexpr int count = G == 3 ? 2 : 1;
};

// Evaluated from global memory: the whole trace, every sample through clamped indices.
template <int G, class T>
__device__ __noinline__ void hat_global(const Args<T>& A, int x, int y, int z, float* hat, float* lo, float* hi) {
  constexpr int F = Fields<G>::count;
  const F3 off = offset_of<G>();
  const F3 p = add3(f3((float)x, (float)y, (float)z), off);
  const F3 vp = global_node<G>(A, x, y, z);
  const F3 mid = sub3(p, mul3(vp, 0.5f * A.dt));
  const F3 src = sub3(p, mul3(global_velocity(A, mid), A.dt));
  const bool outside = G == 3 && A.uses_outside == 1 && is_outside_open_face(src, A.info);
  const F3 g = sub3(src, off);
  const Ax gx = split(g[0]), gy = split(g[1]), gz = split(g[2]);
  for (int f = 0; f < F; ++f) {
    if (outside) {
      hat[f] = lo[f] = hi[f] = A.outside[f];
      continue;
    }
    float a[8];
    const T* src_field = G == 3 ? A.field[f] : A.vel[G];
    global_corners(src_field, group_dims(A.info, G), gx.i, gy.i, gz.i, a);
    hat[f] = blend8(a, gx.t, gy.t, gz.t);
    range8(a, lo[f], hi[f]);
  }
}

// From the staged rings when the trace stays inside them, else hat_global.
template <int G, class T>
__device__ __forceinline__ void hat_at(const Args<T>& A, const float* vring, const float* sring, int rowbase, int x, int y,
                                       int z, float* hat, float* lo, float* hi) {
  constexpr int F = Fields<G>::count;
  const F3 off = offset_of<G>();
  const F3 p = add3(f3((float)x, (float)y, (float)z), off);
  const int inplane = y * RZ + z - rowbase;
  const F3 vp = ring_node<G>(vring, x, inplane);
  bool fast = within_reach(vp, fabsf(A.dt));
  F3 src = p;
  if (fast) {
    const F3 mid = sub3(p, mul3(vp, 0.5f * A.dt));
    const F3 vm = ring_velocity<Stride<G>::value>(vring, rowbase, mid);
    fast = within_reach(vm, fabsf(A.dt));
    src = sub3(p, mul3(vm, A.dt));
  }
  if (!fast) {
    hat_global<G>(A, x, y, z, hat, lo, hi);
    return;
  }
  const bool outside = G == 3 && A.uses_outside == 1 && is_outside_open_face(src, A.info);
  const F3 g = sub3(src, off);
  const Ax gx = split(g[0]), gy = split(g[1]), gz = split(g[2]);
  const int gin = gy.i * RZ + gz.i - rowbase;
#pragma unroll
  for (int f = 0; f < F; ++f) {
    if (outside) {
      hat[f] = lo[f] = hi[f] = A.outside[f];
      continue;
    }
    float a[8];
    if constexpr (G == 3) ring_corners<SR, RPN>(sring + f * SR * RPN, gx.i, gin, a);
    else ring_corners<VR, RP>(vring + G * VR * RP, gx.i, gin, a);
    hat[f] = blend8(a, gx.t, gy.t, gz.t);
    range8(a, lo[f], hi[f]);
  }
}

// ---- the backward sample of hat (the reference's `back`) ---------------------------------------------------
// From the hat ring when the backward trace stays inside it, else each corner's hat from wherever it is: the
// ring for corners inside the staged hat planes, hat_global for the rest.
template <int G, int ROWS, int PLANE, class T>
__device__ __noinline__ void back_global(const Args<T>& A, const float* hring, int hbase, int j0, int k0, int plane_lo,
                                         int x, int y, int z, float* back) {
  constexpr int F = Fields<G>::count;
  const F3 off = offset_of<G>();
  const Dims gd = group_dims(A.info, G);
  const F3 p = add3(f3((float)x, (float)y, (float)z), off);
  const F3 vp = global_node<G>(A, x, y, z);
  const F3 mid = sub3(p, mul3(vp, 0.5f * -A.dt));
  const F3 bsrc = sub3(p, mul3(global_velocity(A, mid), -A.dt));
  if (G == 3 && A.uses_outside == 1 && is_outside_open_face(bsrc, A.info)) {
    for (int f = 0; f < F; ++f) back[f] = A.outside[f];
    return;
  }
  const F3 g = sub3(bsrc, off);
  const Ax gx = split(g[0]), gy = split(g[1]), gz = split(g[2]);
  float a[F][8];
  for (int c = 0; c < 8; ++c) {
    const int cx = imin_(imin_(gx.i, gd.n0 - 1) + (c & 1), gd.n0 - 1);
    const int cy = imin_(imin_(gy.i, gd.n1 - 1) + ((c >> 1) & 1), gd.n1 - 1);
    const int cz = imin_(imin_(gz.i, gd.n2 - 1) + (c >> 2), gd.n2 - 1);
    const bool staged = cx >= plane_lo && cx <= plane_lo + 2 && cy >= j0 - 1 && cy <= j0 + ROWS && cz >= k0 - 1 &&
                        cz <= k0 + TZ;
    if (staged) {
      for (int f = 0; f < F; ++f) a[f][c] = hring[(f * HR + (cx & (HR - 1))) * PLANE + cy * HZ + cz - hbase];
    } else {
      float h[F], lo[F], hi[F];
      hat_global<G>(A, cx, cy, cz, h, lo, hi);
      for (int f = 0; f < F; ++f) a[f][c] = h[f];
    }
  }
  for (int f = 0; f < F; ++f) back[f] = blend8(a[f], gx.t, gy.t, gz.t);
}

// ---- staging ------------------------------------------------------------------------------------------------
// Each thread stages the plane elements e = t, t + NT, ... (while e < RPN); its offsets inside a plane of each
// array shape are fixed for the whole march.
struct StageOffsets {
  int off[3][STAGE_PER_THREAD];  // per array shape: u and the cells share (ny, nz); v (ny+1, nz); w (ny, nz+1)
};

template <class T>
__device__ __forceinline__ void stage_plane(const T* __restrict__ src, const Dims& d, int shape, int plane,
                                            float* ring_plane, const StageOffsets& so) {
  const int pc = imin_(imax_(plane, 0), d.n0 - 1);
  const T* base = src + (size_t)pc * d.n1 * d.n2;
#pragma unroll
  for (int n = 0; n < STAGE_PER_THREAD; ++n) {
    const int e = threadIdx.x + n * NT;
    if (e < RPN) {
      if constexpr (sizeof(T) == 4) {
        const unsigned dst = (unsigned)__cvta_generic_to_shared(ring_plane + e);
        const size_t from = __cvta_generic_to_global(base + so.off[shape][n]);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(from));
      } else {
        ring_plane[e] = ldg_f(base + so.off[shape][n]);
      }
    }
  }
}

__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// ---- the march -----------------------------------------------------------------------------------------------
template <class T, int G>
__device__ __forceinline__ void march(const Args<T>& A, int seg, float* sm) {
  constexpr int F = Fields<G>::count;
  const int nx = A.info.dims[0], ny = A.info.dims[1], nz = A.info.dims[2];
  const Dims gd = group_dims(A.info, G);
  const int k0 = blockIdx.x * TZ, j0 = blockIdx.y * TY;
  if (j0 >= gd.n1 || k0 >= gd.n2) return;  // a tile past this group's extent (the v and w end rows)
  const int s = seg * A.seg_len;
  if (s >= gd.n0) return;
  const int e = imin_(s + A.seg_len, gd.n0);

  constexpr int VS = Stride<G>::value;                 // velocity ring plane stride
  float* vring = sm;                                  // [3][VR][VS]
  float* sring = vring + 3 * VR * VS;                 // [2][SR][RPN] (scalar march)
  float* hring = sring + (G == 3 ? 2 * SR * RPN : 0);  // [F][HR][HP]
  const int t = threadIdx.x, ty = t / TZ, tz = t % TZ;
  const int rowbase = (j0 - 2) * RZ + (k0 - 2), hbase = (j0 - 1) * HZ + (k0 - 1);

  // staging offsets inside one plane of each array shape (edge-clamped)
  StageOffsets so;
  {
    const Dims shapes[3] = {Dims{0, ny, nz}, Dims{0, ny + 1, nz}, Dims{0, ny, nz + 1}};
#pragma unroll
    for (int sh = 0; sh < 3; ++sh)
#pragma unroll
      for (int n = 0; n < STAGE_PER_THREAD; ++n) {
        const int el = imin_(t + n * NT, RPN - 1), r = el / RZ, q = el % RZ;
        const int y = imin_(imax_(j0 - 2 + r, 0), shapes[sh].n1 - 1);
        const int z = imin_(imax_(k0 - 2 + q, 0), shapes[sh].n2 - 1);
        so.off[sh][n] = y * shapes[sh].n2 + z;
      }
  }
  const Dims vd[3] = {Dims{nx + 1, ny, nz}, Dims{nx, ny + 1, nz}, Dims{nx, ny, nz + 1}};
  const Dims cd{nx, ny, nz};
  auto stage_velocity = [&](int plane) {
#pragma unroll
    for (int c = 0; c < 3; ++c) stage_plane(A.vel[c], vd[c], c, plane, vring + (c * VR + (plane & (VR - 1))) * VS, so);
  };
  auto stage_scalars = [&](int plane) {
    if constexpr (G == 3) {
#pragma unroll
      for (int f = 0; f < 2; ++f) stage_plane(A.field[f], cd, 0, plane, sring + (f * SR + (plane & (SR - 1))) * RPN, so);
    }
  };

  // this thread's tile element, and its element of the hat plane's ring (t < HALO)
  const int tj = j0 + ty, tk = k0 + tz;
  const bool valid = tj < gd.n1 && tk < gd.n2;
  const int cj = imin_(tj, gd.n1 - 1), ck = imin_(tk, gd.n2 - 1);
  int hj, hk;  // position in the hat plane (0..HY-1, 0..HZ-1)
  if (t < HZ) {
    hj = 0;
    hk = t;
  } else if (t < 2 * HZ) {
    hj = HY - 1;
    hk = t - HZ;
  } else if (t < 2 * HZ + TY) {
    hj = 1 + t - 2 * HZ;
    hk = 0;
  } else {
    hj = 1 + t - 2 * HZ - TY;
    hk = HZ - 1;
  }
  const bool has_halo = t < HALO;
  const int rj = imin_(imax_(j0 - 1 + hj, 0), gd.n1 - 1), rk = imin_(imax_(k0 - 1 + hk, 0), gd.n2 - 1);
  const int tile_h = (ty + 1) * HZ + (tz + 1), ring_h = hj * HZ + hk;

  float range_lo[F], range_hi[F], own_hat[F];
  float sum_data = 0.0f, sum_hat = 0.0f, sum_next = 0.0f;

  // The hat plane x (clamped to the array), this thread's two elements; the tile element's range and hat
  // are kept for its correction.
  auto hat_plane = [&](int x, float* keep_lo, float* keep_hi, float* keep_hat) {
    const int xc = imin_(imax_(x, 0), gd.n0 - 1);
    float h[F], lo[F], hi[F];
    hat_at<G>(A, vring, sring, rowbase, xc, cj, ck, h, lo, hi);
#pragma unroll
    for (int f = 0; f < F; ++f) {
      hring[(f * HR + (x & (HR - 1))) * HP + tile_h] = h[f];
      keep_lo[f] = lo[f];
      keep_hi[f] = hi[f];
      keep_hat[f] = h[f];
    }
    if (has_halo) {
      hat_at<G>(A, vring, sring, rowbase, xc, rj, rk, h, lo, hi);
#pragma unroll
      for (int f = 0; f < F; ++f) hring[(f * HR + (x & (HR - 1))) * HP + ring_h] = h[f];
    }
  };
  // hat plane `to` copied from plane `from` (the array's edge planes, replicated); each thread copies the
  // elements it wrote itself
  auto copy_hat_plane = [&](int from, int to) {
#pragma unroll
    for (int f = 0; f < F; ++f) {
      hring[(f * HR + (to & (HR - 1))) * HP + tile_h] = hring[(f * HR + (from & (HR - 1))) * HP + tile_h];
      if (has_halo) hring[(f * HR + (to & (HR - 1))) * HP + ring_h] = hring[(f * HR + (from & (HR - 1))) * HP + ring_h];
    }
  };

  // prologue: planes s-2..s+2 of the velocity (and s-2..s+1 of the scalars), hat planes s-1 and s
  for (int p = s - 2; p <= s + 2; ++p) stage_velocity(p);
  for (int p = s - 2; p <= s + 1; ++p) stage_scalars(p);
  stage_commit();
  stage_wait();
  __syncthreads();
  {
    float lo[F], hi[F], h[F];
    if (s == 0) {
      hat_plane(0, range_lo, range_hi, own_hat);
      copy_hat_plane(0, -1);
    } else {
      hat_plane(s - 1, lo, hi, h);
      hat_plane(s, range_lo, range_hi, own_hat);
    }
  }
  if (G == 3) {
    __syncthreads();  // the scalar ring's slot of plane s-2 is free
    stage_scalars(s + 2);
    stage_commit();
    stage_wait();
  }
  if (G == 3 && valid) sum_hat = own_hat[0];
  __syncthreads();

  const size_t plane_stride = (size_t)gd.n1 * gd.n2;
  for (int i = s; i < e; ++i) {
    // planes i+3 start landing while hat plane i+1 is computed
    stage_velocity(i + 3);
    stage_scalars(i + 3);
    stage_commit();
    float next_lo[F] = {}, next_hi[F] = {}, next_hat[F] = {};
    if (i + 1 <= gd.n0 - 1) {
      hat_plane(i + 1, next_lo, next_hi, next_hat);
      if (G == 3 && valid && i + 1 < e) sum_hat += next_hat[0];
    } else {
      copy_hat_plane(i, i + 1);
    }
    stage_wait();
    __syncthreads();

    if (valid) {
      // the correction (advect.py:34-50, 64): back = hat sampled along the backward trace
      const F3 off = offset_of<G>();
      const F3 p = add3(f3((float)i, (float)tj, (float)tk), off);
      const int inplane = tj * RZ + tk - rowbase;
      const F3 vp = ring_node<G>(vring, i, inplane);
      bool fast = within_reach(vp, fabsf(A.dt));
      float back[F];
      if (fast) {
        const F3 mid = sub3(p, mul3(vp, 0.5f * -A.dt));
        const F3 vm = ring_velocity<VS>(vring, rowbase, mid);
        fast = within_reach(vm, fabsf(A.dt));
        if (fast) {
          const F3 bsrc = sub3(p, mul3(vm, -A.dt));
          if (G == 3 && A.uses_outside == 1 && is_outside_open_face(bsrc, A.info)) {
#pragma unroll
            for (int f = 0; f < F; ++f) back[f] = A.outside[f];
          } else {
            const F3 g = sub3(bsrc, off);
            const Ax gx = split(g[0]), gy = split(g[1]), gz = split(g[2]);
            const int gin = gy.i * HZ + gz.i - hbase;
#pragma unroll
            for (int f = 0; f < F; ++f) {
              const float* h0 = hring + (f * HR + (gx.i & (HR - 1))) * HP + gin;
              const float* h1 = hring + (f * HR + ((gx.i + 1) & (HR - 1))) * HP + gin;
              const float a[8] = {h0[0], h1[0], h0[HZ], h1[HZ], h0[1], h1[1], h0[HZ + 1], h1[HZ + 1]};
              back[f] = blend8(a, gx.t, gy.t, gz.t);
            }
          }
        }
      }
      if (!fast) back_global<G, TY, HP>(A, hring, hbase, j0, k0, i - 1, i, tj, tk, back);
      const size_t out = (size_t)i * plane_stride + (size_t)tj * gd.n2 + tk;
#pragma unroll
      for (int f = 0; f < F; ++f) {
        const float data = G == 3 ? ldg_f(A.field[f] + out) : vring[(G * VR + (i & (VR - 1))) * VS + inplane];
        const float corrected = own_hat[f] + 0.5f * (data - back[f]);
        float value = clampf_(corrected, range_lo[f], range_hi[f]);
        if (G == 3 && f == 0) {
          sum_data += data;
          sum_next += value;
        }
        if (G == 3 && f == 1 && A.dissipate) value = A.ambient + (to_f<T>(from_f<T>(value)) - A.ambient) * A.heat_keep;
        st_f(A.next[G == 3 ? f : G] + out, value);
      }
    }
#pragma unroll
    for (int f = 0; f < F; ++f) {
      range_lo[f] = next_lo[f];
      range_hi[f] = next_hi[f];
      own_hat[f] = next_hat[f];
    }
  }
  if (G == 3 && valid) {
    const size_t lines = (size_t)ny * nz, line = (size_t)tj * nz + tk;
    const int segs = A.segs[3];
    A.partials[(size_t)(0 * segs + seg) * lines + line] = sum_data;
    A.partials[(size_t)(1 * segs + seg) * lines + line] = sum_hat;
    A.partials[(size_t)(2 * segs + seg) * lines + line] = sum_next;
  }
}

// ---- the velocity march -----------------------------------------------------------------------------------------
// One component (G) of the velocity by itself. The forward and the backward trace of an element start from the same
// velocity and step half a cell either way, so both midpoint velocities are formed together when the element's hat
// is, each operation once for the pair (two-wide fused multiply-adds: lane 0 forward, lane 1 backward, each lane the
// scalar operation), and the backward trace's end point is kept until the correction of that plane, which then needs
// only the hat ring. Coordinates are split into index and fraction by adding 2^23 rounding down, on the float adders
// instead of the conversion unit.
//
// Elements whose trace leaves the staged planes (|velocity| dt >= REACH cells) compute with a zero velocity, to keep
// every index inside the rings, and are evaluated from global memory after the block has met, if any thread has one:
// one uniform branch per plane instead of two per element.
//
// Bound by shared-memory wavefronts (65% of their peak at 128x192x128, four in ten of them bank conflicts of lanes whose
// samples lie in different rows or planes) and instruction issue (64%; about 710 instructions for 32 elements). Measured on B200,
// velocity advection with the traces formed one after the other, the backward one in its plane's step, against this:
// 38x48x38 46 and 27 us, 64x96x64 84 and 59 us, 128x192x128 356 and 295 us, 256x384x256 2245 and 1975 us. Planes arrive
// through registers: 4-byte asynchronous copies took five wavefronts each (2140 us against 2080 us at 256x384x256).
// Rejected: rows 256 floats apart with a row's four planes side by side, so that rows and planes share banks (2496 us).
constexpr float TWO23 = 8388608.0f;

// A sample's coordinate: `bits` is its floor plus the constant bits of 2^23 (wrap-around cancels it in an index whose base
// subtracts SPLIT_BITS), and t its fraction. Coordinates lie in [0, 2^22).
constexpr int SPLIT_BITS = 0x4B000000;
struct AxBits {
  int bits;
  float t;
};
__device__ __forceinline__ AxBits split_bits(float g) {
  const float x = fmaxf(g, 0.0f);
  const float shifted = __fadd_rd(x, TWO23);
  return AxBits{__float_as_int(shifted), x - (shifted - TWO23)};
}

__device__ __forceinline__ float2 lerp2(float2 a, float2 b, float2 t) {  // lerpm in each lane: b - a as fma(a, -1, b)
  return __ffma2_rn(t, __ffma2_rn(a, make_float2(-1.0f, -1.0f), b), a);
}

// The staged planes' float offsets of a sample's lower corner in the planes x and x + 1.
struct RingAt {
  int lo, hi;
};
template <int PLANE>
__device__ __forceinline__ RingAt ring_at(int x_bits, int y_bits, int z_bits, int row_base) {
  const int inplane = y_bits * RZ + z_bits - row_base;  // row_base holds SPLIT_BITS * (RZ + 1)
  return RingAt{(x_bits & (VR - 1)) * PLANE + inplane, ((x_bits + 1) & (VR - 1)) * PLANE + inplane};
}

// blend8's operations for two samples at once, of the component whose ring starts at `ring`.
__device__ __forceinline__ float2 blend_pair(const float* ring, const RingAt& f, const RingAt& b, float2 tx, float2 ty, float2 tz) {
  auto corner = [&](int at_f, int at_b, int step) { return make_float2(ring[at_f + step], ring[at_b + step]); };
  const float2 c00 = lerp2(corner(f.lo, b.lo, 0), corner(f.hi, b.hi, 0), tx);
  const float2 c10 = lerp2(corner(f.lo, b.lo, RZ), corner(f.hi, b.hi, RZ), tx);
  const float2 c01 = lerp2(corner(f.lo, b.lo, 1), corner(f.hi, b.hi, 1), tx);
  const float2 c11 = lerp2(corner(f.lo, b.lo, RZ + 1), corner(f.hi, b.hi, RZ + 1), tx);
  return lerp2(lerp2(c00, c10, ty), lerp2(c01, c11, ty), tz);
}

__device__ __forceinline__ void ring_corners_at(const float* ring, const RingAt& r, float* a) {
  a[0] = ring[r.lo];
  a[1] = ring[r.hi];
  a[2] = ring[r.lo + RZ];
  a[3] = ring[r.hi + RZ];
  a[4] = ring[r.lo + 1];
  a[5] = ring[r.hi + 1];
  a[6] = ring[r.lo + RZ + 1];
  a[7] = ring[r.hi + RZ + 1];
}

__device__ __forceinline__ F3 zero_unless(bool keep, F3 v) { return f3(keep ? v[0] : 0.0f, keep ? v[1] : 0.0f, keep ? v[2] : 0.0f); }

template <class T, int G, int EPT>
__device__ __forceinline__ void velocity_march(const Args<T>& A, int seg, float* sm) {
  const int nx = A.info.dims[0], ny = A.info.dims[1], nz = A.info.dims[2];
  using M = March<EPT>;
  constexpr int VRP = M::plane, VHP = M::hat_plane;
  const Dims gd = group_dims(A.info, G);
  const int k0 = blockIdx.x * TZ, j0 = blockIdx.y * M::tile;
  if (j0 >= gd.n1 || k0 >= gd.n2) return;  // a tile past this group's extent (the v and w end rows)
  const int s = seg * A.seg_len;
  if (s >= gd.n0) return;
  const int e = imin_(s + A.seg_len, gd.n0);

  float* vring = sm;                   // [3][VR][VRP]
  float* hring = vring + 3 * VR * VRP;  // [HR][VHP]
  const int t = threadIdx.x, ty = t / TZ, tz = t % TZ;
  const int rowbase = (j0 - 2) * RZ + (k0 - 2), hbase = (j0 - 1) * HZ + (k0 - 1);
  const int bits_rowbase = (int)((unsigned)rowbase + (unsigned)SPLIT_BITS * (RZ + 1));
  const int bits_hbase = (int)((unsigned)hbase + (unsigned)SPLIT_BITS * (HZ + 1));

  // staging offsets inside one plane of each component (edge-clamped)
  int from[3][M::per_thread];
#pragma unroll
  for (int n = 0; n < M::per_thread; ++n) {
    const int el = imin_(t + n * NT, M::staged - 1), r = el / RZ, q = el % RZ;
#pragma unroll
    for (int c = 0; c < 3; ++c)
      from[c][n] = imin_(imax_(j0 - 2 + r, 0), ny + (c == 1) - 1) * (nz + (c == 2)) + imin_(imax_(k0 - 2 + q, 0), nz + (c == 2) - 1);
  }
  const Dims vd[3] = {Dims{nx + 1, ny, nz}, Dims{nx, ny + 1, nz}, Dims{nx, ny, nz + 1}};
  // plane `plane` of the three components: loaded into registers, and later stored into the rings' slot
  float landing[3][M::per_thread];
  auto fetch = [&](int plane) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const T* base = A.vel[c] + (size_t)imin_(imax_(plane, 0), vd[c].n0 - 1) * vd[c].n1 * vd[c].n2;
#pragma unroll
      for (int n = 0; n < M::per_thread; ++n) landing[c][n] = ldg_f(base + from[c][n]);
    }
  };
  auto land = [&](int plane) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int n = 0; n < M::per_thread; ++n)
        if (t + n * NT < M::staged) vring[(c * VR + (plane & (VR - 1))) * VRP + t + n * NT] = landing[c][n];
  };

  // this thread's tile elements (rows j0 + ty + TY n), and its element of the hat plane's ring (t < M::halo)
  const int tk = k0 + tz, ck = imin_(tk, gd.n2 - 1);
  int hj, hk;  // position in the hat plane (0..HY-1, 0..HZ-1)
  if (t < HZ) {
    hj = 0;
    hk = t;
  } else if (t < 2 * HZ) {
    hj = M::hat_rows - 1;
    hk = t - HZ;
  } else if (t < 2 * HZ + M::tile) {
    hj = 1 + t - 2 * HZ;
    hk = 0;
  } else {
    hj = 1 + t - 2 * HZ - M::tile;
    hk = HZ - 1;
  }
  const bool has_halo = t < M::halo;
  const int rj = imin_(imax_(j0 - 1 + hj, 0), gd.n1 - 1), rk = imin_(imax_(k0 - 1 + hk, 0), gd.n2 - 1);
  const int tile_h = (ty + 1) * HZ + (tz + 1), ring_h = hj * HZ + hk;
  const F3 off = offset_of<G>();
  const float half = 0.5f * A.dt, reach_dt = fabsf(A.dt);

  // what the correction of a plane needs of this thread's element
  struct Kept {
    float lo, hi, hat, data;
    F3 back;      // the backward sample's index-space coordinates
    bool global;  // the backward sample is to be taken from global memory
  };

  // The tile element's hat in plane x (an array plane), and what its correction needs; returns whether its hat is to be
  // taken from global memory.
  auto tile_hat = [&](int x, int slot, int n, Kept& kept) -> bool {
    const int cj = imin_(j0 + ty + n * TY, gd.n1 - 1);
    const F3 p = add3(f3((float)x, (float)cj, (float)ck), off);
    const F3 node = ring_node<G, VRP>(vring, x, cj * RZ + ck - rowbase);
    const bool near = within_reach(node, reach_dt);
    const F3 vp = zero_unless(near, node);
    const F3 step = mul3(vp, half);
    float2 m[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) m[a] = make_float2(p[a] - step[a], p[a] + step[a]);
    AxBits whole_f[3], whole_b[3], face_f[3], face_b[3];  // at m and at m - 1/2
    float2 tw[3], tf[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      whole_f[a] = split_bits(m[a].x);
      whole_b[a] = split_bits(m[a].y);
      face_f[a] = split_bits(m[a].x - 0.5f);
      face_b[a] = split_bits(m[a].y - 0.5f);
      tw[a] = make_float2(whole_f[a].t, whole_b[a].t);
      tf[a] = make_float2(face_f[a].t, face_b[a].t);
    }
    const float2 u = blend_pair(vring, ring_at<VRP>(whole_f[0].bits, face_f[1].bits, face_f[2].bits, bits_rowbase),
                                ring_at<VRP>(whole_b[0].bits, face_b[1].bits, face_b[2].bits, bits_rowbase), tw[0], tf[1], tf[2]);
    const float2 v = blend_pair(vring + VR * VRP, ring_at<VRP>(face_f[0].bits, whole_f[1].bits, face_f[2].bits, bits_rowbase),
                                ring_at<VRP>(face_b[0].bits, whole_b[1].bits, face_b[2].bits, bits_rowbase), tf[0], tw[1], tf[2]);
    const float2 w = blend_pair(vring + 2 * VR * VRP, ring_at<VRP>(face_f[0].bits, face_f[1].bits, whole_f[2].bits, bits_rowbase),
                                ring_at<VRP>(face_b[0].bits, face_b[1].bits, whole_b[2].bits, bits_rowbase), tf[0], tf[1], tw[2]);
    const bool fast = near && within_reach(f3(u.x, v.x, w.x), reach_dt);
    const bool fast_back = near && within_reach(f3(u.y, v.y, w.y), reach_dt);
    const F3 src = sub3(p, mul3(zero_unless(fast, f3(u.x, v.x, w.x)), A.dt));
    kept.back = sub3(sub3(p, mul3(zero_unless(fast_back, f3(u.y, v.y, w.y)), -A.dt)), off);
    kept.global = !fast_back;
    kept.data = node[G];  // the component at its own face
    const F3 g = sub3(src, off);
    const AxBits gx = split_bits(g[0]), gy = split_bits(g[1]), gz = split_bits(g[2]);
    float a[8];
    ring_corners_at(vring + G * VR * VRP, ring_at<VRP>(gx.bits, gy.bits, gz.bits, bits_rowbase), a);
    kept.hat = blend8(a, gx.t, gy.t, gz.t);
    range8(a, kept.lo, kept.hi);
    hring[slot * VHP + tile_h + n * TY * HZ] = kept.hat;
    return !fast;
  };
  // The ring element's hat: the forward trace alone.
  auto halo_hat = [&](int x, int slot) -> bool {
    const F3 p = add3(f3((float)x, (float)rj, (float)rk), off);
    const F3 node = ring_node<G, VRP>(vring, x, rj * RZ + rk - rowbase);
    const bool near = within_reach(node, reach_dt);
    const F3 m = sub3(p, mul3(zero_unless(near, node), half));
    AxBits whole[3], face[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      whole[a] = split_bits(m[a]);
      face[a] = split_bits(m[a] - 0.5f);
    }
    float a[8];
    ring_corners_at(vring, ring_at<VRP>(whole[0].bits, face[1].bits, face[2].bits, bits_rowbase), a);
    const float u = blend8(a, whole[0].t, face[1].t, face[2].t);
    ring_corners_at(vring + VR * VRP, ring_at<VRP>(face[0].bits, whole[1].bits, face[2].bits, bits_rowbase), a);
    const float v = blend8(a, face[0].t, whole[1].t, face[2].t);
    ring_corners_at(vring + 2 * VR * VRP, ring_at<VRP>(face[0].bits, face[1].bits, whole[2].bits, bits_rowbase), a);
    const float w = blend8(a, face[0].t, face[1].t, whole[2].t);
    const bool fast = near && within_reach(f3(u, v, w), reach_dt);
    const F3 g = sub3(sub3(p, mul3(zero_unless(fast, f3(u, v, w)), A.dt)), off);
    const AxBits gx = split_bits(g[0]), gy = split_bits(g[1]), gz = split_bits(g[2]);
    ring_corners_at(vring + G * VR * VRP, ring_at<VRP>(gx.bits, gy.bits, gz.bits, bits_rowbase), a);
    hring[slot * VHP + ring_h] = blend8(a, gx.t, gy.t, gz.t);
    return !fast;
  };
  // Hat plane x (clamped to the array) into the ring's slot of x; every thread takes part. Returns, the block having met,
  // whether some element's backward sample is to be taken from global memory.
  auto hat_plane = [&](int x, Kept* kept, int arriving) -> bool {
    const int xc = imin_(imax_(x, 0), gd.n0 - 1), slot = x & (HR - 1);
    bool slow[EPT], any = false;
#pragma unroll
    for (int n = 0; n < EPT; ++n) {
      slow[n] = tile_hat(xc, slot, n, kept[n]);
      any = any || slow[n] || kept[n].global;
    }
    bool slow_halo = false;
    if (has_halo) slow_halo = halo_hat(xc, slot);
    land(arriving);
    if (!__syncthreads_or(any || slow_halo)) return false;
    float hat, lo, hi;
    bool global = false;
#pragma unroll
    for (int n = 0; n < EPT; ++n) {
      global = global || kept[n].global;
      if (!slow[n]) continue;
      hat_global<G>(A, xc, imin_(j0 + ty + n * TY, gd.n1 - 1), ck, &hat, &lo, &hi);
      hring[slot * VHP + tile_h + n * TY * HZ] = hat;
      kept[n].hat = hat;
      kept[n].lo = lo;
      kept[n].hi = hi;
    }
    if (slow_halo) {
      hat_global<G>(A, xc, rj, rk, &hat, &lo, &hi);
      hring[slot * VHP + ring_h] = hat;
    }
    return __syncthreads_or(global);
  };

  // prologue: planes s-2 .. s+2 of the velocity, hat planes s-1 and s
#pragma unroll 1
  for (int p = s - 2; p <= s + 1; ++p) {
    fetch(p);
    land(p);
  }
  fetch(s + 2);
  __syncthreads();
  Kept kept[EPT];
  hat_plane(s - 1, kept, s + 2);  // below the array: plane 0's hat, as the correction's clamped sample reads it
  bool global = hat_plane(s, kept, s + 2);

  const size_t plane_stride = (size_t)gd.n1 * gd.n2;
  T* const next = A.next[G];
  for (int i = s; i < e; ++i) {
    // planes i+3 start landing while hat plane i+1 is computed
    fetch(i + 3);
    Kept following[EPT];
    const bool following_global = hat_plane(i + 1, following, i + 3);
    // the correction (advect.py:34-50, 64): back = hat sampled along the backward trace
#pragma unroll
    for (int n = 0; n < EPT; ++n) {
      const int tj = j0 + ty + n * TY;
      const AxBits gx = split_bits(kept[n].back[0]), gy = split_bits(kept[n].back[1]), gz = split_bits(kept[n].back[2]);
      const int gin = gy.bits * HZ + gz.bits - bits_hbase;
      const float* h0 = hring + (gx.bits & (HR - 1)) * VHP + gin;
      const float* h1 = hring + ((gx.bits + 1) & (HR - 1)) * VHP + gin;
      const float a[8] = {h0[0], h1[0], h0[HZ], h1[HZ], h0[1], h1[1], h0[HZ + 1], h1[HZ + 1]};
      float back = blend8(a, gx.t, gy.t, gz.t);
      if (global) {
        float far = back;
        if (kept[n].global) back_global<G, M::tile, VHP>(A, hring, hbase, j0, k0, i - 1, i, imin_(tj, gd.n1 - 1), ck, &far);
        back = far;
      }
      const float corrected = kept[n].hat + 0.5f * (kept[n].data - back);
      if (tj < gd.n1 && tk < gd.n2)
        st_f(next + ((size_t)i * plane_stride + (size_t)tj * gd.n2 + tk), clampf_(corrected, kept[n].lo, kept[n].hi));
      kept[n] = following[n];
    }
    global = following_global;
  }
}

// EPT elements per thread and MINB resident blocks per SM: 1 and 3 (80 registers a thread, of which 272 bytes spill to 396
// bytes of loads a thread, in float) or 2 and 2 (128 registers; 132 and 136 bytes).
template <class T, int EPT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_mac_velocity(const __grid_constant__ Args<T> A) {
  extern __shared__ float sm[];
  int z = blockIdx.z;
  if (z < A.segs[0]) return velocity_march<T, 0, EPT>(A, z, sm);
  z -= A.segs[0];
  if (z < A.segs[1]) return velocity_march<T, 1, EPT>(A, z, sm);
  velocity_march<T, 2, EPT>(A, z - A.segs[1], sm);
}

// Grids with an axis of 2^22 cells or more, whose coordinates split_bits does not cover, and time steps that are not finite
// (march_form).
template <class T>
__global__ void __launch_bounds__(NT, 2) k_mac_velocity_long(const __grid_constant__ Args<T> A) {
  extern __shared__ float sm[];
  int z = blockIdx.z;
  if (z < A.segs[0]) return march<T, 0>(A, z, sm);
  z -= A.segs[0];
  if (z < A.segs[1]) return march<T, 1>(A, z, sm);
  march<T, 2>(A, z - A.segs[1], sm);
}

// MINB: resident blocks per SM the kernel is compiled for (4 at 256 threads: at most 64 registers a thread;
// 3: 80; 2: 128).
template <class T, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_mac_scalars(const __grid_constant__ Args<T> A) {
  extern __shared__ float sm[];
  march<T, 3>(A, blockIdx.z, sm);
}

// Line totals from the segment sums (in segment order, float), then 256 lines per block added in double by a
// halving tree, as k_line_partials lays them out: partial[f * blocks + block].
constexpr int LINE_BLOCK = 256;
__global__ void k_segment_lines(const float* __restrict__ seg_sums, int segs, long lines, double* __restrict__ partial,
                                int blocks) {
  __shared__ double slot[LINE_BLOCK];
  const int f = blockIdx.y;
  const long line = (long)blockIdx.x * LINE_BLOCK + threadIdx.x;
  double value = 0.0;
  if (line < lines) {
    float total = 0.0f;
    for (int s = 0; s < segs; ++s) total = total + seg_sums[((long)f * segs + s) * lines + line];
    value = (double)total;
  }
  slot[threadIdx.x] = value;
  __syncthreads();
  for (int h = LINE_BLOCK / 2; h >= 1; h >>= 1) {
    if ((int)threadIdx.x < h) slot[threadIdx.x] = slot[threadIdx.x] + slot[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[f * blocks + blockIdx.x] = slot[0];
}

constexpr size_t SCALAR_SMEM = sizeof(float) * (3 * VR * RPN + 2 * SR * RPN + 2 * HR * HP + SLACK);

// Segments along x: enough blocks for about six waves of the resident blocks, each segment at least 8 planes.
static int segments(int n0, long tiles, int groups) {
  const long target = 6L * BLOCKS_PER_SM * 148;
  long segs = (target + tiles * groups - 1) / (tiles * groups);
  segs = std::max(1L, std::min(segs, (long)std::max(1, n0 / 8)));
  return (int)segs;
}

static int env_int(const char* name) {
  const char* v = getenv(name);
  return v ? atoi(v) : 0;
}

// Blocks per SM the scalar march is compiled for: PLUME_MAC_BLOCKS = 2, 3 or 4 (the default, BLOCKS_PER_SM).
static int blocks_per_sm() {
  static const int b = [] {
    const int v = env_int("PLUME_MAC_BLOCKS");
    return v == 2 || v == 3 ? v : BLOCKS_PER_SM;
  }();
  return b;
}


// Lets the kernel use `smem` bytes of shared memory on the current device.
template <class Kernel>
static int configure(Kernel k, size_t smem, OncePerDevice& done) {
  int device = 0;
  const int status = runtime_status("current device", cudaGetDevice(&device));
  if (status != PLUME_OK) return status;
  return done.run(device, [&] {
    return runtime_status("fused advection: shared memory",
                          cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  });
}

}  // namespace mac

int mac_segments_for_scalars(const PlumeGridInfo& info) {
  const int nx = info.dims[0], ny = info.dims[1], nz = info.dims[2];
  const long tiles = (long)((ny + mac::TY - 1) / mac::TY) * ((nz + mac::TZ - 1) / mac::TZ);
  int segs = mac::env_int("PLUME_MAC_SCALAR_SEGS");
  if (segs <= 0) segs = mac::segments(nx, tiles, 1);
  segs = std::max(1, std::min(segs, nx));
  const int len = (nx + segs - 1) / segs;
  return (nx + len - 1) / len;  // every segment non-empty
}

long long mac_partial_floats(const PlumeGridInfo& info) {
  return 3LL * mac_segments_for_scalars(info) * info.dims[1] * info.dims[2];
}

template <class T>
int launch_mac_velocity(const PlumeGridInfo& info, const T* u, const T* v, const T* w, T* u_next, T* v_next,
                        T* w_next, float dt_over_cell, cudaStream_t st) {
  static OncePerDevice configured[3];
  const int form = mac::march_form(info.dims, dt_over_cell, mac::env_int("PLUME_MAC_ELEMENTS")), ept = form == 2 ? 2 : 1;
  auto kernel = form == 3 ? mac::k_mac_velocity_long<T>
                          : (form == 2 ? mac::k_mac_velocity<T, 2, 2> : mac::k_mac_velocity<T, 1, 3>);
  const size_t smem = ept == 2 ? mac::March<2>::smem : mac::March<1>::smem;
  const int rows = ept * mac::TY;
  int status = mac::configure(kernel, smem, configured[form - 1]);
  if (status != PLUME_OK) return status;
  const int nx = info.dims[0], ny = info.dims[1], nz = info.dims[2];
  mac::Args<T> A{};
  A.info = info;
  A.vel[0] = u;
  A.vel[1] = v;
  A.vel[2] = w;
  A.next[0] = u_next;
  A.next[1] = v_next;
  A.next[2] = w_next;
  A.dt = dt_over_cell;
  const int jt = (ny + 1 + rows - 1) / rows, kt = (nz + 1 + mac::TZ - 1) / mac::TZ;
  const int segs = mac::march_segments(info.dims, ept, mac::TY, mac::TZ, mac::env_int("PLUME_MAC_VELOCITY_SEGS"));
  A.seg_len = (nx + segs - 1) / segs;
  for (int g = 0; g < 3; ++g) A.segs[g] = (nx + (g == 0) + A.seg_len - 1) / A.seg_len;
  const dim3 grid(kt, jt, A.segs[0] + A.segs[1] + A.segs[2]);
  kernel<<<grid, mac::NT, smem, st>>>(A);
  return launch_status("fused velocity advection");
}

template <class T>
int launch_mac_scalars(const PlumeGridInfo& info, const T* u, const T* v, const T* w, const T* smoke,
                       const T* temperature, T* smoke_next, T* temperature_next, float smoke_outside,
                       float heat_outside, int uses_outside, float* seg_sums, double* line_partials, int dissipate,
                       float heat_keep, float ambient, float dt_over_cell, cudaStream_t st) {
  static OncePerDevice configured[5];
  const int bps = mac::blocks_per_sm();
  auto kernel = bps == 2 ? mac::k_mac_scalars<T, 2> : (bps == 3 ? mac::k_mac_scalars<T, 3> : mac::k_mac_scalars<T, 4>);
  int status = mac::configure(kernel, mac::SCALAR_SMEM, configured[bps]);
  if (status != PLUME_OK) return status;
  const int nx = info.dims[0], ny = info.dims[1], nz = info.dims[2];
  mac::Args<T> A{};
  A.info = info;
  A.vel[0] = u;
  A.vel[1] = v;
  A.vel[2] = w;
  A.field[0] = smoke;
  A.field[1] = temperature;
  A.next[0] = smoke_next;
  A.next[1] = temperature_next;
  A.outside[0] = smoke_outside;
  A.outside[1] = heat_outside;
  A.uses_outside = uses_outside;
  A.dt = dt_over_cell;
  const int segs = mac_segments_for_scalars(info);
  A.seg_len = (nx + segs - 1) / segs;
  A.segs[3] = segs;
  A.partials = seg_sums;
  A.dissipate = dissipate;
  A.heat_keep = heat_keep;
  A.ambient = ambient;
  const dim3 grid((nz + mac::TZ - 1) / mac::TZ, (ny + mac::TY - 1) / mac::TY, segs);
  kernel<<<grid, mac::NT, mac::SCALAR_SMEM, st>>>(A);
  status = launch_status("fused scalar advection");
  if (status != PLUME_OK) return status;
  const long lines = (long)ny * nz;
  const int blocks = (int)((lines + mac::LINE_BLOCK - 1) / mac::LINE_BLOCK);
  mac::k_segment_lines<<<dim3(blocks, 3), mac::LINE_BLOCK, 0, st>>>(seg_sums, segs, lines, line_partials, blocks);
  return launch_status("smoke budget line sums");
}

#define PLUME_MAC_INSTANTIATE(T)                                                                              \
  template int launch_mac_velocity<T>(const PlumeGridInfo&, const T*, const T*, const T*, T*, T*, T*, float,   \
                                      cudaStream_t);                                                           \
  template int launch_mac_scalars<T>(const PlumeGridInfo&, const T*, const T*, const T*, const T*, const T*,  \
                                     T*, T*, float, float, int, float*, double*, int, float, float, float,     \
                                     cudaStream_t);
PLUME_MAC_INSTANTIATE(float)
PLUME_MAC_INSTANTIATE(__nv_bfloat16)
PLUME_MAC_INSTANTIATE(__half)

}  // namespace plume
