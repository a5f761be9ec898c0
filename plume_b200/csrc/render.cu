// Volume-render kernels of libplume_b200.so for sm_100a: the light volume (shadow march), the normal field
// and the camera ray march of chadmv/plume (src/plume/render/*), with their C ABI.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "light_range.cuh"

namespace plume {

__device__ __forceinline__ void slab_range(F3 origin, F3 dir, F3 bmin, F3 bmax, float& t0out, float& t1out) {
  float t_enter = -1.0e30f, t_exit = 1.0e30f;  // raymarch.py:55-69
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (fabsf(dir[a]) < 1.0e-12f) {
      if (origin[a] < bmin[a] || origin[a] > bmax[a]) {
        t0out = 1.0f;
        t1out = 0.0f;
        return;
      }
    } else {
      float t0 = (bmin[a] - origin[a]) / dir[a];
      float t1 = (bmax[a] - origin[a]) / dir[a];
      t_enter = fmax_(t_enter, fmin_(t0, t1));
      t_exit = fmin_(t_exit, fmax_(t0, t1));
    }
  }
  t0out = t_enter;
  t1out = t_exit;
}

// ---- empty-space skipping ------------------------------------------------------------------------------------
// A brick map holds, for each 4x4x4 brick of cells, the largest smoke value of the brick and of the next cell
// past it on each axis: every corner a trilinear sample with lower corner in the brick can blend. When that
// is <= 0, every corner is <= 0, their blend is <= 0 (each weighted term is), max(sample, 0) is +0 and the
// sample adds exactly nothing: skipping it changes no bit of the result.
constexpr int BRICK = 4;
constexpr int LIGHT_ROWS = 8;  // rows of the light volume's block
constexpr int LIGHT_RUN = 4;   // samples of a light march per look at the map

__host__ __device__ __forceinline__ Dims brick_dims(const Dims& d) {
  return Dims{(d.n0 + BRICK - 1) / BRICK, (d.n1 + BRICK - 1) / BRICK, (d.n2 + BRICK - 1) / BRICK};
}

// The map's entries for empty bricks hold how far they are from the next brick that is not: -r when every brick within r
// bricks on each axis (0 to EMPTY_REACH) is empty, so that a march crosses the whole cube of them in one step.
constexpr int EMPTY_REACH = 3;

// What a march that advances `delta` cells per sample needs of each axis to count the samples it may pass over.
struct SkipAxis {
  float per_cell;  // samples per cell: 1 / |delta|
  float sign;      // of delta
  float ahead;     // from a brick's lower face to the one the march leaves by: BRICK or 0
  int end;         // the last brick that way, which reaches to infinity
};
__device__ __forceinline__ SkipAxis skip_axis(float delta, int n) {
  const bool up = delta > 0.0f;
  return SkipAxis{delta == 0.0f ? 3.0e38f : 1.0f / fabsf(delta), up ? 1.0f : -1.0f, up ? (float)BRICK : 0.0f,
                  up ? (n - 1) / BRICK : 0};
}

// How many samples after the one at coordinate g stay, on this axis, within `reach` bricks of its brick b, as a float,
// possibly negative or huge (the caller floors and caps the least of the axes). A sample's brick is that of its clamped
// lower corner, so the first brick reaches to -inf and the last to +inf. Samples nearer than `margin` cells to the face
// are not counted: the margin bounds twice the float error of a computed sample point against the exact line through
// the march, so every counted sample, as computed, lies inside.
__device__ __forceinline__ float samples_within(const SkipAxis& a, float g, int b, float reach, float margin) {
  const float room = a.sign * ((float)(b * BRICK) + a.ahead - g) + reach * BRICK;
  const bool unbounded = a.per_cell > 1.0e38f || fabsf((float)(a.end - b)) <= reach;
  return unbounded ? 3.0e38f : (room - margin) * a.per_cell;
}

// Index of the sample a march continues from after the sample `s` in an empty brick: `count` samples further (those that
// cannot leave the empty bricks around it), and at most `end`.
__device__ __forceinline__ int past_brick(int s, int end, float count) {
  return count >= 1.0f ? s + (int)fminf(count, (float)(end - s)) : s;
}

// A warp takes seven bricks of a row along z: 29 columns of cells, 5 x 5 loads each along the rows, then the columns of
// each brick. A thread per brick read its 125 cells one row of five after the other, each lane on another cache line.
constexpr int ROW_BRICKS = 7, ROW_WARPS = 4;
static dim3 brick_row_grid(const Dims& b) {  // tiles of (j, k) along x, which has room for any axis
  return dim3((unsigned)((b.n2 + ROW_BRICKS - 1) / ROW_BRICKS) * ((b.n1 + ROW_WARPS - 1) / ROW_WARPS), 1, b.n0);
}
struct BrickRow {
  int i, j, k;  // the first cell on each axis, k this lane's column
  int brick;    // entry of this lane's brick; -1: none
};
__device__ __forceinline__ bool brick_row(const Dims& d, BrickRow& r) {
  const Dims b = brick_dims(d);
  const unsigned across = (b.n2 + ROW_BRICKS - 1) / ROW_BRICKS, tile_j = blockIdx.x / across, tile_k = blockIdx.x - tile_j * across;
  const int bi = blockIdx.z, bj = tile_j * ROW_WARPS + threadIdx.y, bk = tile_k * ROW_BRICKS + threadIdx.x / BRICK;
  if (bj >= b.n1) return false;
  r.i = bi * BRICK;
  r.j = bj * BRICK;
  r.k = imin_(tile_k * ROW_BRICKS * BRICK + threadIdx.x, d.n2 - 1);
  r.brick = threadIdx.x % BRICK == 0 && threadIdx.x < ROW_BRICKS * BRICK && bk < b.n2 ? at(b, bi, bj, bk) : -1;
  return true;
}
template <class Combine>
__device__ __forceinline__ float over_columns(float x, Combine combine) {  // of this lane's column and the next four
  float best = x;
#pragma unroll
  for (int o = 1; o <= BRICK; ++o) best = combine(best, __shfl_down_sync(0xffffffffu, x, o));
  return best;
}

template <class T>
__global__ void __launch_bounds__(32 * ROW_WARPS) k_brick_max(Dims d, const T* __restrict__ f, float* __restrict__ bricks) {
  BrickRow r;
  if (!brick_row(d, r)) return;
  float best = -3.0e38f;
#pragma unroll
  for (int a = 0; a <= BRICK; ++a)
#pragma unroll
    for (int b = 0; b <= BRICK; ++b)
      best = fmaxf(best, ldg_f(f + at(d, imin_(r.i + a, d.n0 - 1), imin_(r.j + b, d.n1 - 1), r.k)));
  best = over_columns(best, [](float x, float y) { return fmaxf(x, y); });
  if (r.brick >= 0) bricks[r.brick] = best;
}

// The map's empty entries (<= 0) as -r, from a tile of 4 x 8 x 8 bricks and EMPTY_REACH around it: the distance to the
// nearest entry that is not empty, axis by axis.
constexpr int REACH_TILE = 8, REACH_SPAN = REACH_TILE + 2 * EMPTY_REACH, REACH_ROWS = 4, REACH_DEEP = REACH_ROWS + 2 * EMPTY_REACH;
__global__ void __launch_bounds__(256) k_brick_reach(Dims b, const float* __restrict__ map, float* __restrict__ bricks) {
  __shared__ signed char near_z[REACH_DEEP][REACH_SPAN][REACH_SPAN];
  __shared__ signed char near_y[REACH_DEEP][REACH_SPAN][REACH_TILE];
  __shared__ signed char near_x[REACH_DEEP][REACH_TILE][REACH_TILE];
  const int i0 = blockIdx.z * REACH_ROWS, j0 = blockIdx.y * REACH_TILE, k0 = blockIdx.x * REACH_TILE;
  constexpr int FAR = EMPTY_REACH + 1;
  for (int e = threadIdx.x; e < REACH_DEEP * REACH_SPAN * REACH_SPAN; e += 256) {
    const int x = e / (REACH_SPAN * REACH_SPAN), y = e / REACH_SPAN % REACH_SPAN, z = e % REACH_SPAN;
    const int i = i0 + x - EMPTY_REACH, j = j0 + y - EMPTY_REACH, k = k0 + z - EMPTY_REACH;
    const bool inside = i >= 0 && j >= 0 && k >= 0 && i < b.n0 && j < b.n1 && k < b.n2;
    near_z[x][y][z] = inside && __ldg(map + at(b, i, j, k)) > 0.0f ? 0 : FAR;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < REACH_DEEP * REACH_SPAN * REACH_TILE; e += 256) {
    const int x = e / (REACH_SPAN * REACH_TILE), y = e / REACH_TILE % REACH_SPAN, z = e % REACH_TILE;
    int best = FAR;
#pragma unroll
    for (int o = -EMPTY_REACH; o <= EMPTY_REACH; ++o) best = imin_(best, imax_(o < 0 ? -o : o, near_z[x][y][z + EMPTY_REACH + o]));
    near_y[x][y][z] = (signed char)best;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < REACH_DEEP * REACH_TILE * REACH_TILE; e += 256) {
    const int x = e / (REACH_TILE * REACH_TILE), y = e / REACH_TILE % REACH_TILE, z = e % REACH_TILE;
    int best = FAR;
#pragma unroll
    for (int o = -EMPTY_REACH; o <= EMPTY_REACH; ++o) best = imin_(best, imax_(o < 0 ? -o : o, near_y[x][y + EMPTY_REACH + o][z]));
    near_x[x][y][z] = (signed char)best;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < REACH_ROWS * REACH_TILE * REACH_TILE; e += 256) {
    const int x = e / (REACH_TILE * REACH_TILE), y = e / REACH_TILE % REACH_TILE, z = e % REACH_TILE;
    const int i = i0 + x, j = j0 + y, k = k0 + z;
    if (i >= b.n0 || j >= b.n1 || k >= b.n2) continue;
    int best = FAR;
#pragma unroll
    for (int o = -EMPTY_REACH; o <= EMPTY_REACH; ++o) best = imin_(best, imax_(o < 0 ? -o : o, near_x[x + EMPTY_REACH + o][y][z]));
    bricks[at(b, i, j, k)] = best == 0 ? __ldg(map + at(b, i, j, k)) : (float)(1 - best);
  }
}
static int brick_reach(const Dims& b, const float* map, float* bricks, cudaStream_t st) {
  const dim3 grid((b.n2 + REACH_TILE - 1) / REACH_TILE, (b.n1 + REACH_TILE - 1) / REACH_TILE, (b.n0 + REACH_ROWS - 1) / REACH_ROWS);
  k_brick_reach<<<grid, 256, 0, st>>>(b, map, bricks);
  return launch_status("brick reach");
}

// light_volume_kernel (light_volume.py:18-33): each lit cell marches toward the light in at most half-cell
// steps to the box edge and gets exp(-opacity * column * cell_m). With `bricks`, samples whose corners are all
// <= 0 add exactly 0: the march steps over the whole run of them that lies in one brick.
//
// With `march_cells`, only the cells a camera march of the same smoke can read get their value: a march sample
// reads the light at its eight corners only when its alpha is > 0, so when one of those corners holds smoke
// > 0; the corners of every sample that reads cell c lie in {c-1, c, c+1}^3. So c is read only if one of those
// 27 cells holds smoke > 0 (tested first through the bricks of the lower corners {c-1, c}^3, which hold the
// largest smoke of every such corner). Every other cell gets 1.
//
// Arithmetic: the trilinear blends are fma(t, b - a, a) and the column adds each sample with one fma, one
// rounding fewer than light_volume_kernel's lerp and multiply-add, so the light agrees with the reference's to
// about an ulp of the column (held to 1e-5 relative); the empty-space skipping and the march_cells form change
// no bit of it.
__device__ __forceinline__ float lerp_fma(float a, float b, float t) { return __fmaf_rn(t, b - a, a); }

template <class T>
__device__ __forceinline__ float sample_fma(const T* __restrict__ f, int cell, int step_x, int step_y, int step_z, float tx,
                                            float ty, float tz) {
  const T* p = f + cell;
  const float c00 = lerp_fma(ldg_f(p), ldg_f(p + step_x), tx);
  const float c10 = lerp_fma(ldg_f(p + step_y), ldg_f(p + step_x + step_y), tx);
  const float c01 = lerp_fma(ldg_f(p + step_z), ldg_f(p + step_x + step_z), tx);
  const float c11 = lerp_fma(ldg_f(p + step_y + step_z), ldg_f(p + step_x + step_y + step_z), tx);
  return lerp_fma(lerp_fma(c00, c10, ty), lerp_fma(c01, c11, ty), tz);
}

// Whether a camera march of this smoke reads the light at cell (i, j, k), for a warp's 32 cells along z (the march_cells
// test above; smoke in one of the 27 cells puts a value > 0 in one of the bricks, so the bricks are only the quick no).
template <class T>
__device__ __forceinline__ bool read_by_march(const Dims& d, const T* __restrict__ smoke, const float* __restrict__ bricks,
                                              int i, int j, int k) {
  const Dims bd = brick_dims(d);
  const int kc = imin_(k, d.n2 - 1), c0 = imax_(kc - 1, 0) / BRICK, c1 = kc / BRICK;
  bool near = false;
  for (int a = imax_(i - 1, 0) / BRICK; a <= i / BRICK; ++a)
    for (int b = imax_(j - 1, 0) / BRICK; b <= j / BRICK; ++b)
      near = near || __ldg(bricks + at(bd, a, b, c0)) > 0.0f || __ldg(bricks + at(bd, a, b, c1)) > 0.0f;
  if (!__any_sync(0xffffffffu, near)) return false;
  auto column = [&](int c) {  // smoke in the column at c of the 3 x 3 rows
    bool smoky = false;
#pragma unroll
    for (int a = -1; a <= 1; ++a)
#pragma unroll
      for (int b = -1; b <= 1; ++b)
        smoky |= ldg_f(smoke + at(d, imin_(imax_(i + a, 0), d.n0 - 1), imin_(imax_(j + b, 0), d.n1 - 1), c)) > 0.0f;
    return smoky;
  };
  const int lane = threadIdx.x;
  const unsigned own = __ballot_sync(0xffffffffu, column(kc));
  bool read = (((own << 1) | own | (own >> 1)) >> lane) & 1u;
  if (lane == 0 || lane == 31) read |= column(imin_(imax_(lane == 0 ? kc - 1 : kc + 1, 0), d.n2 - 1));
  return read;
}

// A coordinate in [0, 2^23) as its floor plus the bits of 2^23 (which wrap-around cancels in an index) and its fraction, on
// the float adders: axis_of's index and weight.
constexpr float TWO23 = 8388608.0f;
constexpr unsigned TWO23_BITS = 0x4B000000u;
constexpr int SPLIT_LIMIT = 1 << 22;  // extents and sample counts below it are exact in both
struct SplitAxis {
  unsigned bits;
  float t;
};
template <bool INSIDE>
__device__ __forceinline__ SplitAxis split_axis(float g, int n) {
  const float x = INSIDE ? g : fminf(fmaxf(g, 0.0f), (float)(n - 1));
  const float shifted = __fadd_rd(x, TWO23);
  return SplitAxis{__float_as_uint(shifted), x - (shifted - TWO23)};
}

// The column of one cell's march when an extent or the sample count passes SPLIT_LIMIT: every sample, indices converted.
template <class T>
__device__ __noinline__ float column_long(const Dims& d, const T* __restrict__ smoke, F3 toward, F3 corner, int steps, float step) {
  float column = 0.0f;
  for (int s = 0; s < steps; ++s) {
    const float t = ((float)s + 0.5f) * step;
    const Axis1 x = axis_of(__fmaf_rn(toward[0], t, corner[0]), d.n0, d.n1 * d.n2);
    const Axis1 y = axis_of(__fmaf_rn(toward[1], t, corner[1]), d.n1, d.n2);
    const Axis1 z = axis_of(__fmaf_rn(toward[2], t, corner[2]), d.n2, 1);
    column = __fmaf_rn(fmax_(sample_fma(smoke, (x.i0 * d.n1 + y.i0) * d.n2 + z.i0, x.step, y.step, z.step, x.t, y.t, z.t), 0.0f), step, column);
  }
  return column;
}

// The light of one cell: its march toward the light.
template <class T>
__device__ __forceinline__ float light_at(const Dims& d, const T* __restrict__ smoke, F3 toward, float cell_m,
                                          float opacity, const float* __restrict__ bricks, int i, int j, int k) {
  const F3 half = f3(0.5f, 0.5f, 0.5f);
  const F3 corner = f3((float)i, (float)j, (float)k);
  F3 start = add3(corner, half);
  F3 box_max = f3((float)d.n0, (float)d.n1, (float)d.n2);
  float t0, length;
  slab_range(start, toward, f3(0.0f, 0.0f, 0.0f), box_max, t0, length);
  const int steps = (int)ceilf(length / 0.5f);
  float column = 0.0f;
  if (steps > 0) {
    const float step = length / (float)steps;
    const int widest = imax_(imax_(d.n0, d.n1), d.n2);
    if (imax_(widest, steps) >= SPLIT_LIMIT) return exp_f(-opacity * column_long(d, smoke, toward, corner, steps, step) * cell_m);
    // the computed points (i, j, k) + toward * ((s + 0.5) * step), from the cell's lower corner, are within
    // (2 * length + 2 * extent) * 2^-24 cells of the exact line
    const float margin = march_margin(length, widest);
    const SkipAxis skip_x = skip_axis(toward[0] * step, d.n0), skip_y = skip_axis(toward[1] * step, d.n1),
                   skip_z = skip_axis(toward[2] * step, d.n2);
    const Dims bd = brick_dims(d);
    const unsigned un1 = d.n1, un2 = d.n2, ub1 = bd.n1, ub2 = bd.n2, brick_bits = TWO23_BITS / BRICK;
    const unsigned cell_base = (TWO23_BITS * un1 + TWO23_BITS) * un2 + TWO23_BITS;
    const unsigned brick_base = (brick_bits * ub1 + brick_bits) * ub2 + brick_bits;
    const int plane = d.n1 * d.n2;
    const float end = (float)(steps - 1);
    auto point = [&](float s) {
      const float t = (s + 0.5f) * step;
      return f3(__fmaf_rn(toward[0], t, corner[0]), __fmaf_rn(toward[1], t, corner[1]), __fmaf_rn(toward[2], t, corner[2]));
    };
    // The sample to continue from when s lies in an empty brick (that of its clamped lower corner), else s itself.
    auto past_empty = [&](float s, const F3& g, unsigned x, unsigned y, unsigned z) {
      const unsigned bx = x / BRICK, by = y / BRICK, bz = z / BRICK;
      const float held = __ldg(bricks + ((bx * ub1 + by) * ub2 + bz - brick_base));
      if (held > 0.0f) return s;
      const float count = fminf(fminf(samples_within(skip_x, g[0], (int)(bx - brick_bits), -held, margin),
                                      samples_within(skip_y, g[1], (int)(by - brick_bits), -held, margin)),
                                samples_within(skip_z, g[2], (int)(bz - brick_bits), -held, margin));
      return s + 1.0f + floorf(fminf(fmaxf(count, 0.0f), end - s));
    };
    // the last sample that lies in [0, extent - 1) on every axis by more than the margin, as all before it then do
    const float inner = fminf(fminf(samples_inside(toward[0] * step, corner[0], d.n0, margin),
                                    samples_inside(toward[1] * step, corner[1], d.n1, margin)),
                              samples_inside(toward[2] * step, corner[2], d.n2, margin));
    const float to = last_run(inner, end, LIGHT_RUN);
    float s = 0.0f;
    // runs of LIGHT_RUN samples whose corners lie in the array; only the first looks its brick up
    while (s <= to) {
      SplitAxis x[LIGHT_RUN], y[LIGHT_RUN], z[LIGHT_RUN];
      F3 g = point(s);
#pragma unroll
      for (int r = 0; r < LIGHT_RUN; ++r) {
        const F3 q = r == 0 ? g : point(s + (float)r);
        x[r] = split_axis<true>(q[0], d.n0);
        y[r] = split_axis<true>(q[1], d.n1);
        z[r] = split_axis<true>(q[2], d.n2);
      }
      if (bricks) {
        const float next = past_empty(s, g, x[0].bits, y[0].bits, z[0].bits);
        if (next != s) {
          s = next;
          continue;
        }
      }
      float sample[LIGHT_RUN];
#pragma unroll
      for (int r = 0; r < LIGHT_RUN; ++r)
        sample[r] = sample_fma(smoke, (int)((x[r].bits * un1 + y[r].bits) * un2 + z[r].bits - cell_base), plane, d.n2, 1,
                               x[r].t, y[r].t, z[r].t);
#pragma unroll
      for (int r = 0; r < LIGHT_RUN; ++r) column = __fmaf_rn(fmaxf(sample[r], 0.0f), step, column);
      s += (float)LIGHT_RUN;
    }
    while (s <= end) {
      const F3 g = point(s);
      const SplitAxis x = split_axis<false>(g[0], d.n0), y = split_axis<false>(g[1], d.n1), z = split_axis<false>(g[2], d.n2);
      if (bricks) {
        const float next = past_empty(s, g, x.bits, y.bits, z.bits);
        if (next != s) {
          s = next;
          continue;
        }
      }
      const float sample = sample_fma(smoke, (int)((x.bits * un1 + y.bits) * un2 + z.bits - cell_base),
                                      x.bits < TWO23_BITS + d.n0 - 1 ? plane : 0, y.bits < TWO23_BITS + d.n1 - 1 ? d.n2 : 0,
                                      z.bits < TWO23_BITS + d.n2 - 1 ? 1 : 0, x.t, y.t, z.t);
      column = __fmaf_rn(fmaxf(sample, 0.0f), step, column);
      s += 1.0f;
    }
  }
  return exp_f(-opacity * column * cell_m);
}

// A block covers 32 cells along z of LIGHT_ROWS rows of one x-plane, a warp per row. The warps give every cell that no
// march reads its 1 and queue the others in shared memory, then march the queue 32 cells at a time, so that lanes stay
// busy where only part of a row is lit.
//
// Bound by instruction issue (75% of the slots; 24 of 32 lanes active). Measured on B200 at 128x192x128 with 11% of the
// cells lit: 560 us with four rows a warp, one sample after the other, clamped indices by conversion, each empty brick
// crossed by itself; 160 us now. The few lit blocks ended late on a chip that was otherwise done (four rows a warp: 360
// us), and of the instructions half were clamps, conversions, addresses and looks at the map (a look and a clamp for
// every sample: 216 us; runs of two 176 us, of three 164 us).
template <class T>
__global__ void __launch_bounds__(32 * LIGHT_ROWS, 4) k_light_volume(Dims d, const T* __restrict__ smoke, F3 toward, float cell_m,
                                                                     float opacity, float* __restrict__ light,
                                                                     const float* __restrict__ bricks, int march_cells) {
  __shared__ unsigned short queue[LIGHT_ROWS * 32];
  __shared__ int queued;
  const int lane = threadIdx.x, warp = threadIdx.y;
  const unsigned across = (d.n2 + 31) / 32, tile_j = blockIdx.x / across, tile_k = blockIdx.x - tile_j * across;
  const int i = blockIdx.z, k0 = tile_k * 32, k = k0 + lane, j0 = tile_j * LIGHT_ROWS;
  if (lane == 0 && warp == 0) queued = 0;
  __syncthreads();
  if (j0 + warp < d.n1) {
    const int j = j0 + warp;
    bool lit = k < d.n2;
    if (march_cells) {
      const bool read = read_by_march(d, smoke, bricks, i, j, k);
      if (lit && !read) light[at(d, i, j, k)] = 1.0f;
      lit = lit && read;
    }
    const unsigned vote = __ballot_sync(0xffffffffu, lit);
    int from = 0;
    if (lane == 0 && vote != 0) from = atomicAdd(&queued, __popc(vote));
    from = __shfl_sync(0xffffffffu, from, 0);
    if (lit) queue[from + __popc(vote & ((1u << lane) - 1u))] = (unsigned short)(warp * 32 + lane);
  }
  __syncthreads();
  const int count = queued;
#pragma unroll 1
  for (int b = warp * 32 + lane; b < count; b += 32 * LIGHT_ROWS) {
    const int e = queue[b], j = j0 + e / 32, kk = k0 + e % 32;
    light[at(d, i, j, kk)] = light_at(d, smoke, toward, cell_m, opacity, bricks, i, j, kk);
  }
}

// blur_axis_kernel (normal_field.py:12-22), the weights passed with the launch. Along x and y a thread forms BLUR_CELLS
// consecutive cells, each value of the line loaded once for all of them; every sum runs in the order of the taps.
constexpr int MAX_BLUR_TAPS = 129, BLUR_CELLS = 4;
struct BlurWeights {
  float w[MAX_BLUR_TAPS];
};

template <int AXIS, class T>
__global__ void __launch_bounds__(256) k_blur_axis(Dims d, const T* __restrict__ src, float* __restrict__ dst, int radius,
                                                   const __grid_constant__ BlurWeights weights) {
  constexpr int Q = AXIS == 2 ? 1 : BLUR_CELLS;
  const int i = blockIdx.z * (AXIS == 0 ? Q : 1), j = (blockIdx.y * blockDim.y + threadIdx.y) * (AXIS == 1 ? Q : 1);
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= d.n1 || k >= d.n2) return;
  const int cell = AXIS == 0 ? i : (AXIS == 1 ? j : k), n = AXIS == 0 ? d.n0 : (AXIS == 1 ? d.n1 : d.n2);
  const int stride = AXIS == 0 ? d.n1 * d.n2 : (AXIS == 1 ? d.n2 : 1);
  const int here = at(d, i, j, k);
  const T* line = src + (here - cell * stride);
  auto value = [&](int c) { return ldg_f(line + imin_(imax_(c, 0), n - 1) * stride); };
  const int taps = 2 * radius + 1;
  float total[Q] = {};
  if (taps >= Q) {
    // value t of the line is tap t - q of output q: the first values reach the first outputs, the last ones the last
#pragma unroll
    for (int t = 0; t < Q - 1; ++t) {
      const float v = value(cell - radius + t);
#pragma unroll
      for (int q = 0; q <= t; ++q) total[q] = total[q] + weights.w[t - q] * v;
    }
#pragma unroll 4
    for (int t = Q - 1; t < taps; ++t) {
      const float v = value(cell - radius + t);
#pragma unroll
      for (int q = 0; q < Q; ++q) total[q] = total[q] + weights.w[t - q] * v;
    }
#pragma unroll
    for (int t = 0; t < Q - 1; ++t) {
      const float v = value(cell + radius + 1 + t);
#pragma unroll
      for (int q = t + 1; q < Q; ++q) total[q] = total[q] + weights.w[taps + t - q] * v;
    }
  } else {
    for (int t = 0; t < taps; ++t)
#pragma unroll
      for (int q = 0; q < Q; ++q) total[q] = total[q] + weights.w[t] * value(cell + q - radius + t);
  }
#pragma unroll
  for (int q = 0; q < Q; ++q)
    if (cell + q < n) dst[here + q * stride] = total[q];
}

// gradient_kernel (normal_field.py:25-38): per-cell central differences, one-sided at the edges; AoS output. A span is
// one or two cells, so the division by it is a product with a power of two. A warp's 96 floats pass through shared memory,
// so that they leave in three whole rows instead of three times in every third place.
constexpr int GRADIENT_ROWS = 8;
__global__ void __launch_bounds__(32 * GRADIENT_ROWS) k_gradient(Dims d, const float* __restrict__ src, float* __restrict__ gradient) {
  __shared__ float out[GRADIENT_ROWS][96];
  const int i = blockIdx.z, j = blockIdx.y * GRADIENT_ROWS + threadIdx.y, k0 = blockIdx.x * 32, lane = threadIdx.x;
  if (j >= d.n1) return;
  const int k = imin_(k0 + lane, d.n2 - 1), plane = d.n1 * d.n2;
  const int here = at(d, i, j, k);
  auto difference = [&](int cell, int n, int stride) {
    const int below = cell > 0 ? stride : 0, above = cell < n - 1 ? stride : 0;
    const float rise = __ldg(src + (here + above)) - __ldg(src + (here - below));
    return below + above == 0 ? 0.0f : rise * (below != 0 && above != 0 ? 0.5f : 1.0f);
  };
  out[threadIdx.y][lane * 3] = difference(i, d.n0, plane);
  out[threadIdx.y][lane * 3 + 1] = difference(j, d.n1, d.n2);
  out[threadIdx.y][lane * 3 + 2] = difference(k, d.n2, 1);
  __syncwarp();
  float* row = gradient + (size_t)at(d, i, j, k0) * 3;
  const int floats = imin_(32, d.n2 - k0) * 3;
#pragma unroll
  for (int e = lane; e < 96; e += 32)
    if (e < floats) row[e] = out[threadIdx.y][e];
}

__device__ __forceinline__ F3 sample_vec(const float* __restrict__ f, const Dims& d, F3 g) {
  float x = clampf_(g[0], 0.0f, (float)(d.n0 - 1));
  float y = clampf_(g[1], 0.0f, (float)(d.n1 - 1));
  float z = clampf_(g[2], 0.0f, (float)(d.n2 - 1));
  int i0 = (int)x, j0 = (int)y, k0 = (int)z;
  int i1 = imin_(i0 + 1, d.n0 - 1), j1 = imin_(j0 + 1, d.n1 - 1), k1 = imin_(k0 + 1, d.n2 - 1);
  float tx = x - (float)i0, ty = y - (float)j0, tz = z - (float)k0;
  auto ld = [&](int i, int j, int k) {
    const float* q = f + (size_t)at(d, i, j, k) * 3;
    return f3(__ldg(q), __ldg(q + 1), __ldg(q + 2));
  };
  F3 c00 = lerp3(ld(i0, j0, k0), ld(i1, j0, k0), tx);
  F3 c10 = lerp3(ld(i0, j1, k0), ld(i1, j1, k0), tx);
  F3 c01 = lerp3(ld(i0, j0, k1), ld(i1, j0, k1), tx);
  F3 c11 = lerp3(ld(i0, j1, k1), ld(i1, j1, k1), tx);
  return lerp3(lerp3(c00, c10, ty), lerp3(c01, c11, ty), tz);
}

// The camera march's brick map: over each brick and the next cell past it on each axis (every corner a sample
// with lower corner in the brick can blend), 2 when some smoke is > 0, plus 1 when the temperature may glow. The
// temperature cannot glow when its largest value is below glow_start by more than the rounding of three lerps (16
// ulps). A sample in a brick without smoke has alpha 0, one where nothing glows glow 0; where neither holds it adds
// nothing. Outside the smoke a temperature of one value <= glow_start does not glow either: its blends are that value to
// a few ulps (exactly, for 0 and powers of two), and ulps above glow_start, which the blends of some other values have
// at a sample in fifty, are not taken for glow there. Within the smoke they are, as they are without the map.
template <class T>
__global__ void __launch_bounds__(32 * ROW_WARPS) k_march_bricks(Dims d, const T* __restrict__ smoke, const T* __restrict__ temperature,
                                                                 float glow_start, float* __restrict__ bricks) {
  BrickRow r;
  if (!brick_row(d, r)) return;
  float most = -3.0e38f, hot = -3.0e38f, cold = 3.0e38f;
#pragma unroll
  for (int a = 0; a <= BRICK; ++a)
#pragma unroll
    for (int b = 0; b <= BRICK; ++b) {
      const int c = at(d, imin_(r.i + a, d.n0 - 1), imin_(r.j + b, d.n1 - 1), r.k);
      most = fmaxf(most, ldg_f(smoke + c));
      const float t = ldg_f(temperature + c);
      hot = fmaxf(hot, t);
      cold = fminf(cold, t);
    }
  auto larger = [](float x, float y) { return fmaxf(x, y); };
  most = over_columns(most, larger);
  hot = over_columns(hot, larger);
  cold = over_columns(cold, [](float x, float y) { return fminf(x, y); });
  const bool smoky = most > 0.0f;
  const bool dark = (hot + fabsf(hot) * 9.5367432e-7f < glow_start) || (!smoky && cold == hot && hot <= glow_start);
  if (r.brick >= 0) bricks[r.brick] = (smoky ? 2.0f : 0.0f) + (dark ? 0.0f : 1.0f);
}

// sample_index_space from its axes; p: the lower corner.
template <class T>
__device__ __forceinline__ float sample_axes(const T* __restrict__ p, const Axis1& x, const Axis1& y, const Axis1& z) {
  const float c00 = lerp_w(ldg_f(p), ldg_f(p + x.step), x);
  const float c10 = lerp_w(ldg_f(p + y.step), ldg_f(p + x.step + y.step), x);
  const float c01 = lerp_w(ldg_f(p + z.step), ldg_f(p + x.step + z.step), x);
  const float c11 = lerp_w(ldg_f(p + y.step + z.step), ldg_f(p + x.step + y.step + z.step), x);
  return lerp_w(lerp_w(c00, c10, y), lerp_w(c01, c11, y), z);
}

struct MarchArgs {
  PlumeGridInfo info;
  PlumeViewParams view;
  PlumeLookParams look;
  Dims d, dg, dl;
};

// raymarch_kernel (raymarch.py:86-140): RAY_LANES lanes per pixel take consecutive samples of its ray, and then add their
// terms in the order of the samples, each lane the same sums: a ray is one chain of transmittances, but a sample's
// density, light and glow are not part of it.
// Terms that are exactly zero are not evaluated: with no smoke at a sample (all eight corners <= 0 in the
// brick map, or a blend <= 0) alpha is exactly 0, so the exp and the light or gradient sample are skipped and the lane's
// term is +0, its factor 1; with no glow the pow is skipped (it would add +0); where the last lane's sample lies among
// empty bricks, the march steps over as many samples as cannot leave them. Every result bit is unchanged.
//
// Bound by instruction issue (75% of the slots). Measured on B200 at 128x192x128, 400 x 404 pixels: a thread per pixel
// 390 us (2.7 warps a scheduler, waiting for loads and for the longest rays), 4 lanes 155 us, 8 lanes 143 us, 16 lanes
// 165 us; at 96x144x96 with the normal field 139 us at 4 lanes and 100 us at 8.
constexpr int RAY_LANES = 8;

template <class T>
__global__ void __launch_bounds__(256, 4) k_raymarch(const __grid_constant__ MarchArgs a, const T* __restrict__ smoke,
                                                     const T* __restrict__ temperature, const float* __restrict__ gradient,
                                                     const float* __restrict__ light, float* __restrict__ image, int height,
                                                     int width, const float* __restrict__ bricks) {
  const int lane = threadIdx.x % RAY_LANES;
  const long ray = ((long)blockIdx.x * blockDim.x + threadIdx.x) / RAY_LANES;
  const int pixel = ray < (long)height * width ? (int)ray : height * width - 1;
  const int px = pixel % width, py = pixel / width;
  const PlumeViewParams& view = a.view;
  const PlumeLookParams& look = a.look;
  const PlumeGridInfo& info = a.info;
  F3 right = f3(view.right[0], view.right[1], view.right[2]);
  F3 up = f3(view.up[0], view.up[1], view.up[2]);
  F3 toward = f3(view.toward[0], view.toward[1], view.toward[2]);
  float plane_x = view.left_m + ((float)px + 0.5f) * view.pixel_m;  // pixel_ray (raymarch.py:72-83)
  float plane_y = view.top_m - ((float)py + 0.5f) * view.pixel_m;
  F3 origin = add3(add3(mul3(right, plane_x), mul3(up, plane_y)), mul3(toward, 1.0e4f));
  F3 direction = f3(-toward[0], -toward[1], -toward[2]);
  if (view.perspective == 1) {
    origin = f3(view.eye[0], view.eye[1], view.eye[2]);
    direction = normalize3(sub3(add3(mul3(right, plane_x), mul3(up, plane_y)), toward));
  }
  F3 box_origin = f3(info.origin_m[0], info.origin_m[1], info.origin_m[2]);
  F3 box_max = add3(box_origin, mul3(f3((float)info.dims[0], (float)info.dims[1], (float)info.dims[2]), info.cell_m));
  float s0, s1;
  slab_range(origin, direction, box_origin, box_max, s0, s1);
  if (view.perspective == 1) s0 = fmax_(s0, 0.0f);
  float tr = 1.0f, heat = 0.0f, shade_sum = 0.0f;
  F3 normal_sum = f3(0.0f, 0.0f, 0.0f);
  int steps = 0;
  float step_m = 0.0f;
  if (s1 > s0) {
    const float length = s1 - s0;
    steps = imin_((int)ceilf(length / (0.5f * info.cell_m)), 0x7ffffff0);  // a group's samples may pass it
    step_m = length / (float)steps;
  }
  const Dims bd = brick_dims(a.d);
  // The computed points origin + direction * (s0 + (s + 0.5) * step_m) lie within
  // (3 |t| + 2 |box coordinate| + |box origin|) * 2^-24 / cell_m + 2 |g| * 2^-24 cells of the exact line; the
  // margin is over twice that.
  float box_far = 0.0f;
#pragma unroll
  for (int c = 0; c < 3; ++c) box_far = fmaxf(box_far, fmaxf(fabsf(box_origin[c]), fabsf(box_max[c])));
  const float cells_far = (float)imax_(imax_(a.d.n0, a.d.n1), a.d.n2);
  const float margin = (8.0f * fmaxf(fabsf(s0), fabsf(s1)) + 6.0f * box_far) * 5.9604645e-8f / info.cell_m +
                       cells_far * 9.5367432e-7f + 1.0e-3f;
  const F3 delta = mul3(direction, step_m / info.cell_m);
  // samples that cross at most one cell on every axis
  const float per_cell = 1.0f / fmaxf(fmaxf(fabsf(delta[0]), fabsf(delta[1])), fabsf(delta[2]));
  const Divisor cell = divisor(info.cell_m);  // (position - origin) / cell_m: a product when cell_m is 2^-e
  const bool light_as_smoke = a.dl.n0 == a.d.n0 && a.dl.n1 == a.d.n1 && a.dl.n2 == a.d.n2;
  for (int first = 0; __any_sync(0xffffffffu, first < steps);) {
    // this lane's sample
    const int s = first + lane;
    const F3 position = add3(origin, mul3(direction, s0 + ((float)s + 0.5f) * step_m));
    const F3 g = sub3(divide3(sub3(position, box_origin), cell), f3(0.5f, 0.5f, 0.5f));
    const Axis1 x = axis_of(g[0], a.d.n0, a.d.n1 * a.d.n2), y = axis_of(g[1], a.d.n1, a.d.n2), z = axis_of(g[2], a.d.n2, 1);
    float kind = s < steps ? 3.0f : 0.0f;
    int past = s;  // the sample the march continues after
    if (bricks && s < steps) {
      const int bi = x.i0 / BRICK, bj = y.i0 / BRICK, bk = z.i0 / BRICK;
      kind = __ldg(bricks + at(bd, bi, bj, bk));
      if (kind <= 0.0f) past = past_brick(s, steps - 1, (-kind * BRICK - margin) * per_cell);
    }
    first = __shfl_sync(0xffffffffu, past, RAY_LANES - 1, RAY_LANES) + 1;
    const int corner = (x.i0 * a.d.n1 + y.i0) * a.d.n2 + z.i0;
    const float density = kind >= 2.0f ? fmax_(sample_axes(smoke + corner, x, y, z), 0.0f) : 0.0f;
    const float alpha = density > 0.0f ? 1.0f - exp_f(-look.opacity_per_density * density * step_m) : 0.0f;
    const bool hot = kind == 1.0f || kind == 3.0f;
    const float glow = hot ? fmax_(sample_axes(temperature + corner, x, y, z) - look.glow_start_k, 0.0f) : 0.0f;
    const bool glows = __any_sync(0xffffffffu, glow > 0.0f), covers = __any_sync(0xffffffffu, alpha > 0.0f);
    if (!glows && !covers) continue;
    // the transmittance before this lane's sample, and after the group's
    const float kept = alpha > 0.0f ? 1.0f - alpha : 1.0f;
    float before = tr;
#pragma unroll
    for (int l = 0; l < RAY_LANES; ++l) {
      if (l == lane) before = tr;
      tr = tr * __shfl_sync(0xffffffffu, kept, l, RAY_LANES);
    }
    if (glows) {
      float term = 0.0f;
      if (glow > 0.0f) term = glow * step_m * pow_f(before, look.smoke_hides_heat);
#pragma unroll
      for (int l = 0; l < RAY_LANES; ++l) heat = heat + __shfl_sync(0xffffffffu, term, l, RAY_LANES);
    }
    if (!covers) continue;
    if (look.shade_layout == 1) {
      float term = 0.0f;
      if (alpha > 0.0f) {
        const float lit = light_as_smoke ? sample_axes(light + corner, x, y, z) : sample_index_space(light, a.dl, g);
        term = before * alpha * (look.shade_fill + (1.0f - look.shade_fill) * lit);
      }
#pragma unroll
      for (int l = 0; l < RAY_LANES; ++l) shade_sum = shade_sum + __shfl_sync(0xffffffffu, term, l, RAY_LANES);
    } else {
      F3 term = f3(0.0f, 0.0f, 0.0f);
      if (alpha > 0.0f) {
        const F3 slope = sample_vec(gradient, a.dg, g);
        if (len3(slope) > 1.0e-9f) term = mul3(normalize3(slope), before * alpha);
      }
#pragma unroll
      for (int l = 0; l < RAY_LANES; ++l)
        normal_sum = sub3(normal_sum, f3(__shfl_sync(0xffffffffu, term[0], l, RAY_LANES),
                                         __shfl_sync(0xffffffffu, term[1], l, RAY_LANES),
                                         __shfl_sync(0xffffffffu, term[2], l, RAY_LANES)));
    }
  }
  if (lane != 0 || ray >= (long)height * width) return;
  float thickness = 1.0f - tr;
  float* out = image + ((size_t)py * width + px) * 5;
  out[0] = heat;
  out[1] = thickness;
  if (look.shade_layout == 1) {
    out[2] = shade_sum;
    out[3] = 0.0f;
    out[4] = 0.0f;
    return;
  }
  F3 facing = f3(0.0f, 0.0f, 1.0f);
  F3 normal = facing;
  F3 cam = f3(dot3(normal_sum, right), dot3(normal_sum, up), dot3(normal_sum, toward));
  if (len3(cam) > 1.0e-9f) {
    normal = normalize3(cam);
    normal = f3(normal[0], normal[1], fabsf(normal[2]));
    float weight = clampf_(thickness / look.normal_fade_thickness, 0.0f, 1.0f);
    normal = normalize3(lerp3(facing, normal, weight));
  }
  out[2] = normal[0];
  out[3] = normal[1];
  out[4] = normal[2];
}

static bool valid_shape(const int32_t* s) {
  return s && s[0] >= 1 && s[1] >= 1 && s[2] >= 1 && (long long)s[0] * s[1] * s[2] * 3 < (1LL << 31);
}

}  // namespace plume

using namespace plume;

extern "C" long long plume_brick_floats(const int32_t shape[3]) {
  if (!valid_shape(shape)) return fail(PLUME_ERR_INVALID, "brick_floats: bad shape");
  const Dims b = brick_dims(Dims{shape[0], shape[1], shape[2]});
  return 2LL * b.n0 * b.n1 * b.n2;  // the map, and the one its empty bricks' reach is formed from
}

namespace plume {

template <class T>
static int light_volume(const Dims& d, const T* smoke, F3 toward, float cell_m, float opacity, float* light,
                        float* bricks, int march_cells, cudaStream_t st) {
  if (bricks) {
    const Dims b = brick_dims(d);
    float* map = bricks + (size_t)b.n0 * b.n1 * b.n2;
    k_brick_max<T><<<brick_row_grid(b), dim3(32, ROW_WARPS), 0, st>>>(d, smoke, map);
    int status = launch_status("smoke brick map");
    if (status != PLUME_OK || (status = brick_reach(b, map, bricks, st)) != PLUME_OK) return status;
  }
  const dim3 grid((unsigned)((d.n2 + 31) / 32) * ((d.n1 + LIGHT_ROWS - 1) / LIGHT_ROWS), 1, d.n0);
  k_light_volume<T><<<grid, dim3(32, LIGHT_ROWS), 0, st>>>(d, smoke, toward, cell_m, opacity, light, bricks, march_cells);
  return launch_status("light volume");
}

template <class T>
static int normal_field(const Dims& d, const T* smoke, float* blurred, float* scratch, float* gradient, int radius,
                        const BlurWeights& weights, cudaStream_t st) {
  k_blur_axis<0><<<cell_grid((d.n0 + BLUR_CELLS - 1) / BLUR_CELLS, d.n1, d.n2), cell_block(), 0, st>>>(d, smoke, blurred, radius, weights);
  int status = launch_status("blur");
  if (status != PLUME_OK) return status;
  k_blur_axis<1><<<cell_grid(d.n0, (d.n1 + BLUR_CELLS - 1) / BLUR_CELLS, d.n2), cell_block(), 0, st>>>(d, blurred, scratch, radius, weights);
  if ((status = launch_status("blur")) != PLUME_OK) return status;
  k_blur_axis<2><<<cell_grid(d.n0, d.n1, d.n2), cell_block(), 0, st>>>(d, scratch, blurred, radius, weights);
  if ((status = launch_status("blur")) != PLUME_OK) return status;
  k_gradient<<<dim3((d.n2 + 31) / 32, (d.n1 + GRADIENT_ROWS - 1) / GRADIENT_ROWS, d.n0), dim3(32, GRADIENT_ROWS), 0, st>>>(d, blurred, gradient);
  return launch_status("gradient");
}

template <class T>
static int brick_max(const Dims& d, const T* field, float* bricks, cudaStream_t st) {
  const Dims b = brick_dims(d);
  k_brick_max<T><<<brick_row_grid(b), dim3(32, ROW_WARPS), 0, st>>>(d, field, bricks);
  return launch_status("brick map");
}

template <class T>
static int raymarch(const MarchArgs& a, const T* smoke, const T* temperature, const float* gradient, const float* light,
                    float* image, int height, int width, float* bricks, cudaStream_t st) {
  if (bricks) {  // the brick map of exactly the smoke and temperature being marched
    const Dims b = brick_dims(a.d);
    float* map = bricks + (size_t)b.n0 * b.n1 * b.n2;
    k_march_bricks<T><<<brick_row_grid(b), dim3(32, ROW_WARPS), 0, st>>>(a.d, smoke, temperature, a.look.glow_start_k, map);
    int status = launch_status("march brick map");
    if (status != PLUME_OK || (status = brick_reach(b, map, bricks, st)) != PLUME_OK) return status;
  }
  const long lanes = (long)height * width * RAY_LANES;
  k_raymarch<T><<<(unsigned)((lanes + 255) / 256), 256, 0, st>>>(a, smoke, temperature, gradient, light, image, height,
                                                              width, bricks);
  return launch_status("raymarch");
}

// Returns the call for the storage code (its arrays of float, bfloat16 or half).
#define PLUME_BY_STORAGE(storage, call_f32, call_bf16, call_f16, what) \
  switch (storage) {                                                 \
    case PLUME_STORAGE_F32: return call_f32;                           \
    case PLUME_STORAGE_BF16: return call_bf16;                         \
    case PLUME_STORAGE_F16: return call_f16;                           \
  }                                                                    \
  return fail(PLUME_ERR_INVALID, "%s: storage %d", what, storage);

}  // namespace plume

static int light_volume_call(const int32_t shape[3], const void* smoke, int32_t storage, const float toward_light[3],
                             float cell_m, float opacity_per_density, float* light, float* bricks, int march_cells,
                             void* stream) {
  const Dims d{shape[0], shape[1], shape[2]};
  const F3 toward = f3(toward_light[0], toward_light[1], toward_light[2]);
  cudaStream_t st = as_stream(stream);
  PLUME_BY_STORAGE(storage,
                   light_volume(d, static_cast<const float*>(smoke), toward, cell_m, opacity_per_density, light, bricks,
                                march_cells, st),
                   light_volume(d, static_cast<const __nv_bfloat16*>(smoke), toward, cell_m, opacity_per_density, light,
                                bricks, march_cells, st),
                   light_volume(d, static_cast<const __half*>(smoke), toward, cell_m, opacity_per_density, light, bricks,
                                march_cells, st),
                   "light_volume")
}

extern "C" int plume_light_volume(const int32_t shape[3], const void* smoke, int32_t storage, const float toward_light[3],
                                  float cell_m, float opacity_per_density, float* light, float* bricks, void* stream) {
  if (!valid_shape(shape) || !smoke || !toward_light || !light) return fail(PLUME_ERR_INVALID, "light_volume: bad argument");
  return light_volume_call(shape, smoke, storage, toward_light, cell_m, opacity_per_density, light, bricks, 0, stream);
}

extern "C" int plume_march_light_volume(const int32_t shape[3], const void* smoke, int32_t storage,
                                        const float toward_light[3], float cell_m, float opacity_per_density,
                                        float* light, float* bricks, void* stream) {
  if (!valid_shape(shape) || !smoke || !toward_light || !light || !bricks)
    return fail(PLUME_ERR_INVALID, "march_light_volume: bad argument");
  return light_volume_call(shape, smoke, storage, toward_light, cell_m, opacity_per_density, light, bricks, 1, stream);
}

extern "C" int plume_normal_field(const int32_t shape[3], const void* smoke, int32_t storage, float* blurred,
                                  float* scratch, float* gradient, const float* weights_host, int32_t radius,
                                  void* stream) {
  if (!valid_shape(shape) || !smoke || !blurred || !scratch || !gradient || !weights_host || radius < 0 ||
      2 * radius + 1 > MAX_BLUR_TAPS)
    return fail(PLUME_ERR_INVALID, "normal_field: bad argument");
  cudaStream_t st = as_stream(stream);
  BlurWeights weights = {};
  std::copy(weights_host, weights_host + 2 * radius + 1, weights.w);
  const Dims d{shape[0], shape[1], shape[2]};
  PLUME_BY_STORAGE(storage, normal_field(d, static_cast<const float*>(smoke), blurred, scratch, gradient, radius, weights, st),
                   normal_field(d, static_cast<const __nv_bfloat16*>(smoke), blurred, scratch, gradient, radius, weights, st),
                   normal_field(d, static_cast<const __half*>(smoke), blurred, scratch, gradient, radius, weights, st),
                   "normal_field")
}

extern "C" int plume_brick_max(const int32_t shape[3], const void* field, int32_t storage, float* bricks, void* stream) {
  if (!valid_shape(shape) || !field || !bricks) return fail(PLUME_ERR_INVALID, "brick_max: bad argument");
  const Dims d{shape[0], shape[1], shape[2]};
  cudaStream_t st = as_stream(stream);
  PLUME_BY_STORAGE(storage, brick_max(d, static_cast<const float*>(field), bricks, st),
                   brick_max(d, static_cast<const __nv_bfloat16*>(field), bricks, st),
                   brick_max(d, static_cast<const __half*>(field), bricks, st), "brick_max")
}

extern "C" int plume_raymarch(const PlumeGridInfo* info, const void* smoke, const void* temperature, int32_t storage,
                              const float* gradient, const int32_t gradient_shape[3], const float* light,
                              const int32_t light_shape[3], const PlumeViewParams* view, const PlumeLookParams* look,
                              float* image, int32_t height, int32_t width, float* bricks, void* stream) {
  if (!info || !smoke || !temperature || !gradient || !light || !view || !look || !image || height < 1 || width < 1 ||
      (long long)height * width >= (1LL << 31) || !valid_shape(info->dims) || !valid_shape(gradient_shape) || !valid_shape(light_shape))
    return fail(PLUME_ERR_INVALID, "raymarch: bad argument");
  MarchArgs a;
  a.info = *info;
  a.view = *view;
  a.look = *look;
  a.d = Dims{info->dims[0], info->dims[1], info->dims[2]};
  a.dg = Dims{gradient_shape[0], gradient_shape[1], gradient_shape[2]};
  a.dl = Dims{light_shape[0], light_shape[1], light_shape[2]};
  cudaStream_t st = as_stream(stream);
  PLUME_BY_STORAGE(storage,
                   raymarch(a, static_cast<const float*>(smoke), static_cast<const float*>(temperature), gradient, light,
                            image, height, width, bricks, st),
                   raymarch(a, static_cast<const __nv_bfloat16*>(smoke), static_cast<const __nv_bfloat16*>(temperature),
                            gradient, light, image, height, width, bricks, st),
                   raymarch(a, static_cast<const __half*>(smoke), static_cast<const __half*>(temperature), gradient,
                            light, image, height, width, bricks, st),
                   "raymarch")
}
