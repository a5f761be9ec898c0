// The stencils of a pressure level by cell class. A cell's couplings depend on its position along each axis only
// through four classes (first cell, inner, last but one, last): fill_hi and the faces enter nowhere else
// (poisson.cuh). So 64 entries hold every stencil of a level, with neighbor_sum's floats.
#pragma once

#include "poisson.cuh"

namespace plume {

// neighbor_sum's couplings (x-, x+, y-, y+, z-, z+; a ghost's coupling, or 0 for a closed face, where the neighbour
// is outside the level), their sum, cell_volume * cell_m * cell_m, and the reciprocals of those two in double.
struct __align__(16) ClassStencil {
  float c[6];
  float sc, vc;
  double inv, inv_vc;
};

__host__ __device__ __forceinline__ int class_of(int index, int n) {
  return index == n - 1 ? 3 : (index == n - 2 ? 2 : (index == 0 ? 0 : 1));
}
__host__ __device__ __forceinline__ int class_index(int cls, int n) {  // a cell index of the class (any, when it has none)
  return cls == 3 ? n - 1 : (cls == 2 ? (n > 2 ? n - 2 : 0) : (cls == 0 ? 0 : (n > 1 ? 1 : 0)));
}

// x / d, correctly rounded, as the product with a double within 2^-52 (relative) of 1 / d. The product is then within
// 2^-51 of x / d. A quotient of two floats never is the midpoint m of two neighbouring normal
// floats, and x - m d, a multiple of the last place of the 49-bit product m d, then differs from 0 by at least
// 2^-49 of x: so the product and x / d round to the same float. (The range of a double holds every case: zeros,
// infinities and NaN come out as the division's too.) Unlike the division, and unlike a float reciprocal with
// remainder steps, this has no branch for operands out of range: where few warps run code once through, a branch
// over a slow path costs more than the arithmetic, since the instructions after it are fetched late. Measured on
// B200, one dependent update on one warp: 115 cycles, with float remainder steps behind a range test 350 (118 only
// as a loop of that body alone).
__device__ __forceinline__ float quotient(float x, double inv) { return (float)((double)x * inv); }

// The table of a level as a kernel parameter: entry 16 a + 4 b + c for the classes a, b, c along x, y, z.
struct LevelTable {
  ClassStencil e[64];
};

inline LevelTable level_table(const PlumeGridInfo& info) {
  LevelTable t;
  for (int n = 0; n < 64; ++n) {
    const int cell[3] = {class_index(n / 16, info.dims[0]), class_index(n / 4 % 4, info.dims[1]),
                         class_index(n % 4, info.dims[2])};
    float fill[3];
    for (int a = 0; a < 3; ++a) fill[a] = cell[a] == info.dims[a] - 1 ? info.fill_hi[a] : 1.0f;
    ClassStencil& e = t.e[n];
    e.sc = 0.0f;
    for (int face = 0; face < 6; ++face) {
      const int axis = face / 2, next = cell[axis] + (face % 2 ? 1 : -1);
      const float area = fill[axis == 0 ? 1 : 0] * fill[axis == 2 ? 1 : 2];
      const bool open = face % 2 ? info.open_hi[axis] == 1 : info.open_lo[axis] == 1;
      e.c[face] = 0.0f;
      if (next >= 0 && next < info.dims[axis])
        e.c[face] = area / (0.5f * (fill[axis] + (next == info.dims[axis] - 1 ? info.fill_hi[axis] : 1.0f)));
      else if (open) e.c[face] = area / (0.5f * fill[axis] + info.ghost_gap);
      e.sc = e.sc + e.c[face];
    }
    e.vc = fill[0] * fill[1] * fill[2] * info.cell_m * info.cell_m;
    e.inv = 1.0 / (double)e.sc;
    e.inv_vc = 1.0 / (double)e.vc;
  }
  return t;
}

}  // namespace plume
