// Which form of the velocity march (advect.cu) a call takes. Host code without CUDA, so that the rule can be checked by itself.
#pragma once

#include <algorithm>
#include <cmath>

namespace plume {
namespace mac {

// 1 or 2: that many elements per thread; 3: k_mac_velocity_long.
//
// Two elements share a tile's halo of hats and its staging between more elements, one leaves more blocks where the grid is
// small. Measured on B200, two against one: 128x192x128 295 and 305 us, 160x240x160 (bfloat16) 512 and 550 us, 256x384x256
// 1975 and 2104 us; 80x100x80 98 and 90 us, 64x96x64 70 and 59 us.
//
// The long form takes the axes whose coordinates split_bits does not cover, and a time step that is infinite or no number:
// the other two keep a trace that leaves the staged planes inside them by giving it a zero velocity, and zero times such a
// step is no number, which leads out of them.
//
// `set` (PLUME_MAC_ELEMENTS = 1, 2 or 3) overrides the choice where it can, for measurements and to compare the kernels:
// they give the same floats.
inline int march_form(const int* dims, float dt, int set) {
  if (std::max(dims[0], std::max(dims[1], dims[2])) >= (1 << 22) - 1 || !std::isfinite(dt)) return 3;
  if (set >= 1 && set <= 3) return set;
  return (long)dims[0] * dims[1] * dims[2] >= 2000000 ? 2 : 1;
}

}  // namespace mac
}  // namespace plume
