// Which form of the velocity march (advect.cu) a call takes, and in how many segments. Host code without CUDA, so that the
// rules can be checked by themselves.
#pragma once

#include <algorithm>
#include <cmath>

namespace plume {
namespace mac {

// 1 or 2: that many elements per thread; 3: k_mac_velocity_long.
//
// Two elements share a tile's halo of hats and its staging between more elements, one leaves more blocks where the grid is
// small. The line lies where two have stopped losing. Measured on B200, two against one: 64x96x64 68 and 66 us, 80x100x80
// 97 and 95; between, by how the tiles fall: 75x113x91 103 and 108, 96x96x96 116 and 110, 96x144x96 148 and 155, 112x112x112
// 157 and 173, 112x144x112 (1.8 million cells) 209 and 200; from two million on: 128x128x128 221 and 230, 112x168x112 239
// and 240, 128x144x128 241 and 257, 128x192x128 306 and 320, 160x160x160 372 and 410, 256x384x256 1975 and 2104.
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

// Segments along x of the march of `ept` elements per thread in tiles of ept * ty rows and tz columns, by a cost fitted to
// measured times: a block of `len` planes takes len + 3 plane times (its prologue forms two more hat planes), each
// 1.75 + 2.3 w long with w waves of resident blocks sharing the SMs, half of a last wave's missing blocks counted. Measured
// on B200 with segments of 5 planes against 10 at 38x48x38: 27 against 33 us; with 5 segments against 10 at 128x192x128
// (one element a thread): 305 against 323 us; with 6 against 5 at 160x240x160 (two elements): 512 against 549 us.
//
// The cost depends on the length alone, so each length is tried once, with the fewest segments that have it: about
// 2 sqrt(nx) tries, where every count up to nx / 4 took 0.2 ms of host time at 2^16 planes and 14 ms at 2^22. The three
// components' segments together stay within a launch's 65535 blocks. `set` (PLUME_MAC_VELOCITY_SEGS > 0) overrides the count.
constexpr int MOST_SEGMENTS = 65535 / 3 - 1;

inline int march_segments(const int* dims, int ept, int ty, int tz, int set) {
  const int nx = dims[0];
  if (set > 0) return std::min(set, std::min(nx, MOST_SEGMENTS));
  const double resident = 148.0 * (ept == 2 ? 2 : 3);
  auto tiles = [&](int g) {
    const int rows = ept * ty;
    return (double)((dims[1] + (g == 1) + rows - 1) / rows) * ((dims[2] + (g == 2) + tz - 1) / tz);
  };
  const int most = std::min(std::max(1, nx / 4), MOST_SEGMENTS);
  int best = 1;
  double least = 0.0;
  for (int segs = 1; segs <= most;) {
    const int len = (nx + segs - 1) / segs;
    double blocks = 0.0;
    for (int g = 0; g < 3; ++g) blocks += tiles(g) * ((nx + (g == 0) + len - 1) / len);
    double w = blocks / resident;
    if (w > 1.0) w = 0.5 * (w + std::ceil(w));
    const double cost = (len + 3.0) * (1.75 + 2.3 * w);
    if (segs == 1 || cost < least) {
      best = segs;
      least = cost;
    }
    if (len == 1) break;
    segs = (nx + len - 2) / (len - 1);  // the fewest whose segments are shorter
  }
  return best;
}

}  // namespace mac
}  // namespace plume
