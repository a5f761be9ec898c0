/* march_segments (plume_b200/csrc/march_plan.cuh, compiled here as it is) against the same cost tried at every count of
 * segments. Prints the grids whose counts differ, the most blocks along z of any grid, and the milliseconds of 100 calls
 * at the longest axis. */
#include <stdio.h>

#include <chrono>

#include "march_plan.cuh"

static int every_count(const int* dims, int ept, int ty, int tz) {
  const int nx = dims[0];
  int best = 1;
  double least = 0.0;
  for (int segs = 1; segs <= std::min(std::max(1, nx / 4), plume::mac::MOST_SEGMENTS); ++segs) {
    const int len = (nx + segs - 1) / segs;
    double blocks = 0.0;
    for (int g = 0; g < 3; ++g) {
      const int rows = ept * ty;
      const double tiles = (double)((dims[1] + (g == 1) + rows - 1) / rows) * ((dims[2] + (g == 2) + tz - 1) / tz);
      blocks += tiles * ((nx + (g == 0) + len - 1) / len);
    }
    double w = blocks / (148.0 * (ept == 2 ? 2 : 3));
    if (w > 1.0) w = 0.5 * (w + std::ceil(w));
    const double cost = (len + 3.0) * (1.75 + 2.3 * w);
    if (segs == 1 || cost < least) {
      best = segs;
      least = cost;
    }
  }
  return best;
}

int main() {
  const int axis[] = {1, 2, 3, 7, 8, 15, 38, 64, 75, 96, 128, 160, 256, 384, 1000, 4096, 65536};
  int differ = 0, most = 0;
  auto look = [&](const int* dims, int ept, bool every) {
    const int segs = plume::mac::march_segments(dims, ept, 8, 32, 0);
    if (every && segs != every_count(dims, ept, 8, 32)) ++differ;
    const int len = (dims[0] + segs - 1) / segs;
    int z = 0;
    for (int g = 0; g < 3; ++g) z += (dims[0] + (g == 0) + len - 1) / len;
    most = std::max(most, z);
  };
  for (int nx : axis)
    for (int ny : axis)
      for (int nz : axis)
        for (int ept = 1; ept <= 2; ++ept) {
          const int dims[3] = {nx, ny, nz};
          look(dims, ept, true);
        }
  for (int nx : {(1 << 22) - 2, 20000000, 100000000, 268435000}) {
    const int dims[3] = {nx, 1, 1};
    look(dims, 1, true);
  }
  const int longest[3] = {(1 << 22) - 2, 2, 2};
  const auto begin = std::chrono::steady_clock::now();
  for (int n = 0; n < 100; ++n) look(longest, 1 + n % 2, false);
  const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - begin).count();
  printf("%d %d %.3f\n", differ, most, ms);
  return 0;
}
