/* The light march's rule for samples that need no clamp (plume_b200/csrc/light_range.cuh, compiled here as it is), held
 * to the sample points as the kernel computes them: every admitted sample's lower corner and the next cell must lie in
 * the axis. A march is monotone along an axis, so the first and last admitted samples stand for all; a few between are
 * checked too. Prints the marches with a sample outside, the marches with admitted samples, and all marches. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include <algorithm>

#define __host__
#define __device__
#define __forceinline__ inline
#include "light_range.cuh"

int main() {
  const int sizes[] = {1, 2, 3, 4, 5, 9, 33, 70, 127, 128, 129, 1000, 4097, 65536, 100003, (1 << 21) + 1, (1 << 22) - 1};
  const float caps[] = {0.2f, 0.5f, 1.0f, 3.0f, 40.0f, 300.0f, 5000.0f, 2.0e5f, 2.0e6f};
  const int run = 4;
  uint64_t bad = 0, with_runs = 0, all = 0;
  for (int n : sizes)
    for (int corner : {0, 1, 2, 3, n / 2, n - 4, n - 3, n - 2, n - 1}) {
      if (corner < 0 || corner >= n) continue;
      for (double exponent = -14.0; exponent <= 0.0; exponent += 0.02)
        for (int sign = -1; sign <= 1; sign += 2)
          for (float cap : caps) {
            const float toward = (float)(sign * pow(10.0, exponent)), at = (float)corner;
            const float room = (sign > 0 ? (float)n - (at + 0.5f) : at + 0.5f) / fabsf(toward);  // to the box face
            const float length = std::min(room, cap);
            const int steps = (int)ceilf(length / 0.5f);
            if (steps < 1) continue;
            const float step = length / (float)steps;
            const float margin = plume::march_margin(length, n);
            const float inner = plume::samples_inside(toward * step, at, n, margin);
            const float to = plume::last_run(inner, (float)(steps - 1), run);
            ++all;
            if (!(to >= 0.0f)) continue;
            ++with_runs;
            const int final = (int)to + run - 1;
            bool inside = final <= steps - 1;
            for (int pick = 0; pick <= 24; ++pick) {
              const int s = pick < 8 ? std::min(pick, final)
                                     : (pick < 16 ? std::max(final - (pick - 8), 0) : (int)((int64_t)final * (pick - 15) / 10));
              const float x = fmaf(toward, ((float)s + 0.5f) * step, at);
              inside = inside && x >= 0.0f && floorf(x) <= (float)(n - 2);
            }
            bad += !inside;
          }
    }
  printf("%llu %llu %llu\n", (unsigned long long)bad, (unsigned long long)with_runs, (unsigned long long)all);
  return 0;
}
