// Which samples of a light march need no clamp (render.cu). Host code too, so that the rule can be checked on the CPU.
#pragma once

#include <math.h>

namespace plume {

// Bounds twice the float error, in cells, of a computed sample point (corner + toward * ((s + 0.5) * step)) against the
// exact line through the march, over a march of `length` cells in a grid of at most `widest` cells on an axis.
__host__ __device__ __forceinline__ float march_margin(float length, int widest) {
  return (4.0f * length + 4.0f * (float)(widest + 1)) * 5.9604645e-8f + 1.0e-3f;
}

// How many steps of `delta` from the cell `corner` stay in [0, n - 1) by more than `margin` cells, possibly negative; none
// when delta is no number, or so small that a sample's side of 0 is a matter of rounding. The line starts inside except
// in the last cell, which a march downward leaves with its first half step: when that is no longer than the margin, a
// sample may still round to n - 1 itself, and there are none either.
__host__ __device__ __forceinline__ float samples_inside(float delta, float corner, int n, float margin) {
  const float last = (float)(n - 1);
  if (!(fabsf(delta) > 1.0e-12f)) return fabsf(delta) <= 1.0e-12f && corner >= 1.0f && corner < last ? 3.0e38f : 0.0f;
  if (delta < 0.0f && corner >= last && !(-0.5f * delta > margin)) return 0.0f;
  return ((delta > 0.0f ? last - corner : corner) - margin) / fabsf(delta);
}

// The last sample that a run of `run` of them may start from, for a march of samples 0 .. end of which `inner` steps lie
// inside on every axis: all of a run from there or before are inside.
__host__ __device__ __forceinline__ float last_run(float inner, float end, int run) {
  return fminf(floorf(inner) - 1.0f, end) - (float)(run - 1);
}

}  // namespace plume
