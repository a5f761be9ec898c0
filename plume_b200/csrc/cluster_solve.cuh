// The small levels of the pressure solve in one launch of one thread-block cluster (cluster_solve.cu).
#pragma once

#include <stddef.h>

#include "common.cuh"

namespace plume {

constexpr int CLUSTER_MAX_LEVELS = 8;

// What one launch solves: levels[0 .. count - 1] of a hierarchy, `cycles` V-cycles of `sweeps` sweeps a side (the
// last level: `last_sweeps` of `last_relaxation`). Levels from `single_from` on live in CTA 0 alone, those before
// it in x-slabs over `ctas` CTAs (1, 8 or 16). Level 0's pressure is read from and left in levels[0].q.
struct ClusterSolve {
  const PlumeLevel* levels;
  int count;
  int single_from;
  int ctas;
  int cycles, sweeps;
  bool from_zero;  // level 0's pressure starts at 0, whatever its array holds
  bool store_all;  // leave the coarser levels' arrays as the last cycle had them; else only level 0's pressure
  int last_sweeps;
  float last_relaxation;
};

// Whether a level has half of another's cells on every axis, rounded up (multigrid.py:71-121): what the passes between two
// levels with several cells a thread, and the cluster, are written for.
inline bool halves(const PlumeGridInfo& fine, const PlumeGridInfo& coarse) {
  for (int a = 0; a < 3; ++a)
    if (coarse.dims[a] != fine.dims[a] / 2 + fine.dims[a] % 2) return false;
  return true;
}
// Whether a level is small enough for one CTA (one cell of each colour per thread).
bool cluster_solve_single(const PlumeGridInfo& info);
// Dynamic shared memory per CTA of such a solve (bytes), and whether this device can run it.
size_t cluster_solve_bytes(const ClusterSolve& solve);
bool cluster_solve_runs(const ClusterSolve& solve);
// Sets the kernel's attributes on the current device (once per device; call it outside any stream capture).
int prepare_cluster_solve();
int launch_cluster_solve(const ClusterSolve& solve, bool dependent, cudaStream_t st);

}  // namespace plume
