"""The levels that run in one thread-block cluster (cluster_solve.cu) give the oracle's pressure bit for bit, at the
sizes where its layout has edges: slabs of one to several planes, fewer planes than CTAs, a last slab that is
shorter, rows that are odd or not a multiple of four cells, a coarsest level too large for one CTA."""

import numpy as np
import pytest

from oracle import oracle as O
from support import ALL_CLOSED, OPEN, assert_same, cuda_grid, host
from test_gpu_solver import seeded_pair

pytestmark = pytest.mark.gpu

CASES = [((16, 16, 64), OPEN), ((17, 31, 23), OPEN), ((33, 40, 21), ALL_CLOSED), ((48, 48, 48), OPEN),
         ((47, 50, 50), ALL_CLOSED), ((7, 40, 45), OPEN), ((2, 60, 61), OPEN), ((61, 60, 2), ALL_CLOSED), ((65, 34, 50), OPEN),
         ((64, 64, 64), OPEN), ((80, 24, 100), ALL_CLOSED), ((3, 5, 4), OPEN), ((1, 1, 1), ALL_CLOSED), ((1, 1, 1), OPEN)]
IDS = ["x".join(map(str, cells)) + ("-open" if faces is OPEN else "-closed") for cells, faces in CASES]


@pytest.mark.parametrize("cells,faces", CASES, ids=IDS)
@pytest.mark.parametrize("cycles,sweeps", [(1, 2), (3, 3)])
def test_multigrid_matches_the_oracle(cuda_device, cells, faces, cycles, sweeps):
    from plume_b200.sim.multigrid import Multigrid
    from plume_b200.sim.pressure import project

    o, c = seeded_pair(cells, faces)
    O.project(o, O.Multigrid(o, cycles, sweeps))
    project(c, Multigrid(c, cycles, sweeps))
    assert_same(host(c.pressure), o.pressure, "pressure")


@pytest.mark.parametrize("cells,faces", CASES[:9], ids=IDS[:9])
def test_the_coarse_arrays_are_those_of_separate_launches(cuda_device, cells, faces):
    from plume_b200.sim.multigrid import Multigrid, solver_tuning, tune_solver
    from plume_b200.sim.pressure import compute_divergence
    import dataclasses

    saved = solver_tuning()
    solved = []
    try:
        for bottom in (saved.bottom_max_cells, 0):  # 0: every level by launches of its own
            tune_solver(dataclasses.replace(saved, bottom_max_cells=bottom))
            _, c = seeded_pair(cells, faces)
            compute_divergence(c)
            solve = Multigrid(c, 2, 2)
            solve(c)
            solved.append(solve)
    finally:
        tune_solver(saved)
    for n, (a, b) in enumerate(zip(solved[0].levels, solved[1].levels)):
        assert_same(host(a.q), host(b.q), f"level {n} pressure")
        assert_same(host(a.rhs), host(b.rhs), f"level {n} right-hand side")


@pytest.mark.parametrize("cells,faces", CASES, ids=IDS)
def test_gauss_seidel_matches_the_oracle(cuda_device, cells, faces):
    from plume_b200.sim.pressure import GaussSeidel, project

    o, c = seeded_pair(cells, faces)
    O.project(o, O.GaussSeidel(5))
    project(c, GaussSeidel(5))
    assert_same(host(c.pressure), o.pressure, "pressure after 5 sweeps")


def test_infinities_and_nan_spread_as_in_separate_launches(cuda_device):
    import dataclasses

    from plume_b200.sim.multigrid import Multigrid, solver_tuning, tune_solver

    saved = solver_tuning()
    got = []
    try:
        for bottom in (saved.bottom_max_cells, 0):
            tune_solver(dataclasses.replace(saved, bottom_max_cells=bottom))
            c = cuda_grid((24, 20, 28), 0.05, OPEN)
            c.divergence[3, 4, 5] = float("inf")
            c.divergence[20, 15, 9] = float("nan")
            c.divergence[12, 2, 20] = -3.0e38
            Multigrid(c, 1, 2)(c)
            got.append(host(c.pressure))
    finally:
        tune_solver(saved)
    assert np.array_equal(np.isnan(got[0]), np.isnan(got[1]))
    finite = ~np.isnan(got[0])
    assert np.array_equal(got[0][finite], got[1][finite])
