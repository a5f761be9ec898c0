"""Hierarchies of a caller's own whose levels do not halve, rounding up, as Multigrid's do (some that round down, one that
steps by other factors, one with a level of more than half the cells): the oracle's pressure bit for bit, by every
strategy. The passes and the cluster written for halved levels are not to be reached by them."""

import dataclasses

import numpy as np
import pytest
import torch

from oracle import oracle as O
from plume_b200 import _native as N
from support import ALL_CLOSED, OPEN, host
from test_gpu_solver import seeded_pair

pytestmark = pytest.mark.gpu

HIERARCHIES = [
    [(13, 11, 9), (6, 5, 4), (3, 2, 2)],
    [(64, 36, 65), (32, 18, 32), (16, 9, 16), (8, 4, 8), (4, 2, 4)],
    [(45, 70, 51), (22, 35, 25), (11, 17, 12), (5, 8, 6), (2, 4, 3)],
    [(40, 30, 28), (20, 15, 14), (9, 7, 7), (5, 4, 4), (2, 2, 2)],  # halves above and below the third level
    [(20, 18, 16), (7, 9, 5), (3, 3, 3)],
    [(12, 10, 8), (8, 5, 4), (4, 2, 2)],  # coarse cells without children
    [(31, 3, 4), (15, 1, 2)],
]


def own_levels(o, c, dims):
    """The same levels for the oracle's solve and the library's."""
    from plume_b200.sim.grid import make_info
    from plume_b200.sim.multigrid import Level, Multigrid

    theirs, ours = O.Multigrid(o, 2, 2), Multigrid(c, 2, 2)
    theirs.levels, ours.levels = theirs.levels[:1], ours.levels[:1]
    for n, cells in enumerate(dims[1:], 1):
        above, top = theirs.levels[-1].info, c.info
        fill = (1.0, 0.75, 1.0) if n == 2 else (1.0, 1.0, 1.0)
        args = (cells, above.cell_m * 2.0, list(top.origin_m), list(top.open_lo), list(top.open_hi))
        theirs.levels.append(O.Level(O.make_info(*args, o.precision, fill_hi=list(fill), ghost_gap=0.5 / 2.0**n), cells,
                                     *(np.zeros(cells, dtype=np.float32) for _ in range(3))))
        ours.levels.append(Level(make_info(*args, fill, 0.5 / 2.0**n), cells, *(torch.zeros(cells, device="cuda:0") for _ in range(3))))
    return theirs, ours


@pytest.mark.parametrize("faces", [OPEN, ALL_CLOSED], ids=["open", "closed"])
@pytest.mark.parametrize("dims", HIERARCHIES, ids=lambda d: "-".join("x".join(map(str, c)) for c in d))
def test_pressure(cuda_device, dims, faces):
    from plume_b200.sim.multigrid import solver_tuning, tune_solver
    from plume_b200.sim.pressure import compute_divergence

    saved = solver_tuning()
    o, c = seeded_pair(dims[0], faces)
    theirs, ours = own_levels(o, c, dims)
    compute_divergence(c)
    start = c.pressure.clone()
    O.compute_divergence(o)
    theirs(o)
    expected = np.array(o.pressure)
    try:
        for change in ({}, {"bottom_max_cells": 0}, {"bottom_max_cells": 1 << 20}, {"bottom_kind": 1}, {"tiled_min_cells": 1}):
            tune_solver(dataclasses.replace(saved, **change))
            c.pressure.copy_(start)
            ours(c)
            assert np.array_equal(host(c.pressure), expected, equal_nan=True), change
    finally:
        tune_solver(saved)
    threshold = N.lib().plume_split_min_cells()
    try:
        N.call("plume_tune_split", 1)
        c.pressure.copy_(start)
        scratch = torch.empty(N.lib().plume_split_scratch_floats(c.info), device="cuda:0")
        N.call("plume_multigrid_split", ours.native_levels(c), len(dims), 2, 2, N.ptr(scratch), N.stream())
    finally:
        N.call("plume_tune_split", threshold)
    assert np.array_equal(host(c.pressure), expected, equal_nan=True), "split"
