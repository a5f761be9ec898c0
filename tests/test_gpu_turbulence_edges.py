"""In the step, the turbulence potentials are formed once per edge of the grid, from a table of the noise's lattice
values where the lattice is coarse; without scratch every face forms its own four. Both give the same floats."""

import dataclasses

import numpy as np
import pytest

from plume_b200.recipe.derived import derive
from plume_b200.workloads import operator_fields, plain_step_recipe
from support import assert_same, host

pytestmark = pytest.mark.gpu

# scale in cells: 8 and 3.3 cells between lattice points (table), 1 and 0.3 (points hashed in place)
CASES = [((24, 32, 20), 8.0), ((17, 21, 13), 3.3), ((33, 16, 19), 1.0), ((16, 18, 22), 0.3), ((70, 5, 9), 8.0), ((8, 8, 8), 100.0)]


@pytest.mark.parametrize("cells,scale_cells", CASES)
@pytest.mark.parametrize("time_s,speed", [(0.0, 0.2), (1.37, 0.9)])
def test_edge_potentials_give_the_faces_own_floats(cuda_device, cells, scale_cells, time_s, speed):
    import torch

    from plume_b200 import _native as N
    from plume_b200.sim.grid import make_grid
    from plume_b200.sim.stepper import Stepper

    recipe = plain_step_recipe(cells, cycles=1)
    cell_m = recipe.domain.cell_m
    turbulence = dataclasses.replace(recipe.forces.turbulence, scale_m=scale_cells * cell_m, strength_mps2=3.0, speed_mps=speed)
    recipe = dataclasses.replace(recipe, forces=dataclasses.replace(recipe.forces, turbulence=turbulence))
    derived = derive(recipe)
    fields = operator_fields(derived.cells, 3, 1.0)
    results = []
    try:
        N.call("plume_use_fused_advection", 0)  # the two-pass kernels run with and without scratch, to the same floats
        for scratch in (True, False):
            grid = make_grid(derived, cell_m, recipe.domain.faces, 1.0, "cuda:0")
            for name, values in fields.items():
                getattr(grid, name).data.copy_(torch.from_numpy(values))
            stepper = Stepper(grid, recipe)
            state = stepper._state()
            if not scratch:
                state.advect_scratch = None
            N.call("plume_step", state, stepper._params(time_s, derived.dt_s), N.stream())
            results.append({name: host(getattr(grid, name).next) for name in fields})
    finally:
        N.call("plume_use_fused_advection", 1)
    for name in fields:
        assert np.isfinite(results[0][name]).all()
        assert_same(results[0][name], results[1][name], name)
