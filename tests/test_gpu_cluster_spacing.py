"""Cell sizes whose square leaves the range of the cluster solve's reciprocals: such levels run by launches of their own,
and the pressure is the oracle's bit for bit as at any other size."""

import numpy as np
import pytest

from oracle import oracle as O
from support import ALL_CLOSED, OPEN, assert_same, cuda_grid, host, load_state, oracle_grid

pytestmark = pytest.mark.gpu


def pair(cells, faces, cell_m):
    o, c = oracle_grid(cells, cell_m, faces), cuda_grid(cells, cell_m, faces)
    rng = np.random.default_rng(7)
    load_state(o, c, {name: rng.uniform(-1, 1, getattr(o, name).data.shape).astype(np.float32) for name in ("u", "v", "w")})
    return o, c


@pytest.mark.parametrize("cell_m", [1e-20, 1.2e-19, 1e19])
@pytest.mark.parametrize("cells,faces", [((12, 10, 14), OPEN), ((17, 9, 11), ALL_CLOSED), ((48, 40, 36), OPEN)])
def test_gauss_seidel(cuda_device, cells, faces, cell_m):
    from plume_b200.sim.pressure import GaussSeidel, project

    o, c = pair(cells, faces, cell_m)
    O.project(o, O.GaussSeidel(5))
    project(c, GaussSeidel(5))
    assert_same(host(c.pressure), o.pressure, "pressure")


@pytest.mark.parametrize("cell_m", [1e-20, 1.2e-19])
@pytest.mark.parametrize("cells,faces", [((12, 10, 14), OPEN), ((17, 9, 11), OPEN), ((48, 40, 36), OPEN)])
def test_multigrid(cuda_device, cells, faces, cell_m):
    from plume_b200.sim.multigrid import Multigrid
    from plume_b200.sim.pressure import project

    o, c = pair(cells, faces, cell_m)
    O.project(o, O.Multigrid(o, 2, 2))
    project(c, Multigrid(c, 2, 2))
    assert_same(host(c.pressure), o.pressure, "pressure")
