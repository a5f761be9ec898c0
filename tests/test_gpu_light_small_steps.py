"""Light marches that hardly move along an axis: their samples round to the last cell's own coordinate, whose upper
neighbour is outside the grid. Light against the oracle, bit for bit with and without the brick map, and untouched by
what lies beyond the last column in memory."""

import numpy as np
import pytest
import torch

from oracle import oracle as O
from plume_b200 import _native as N
from plume_b200.render.light_volume import LightVolume
from support import assert_same, host
from test_gpu_render_edges import sparse

pytestmark = pytest.mark.gpu

CELLS = [(2, 9, 3), (40, 36, 70), (130, 12, 129)]
DIRECTIONS = [(-1e-7, 1, 0), (0, 1, -1e-6), (-1e-9, 0.7, -1e-5), (-1e-4, 1, -3e-3), (1, -1e-6, -2e-8), (-1e-12, -1e-5, 1)]


@pytest.mark.parametrize("direction", DIRECTIONS)
@pytest.mark.parametrize("cells", CELLS, ids=lambda c: "x".join(map(str, c)))
def test_light(cuda_device, cells, direction):
    smoke = sparse(cells)
    volume = LightVolume(cells, direction, 1.0, "cuda:0")
    field = torch.from_numpy(smoke).to("cuda:0")
    light = host(volume.compute(field, 0.05).clone())
    without = torch.empty_like(field)
    N.call("plume_light_volume", N.shape3(field), N.ptr(field), 0, N.f3(volume.toward_light), 0.05, 1.0, N.ptr(without),
           None, N.stream())
    assert_same(light, host(without), "without the brick map")
    # as for the other edges: sample points round by 2^-24 of their coordinates (up to 130) twice on either side, smoke
    # changes by at most 2 a cell, a march has up to 2 * 130 half-cell samples
    expected = O.light_volume(smoke, np.array(direction) / np.linalg.norm(direction), 0.05, 1.0)
    assert float(np.abs(light / expected - 1.0).max()) < 260 * 0.5 * 2 * 4 * 130 * 2**-24 * 0.05


@pytest.mark.parametrize("direction", [(0, 1, -1e-6), (0, -1, -1e-7), (1, 0, -3e-6)])
def test_the_next_rows_first_column_stays_out_of_the_last_columns_light(cuda_device, direction):
    cells = (24, 20, 70)
    smoke = np.full(cells, 0.5, dtype=np.float32)
    smoke[:, :, 0] = np.inf
    light = host(LightVolume(cells, direction, 1.0, "cuda:0").compute(torch.from_numpy(smoke).to("cuda:0"), 0.05))
    expected = O.light_volume(smoke, np.array(direction) / np.linalg.norm(direction), 0.05, 1.0)
    assert np.isfinite(light[:, :, 2:]).all()
    # constant smoke: the column is a sum of up to 48 equal terms of at most 0.25, each side rounding each by 2^-24 of it
    assert float(np.abs(light[:, :, 2:] / expected[:, :, 2:] - 1.0).max()) < 48 * 2 * 2**-24 * 12 * 0.05 + 4 * 2**-24
