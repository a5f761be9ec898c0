"""The render kernels where their tiles, runs and maps end: axes of one cell up to beyond a warp, marches along and against
every axis, grids with no room for a run of unclamped samples, blurs wider than the grid, an extent beyond the coordinate
split. Light against the oracle, and bit for bit with and without the brick map; gradients bit for bit."""

import numpy as np
import pytest
import torch

from oracle import oracle as O
from plume_b200 import _native as N
from plume_b200.recipe.schema import NORMAL_LAYOUT, RenderSettings
from plume_b200.render.camera import make_camera, make_domain_view
from plume_b200.render.light_volume import LightVolume
from plume_b200.render.normal_field import NormalField
from support import assert_same, host
from test_gpu_render import read_by_march

pytestmark = pytest.mark.gpu

CELLS = [(1, 1, 1), (2, 3, 2), (5, 4, 33), (9, 8, 31), (33, 1, 6), (40, 36, 70)]
DIRECTIONS = [(0, 1, 0), (0, -1, 0), (1, 0, 0), (0, 0, -1), (-1e-13, 1, 1e-13), (-0.6, 0.7, -0.4), (0.5, -0.8, 0.3)]


def sparse(cells, seed=5):
    g = np.random.default_rng(seed)
    smoke = g.uniform(0.0, 2.0, cells).astype(np.float32)
    keep = g.uniform(0.0, 1.0, tuple((n + 3) // 4 for n in cells)) < 0.15
    for axis, n in enumerate(cells):
        keep = np.take(np.repeat(keep, 4, axis), np.arange(n), axis)
    smoke[~keep] = 0.0
    smoke[tuple(n // 2 for n in cells)] = 1.0
    return smoke


@pytest.mark.parametrize("direction", DIRECTIONS)
@pytest.mark.parametrize("cells", CELLS, ids=lambda c: "x".join(map(str, c)))
def test_light(cuda_device, cells, direction):
    smoke = sparse(cells)
    toward = np.array(direction) / np.linalg.norm(direction)
    field = torch.from_numpy(smoke).to("cuda:0")
    volume = LightVolume(cells, toward, 1.0, "cuda:0")
    light = host(volume.compute(field, 0.05).clone())
    read_only = host(volume.compute(field, 0.05, march_cells=True).clone())
    without = torch.empty_like(field)
    N.call("plume_light_volume", N.shape3(field), N.ptr(field), 0, N.f3(volume.toward_light), 0.05, 1.0, N.ptr(without),
           None, N.stream())
    assert_same(light, host(without), "without the brick map")
    read = read_by_march(smoke)
    assert_same(read_only[read], light[read], "read cells")
    assert np.all(read_only[~read] == 1.0)
    # sample points round by 2^-24 of their coordinates (below 70) twice on either side, smoke changes by at most 2 a
    # cell, a march has 160 half-cell samples: 160 * 0.5 * 2 * 4 * 70 * 2^-24 * 0.05 in the exponent at the most
    expected = O.light_volume(smoke, toward, 0.05, 1.0)
    assert float(np.abs(light / expected - 1.0).max()) < 1.4e-4


def test_light_beyond_the_coordinate_split(cuda_device):
    """The march of an extent of 2^22 cells, across its short axis: the light of a part of it alone, bit for bit."""
    smoke = torch.from_numpy(sparse((1, 6, 4096))).to("cuda:0").repeat(1, 1, 1025).contiguous()
    lights = [host(LightVolume(tuple(x.shape), (0.0, 1.0, 0.0), 1.0, "cuda:0").compute(x, 0.05))
              for x in (smoke, smoke[..., :4096].contiguous())]
    assert_same(lights[0][..., :4096], lights[1], "light")
    assert_same(lights[0][..., -4096:], lights[1], "light")


@pytest.mark.parametrize("blur_cells", [0.0, 0.3, 0.6, 1.5, 6.0])  # 1, 3, 5, 11 and 37 taps
@pytest.mark.parametrize("cells", CELLS, ids=lambda c: "x".join(map(str, c)))
def test_gradient(cuda_device, cells, blur_cells):
    smoke = sparse(cells)
    gradient = NormalField(cells, blur_cells, "cuda:0").compute(torch.from_numpy(smoke).to("cuda:0"))
    renderer = O.FrameRenderer(make_domain_view(make_camera(0, 0), (0, 0, 0), (1, 1, 1), 0.05, 2.0),
                               RenderSettings(normal_blur_cells=blur_cells), cells, NORMAL_LAYOUT)
    renderer.prepare(smoke, 0.05)
    assert_same(host(gradient), renderer.gradient, "gradient")


def test_light_of_a_long_second_axis(cuda_device):
    """More rows than a launch has blocks along its second axis."""
    smoke = torch.from_numpy(sparse((1, 2048, 3))).to("cuda:0").repeat(1, 300, 1).contiguous()
    light = host(LightVolume(tuple(smoke.shape), (0.0, 0.0, 1.0), 1.0, "cuda:0").compute(smoke, 0.05, march_cells=True))
    part = smoke[:, :4096].contiguous()
    expected = host(LightVolume(tuple(part.shape), (0.0, 0.0, 1.0), 1.0, "cuda:0").compute(part, 0.05, march_cells=True))
    assert_same(light[:, :4095], expected[:, :4095], "first rows")  # the part's last row has no neighbour beyond it
    assert_same(light[:, -2048:-1], expected[:, 2048:4095], "last rows")
