"""Smoke at one temperature that is also where glow starts: the blends of a value such as 300.1 K are off by an ulp at
some samples (the oracle's heat is above 0 in one pixel of thirteen here), and the march with its brick map takes them as it does without one."""

import pytest
import torch

from plume_b200 import _native as N
from plume_b200.recipe.schema import NORMAL_LAYOUT, SHADE_LAYOUT, RenderSettings
from plume_b200.render.camera import make_camera, make_domain_view
from plume_b200.render.frame_renderer import FrameRenderer
from support import OPEN, cuda_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [SHADE_LAYOUT, NORMAL_LAYOUT])
@pytest.mark.parametrize("ambient", [300.1, 1.0])
def test_smoke_at_the_temperature_where_glow_starts(cuda_device, channels, ambient):
    cells = (24, 32, 20)
    c = cuda_grid(cells, 0.05, OPEN, ambient)
    c.smoke.data.fill_(0.01)
    c.temperature.data.fill_(ambient)
    size = tuple(n * 0.05 for n in cells)
    view = make_domain_view(make_camera(20.0, 30.0), (-size[0] / 2, 0.0, -size[2] / 2), size, 0.05, 2.0)
    renderer = FrameRenderer(view, RenderSettings(glow_start_k=ambient), cells, channels, "cuda:0")
    renderer.prepare(c.smoke.data, c.info.cell_m)
    image, without = torch.zeros_like(renderer.image), torch.zeros_like(renderer.image)
    renderer.march(c.smoke.data, c.temperature.data, c.info, renderer.view_params, image)
    N.call("plume_raymarch", c.info, N.ptr(c.smoke.data), N.ptr(c.temperature.data), 0, N.ptr(renderer.gradient),
           N.c_int3(*renderer.gradient.shape[:3]), N.ptr(renderer.light), N.shape3(renderer.light), renderer.view_params,
           renderer.look_params, N.ptr(without), without.shape[0], without.shape[1], None, N.stream())
    assert torch.equal(image, without)
    assert (float(without[..., 0].max()) > 0.0) == (ambient == 300.1)
