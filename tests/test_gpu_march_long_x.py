"""The velocity march along an x axis of more planes than a launch has blocks for at four planes a block."""

import pytest
import torch

from plume_b200 import _native as N

pytestmark = pytest.mark.gpu


def test_an_x_axis_of_twenty_million_planes(cuda_device):
    from support import cuda_grid

    info = cuda_grid((4, 1, 1)).info
    info.dims = N.c_int3(20_000_000, 1, 1)
    # constant velocities: every sample, and so every result, is the constant itself
    fields = [torch.full(shape, value, device="cuda:0") for shape, value in
              (((20_000_001, 1, 1), 0.75), ((20_000_000, 2, 1), -0.5), ((20_000_000, 1, 2), 0.25))]
    out = [torch.full_like(x, float("nan")) for x in fields]
    N.call("plume_maccormack_velocity", info, *(N.ptr(x) for x in fields), *(N.ptr(x) for x in out), 0.6, N.stream())
    for x, y in zip(fields, out):
        assert bool((x == y).all())
