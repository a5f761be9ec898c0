"""The divergence and the pressure gradient where their planes end: axes of one and two cells, planes and rows beyond a
block's last, open and closed walls, spacings with and without a division: the oracle's floats."""

import numpy as np
import pytest
import torch

from oracle import oracle as O
from plume_b200 import _native as N
from support import ALL_CLOSED, OPEN, assert_same, host
from test_gpu_fused_advection import pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell_m", [1.0 / 64.0, 0.05])
@pytest.mark.parametrize("faces", [OPEN, ALL_CLOSED], ids=["open", "closed"])
@pytest.mark.parametrize("cells", [(1, 1, 1), (2, 1, 3), (1, 2, 33), (5, 9, 33), (9, 8, 70), (3, 2, 32)],
                         ids=lambda c: "x".join(map(str, c)))
def test_divergence_and_gradient(cuda_device, cells, faces, cell_m):
    o, c = pair(cells, faces, cell_m=cell_m)
    velocity = [getattr(o, name).data.copy() for name in ("u", "v", "w")]
    q = np.random.default_rng(3).standard_normal(cells).astype(np.float32)
    device = [getattr(c, name).data for name in ("u", "v", "w")]
    divergence = torch.empty(cells, dtype=torch.float32, device="cuda:0")
    N.call("plume_divergence", c.info, *(N.ptr(x) for x in device), N.ptr(divergence), N.stream())
    h = np.float32(cell_m)
    expected = sum_in_order([np.diff(x, axis=axis) for axis, x in enumerate(velocity)]) / h
    assert_same(host(divergence), expected, "divergence")
    N.call("plume_subtract_gradient", c.info, *(N.ptr(x) for x in device), N.ptr(torch.from_numpy(q).to("cuda:0")), N.stream())
    for axis, name in enumerate("uvw"):
        padded = np.pad(q, [(1, 1) if a == axis else (0, 0) for a in range(3)])
        step = np.diff(padded, axis=axis) / h
        edge = [slice(None)] * 3
        for side, is_open in ((0, o.info.open_lo[axis]), (-1, o.info.open_hi[axis])):
            if not is_open:
                edge[axis] = side
                step[tuple(edge)] = 0.0
        assert_same(host(device[axis]), velocity[axis] - step, name)


def sum_in_order(parts):
    return (parts[0] + parts[1]) + parts[2]
