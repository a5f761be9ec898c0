"""Faces that are no number, infinite or huge do not take the fused marches out of their arrays or rings: their traces run
from global memory with clamped indices, and the result differs from that of the field without them only nearby."""

import pytest
import torch

from plume_b200 import _native as N
from support import OPEN
from test_gpu_fused_advection import pair, scalars

pytestmark = pytest.mark.gpu

BROKEN = ((0, (12, 20, 35), float("nan")), (1, (5, 9, 68), -float("inf")), (2, (20, 30, 36), float("inf")),
          (2, (2, 0, 0), 3.0e38), (0, (3, 33, 5), -3.0e38))


def test_the_velocity_march(cuda_device):
    _, c = pair((24, 40, 70), OPEN)
    clean = [getattr(c, n).data.clone() for n in ("u", "v", "w")]
    broken = [x.clone() for x in clean]
    for component, cell, value in BROKEN:
        broken[component][cell] = value
    dt_over_cell = 0.7 / max(float(x.abs().max()) for x in clean)
    results = []
    for fields in (clean, broken):
        out = [torch.empty_like(x) for x in fields]
        N.call("plume_maccormack_velocity", c.info, *(N.ptr(x) for x in fields), *(N.ptr(x) for x in out), dt_over_cell,
               N.stream())
        results.append(out)
    torch.cuda.synchronize()
    centres = torch.tensor([cell for _, cell, _ in BROKEN], device="cuda:0")
    for a, b in zip(*results):
        where = (~(a == b)).nonzero()
        assert where.shape[0] > 0
        distance = (where[:, None, :] - centres[None]).abs().amax(dim=2).amin(dim=1)
        assert int(distance.max()) <= 5


def test_the_scalar_march(cuda_device):
    _, c = pair((24, 40, 70), OPEN)
    fields = [getattr(c, n).data for n in ("u", "v", "w")]
    dt = 0.7 * c.info.cell_m / max(float(x.abs().max()) for x in fields)
    clean = scalars(c, dt)
    for component, cell, value in BROKEN:
        fields[component][cell] = value
    broken = scalars(c, dt)
    centres = torch.tensor([cell for _, cell, _ in BROKEN])
    for a, b in zip(clean[:2], broken[:2]):
        where = (~(torch.from_numpy(a) == torch.from_numpy(b))).nonzero()
        distance = (where[:, None, :] - centres[None]).abs().amax(dim=2).amin(dim=1)
        assert where.shape[0] == 0 or int(distance.max()) <= 5
