"""The velocity march's forms (one or two elements per thread, any segment length) give the floats of the march that
forms every trace by itself (the one long axes use), at the sizes where tiles have edges: rows and columns beyond a
tile's last, a single plane, traces that leave the staged planes in some cells, faces that are no number. That march
against the oracle is in test_gpu_fused_advection.py; a last case runs it where a coordinate needs it."""

import numpy as np
import pytest
import torch

from oracle import oracle as O
from plume_b200 import _native as N
from support import ALL_CLOSED, OPEN
from test_gpu_fused_advection import host, pair

pytestmark = pytest.mark.gpu

CASES = [((1, 1, 1), OPEN), ((2, 3, 2), ALL_CLOSED), ((4, 8, 32), OPEN), ((9, 17, 31), OPEN), ((5, 7, 33), ALL_CLOSED),
         ((70, 9, 34), OPEN), ((40, 70, 100), OPEN), ((21, 321, 307), OPEN), ((64, 180, 180), ALL_CLOSED), ((3, 831, 827), OPEN)]
IDS = ["x".join(map(str, cells)) for cells, _ in CASES]


def march(info, fields, dt_over_cell):
    out = [torch.full_like(x, float("nan")) for x in fields]
    N.call("plume_maccormack_velocity", info, *(N.ptr(x) for x in fields), *(N.ptr(x) for x in out), dt_over_cell, N.stream())
    torch.cuda.synchronize()
    return out


def same(a, b):
    return bool(((a == b) | (torch.isnan(a) & torch.isnan(b))).all())


@pytest.mark.parametrize("cells_moved", [0.5, 1.0, 6.0])
@pytest.mark.parametrize("cells,faces", CASES, ids=IDS)
def test_every_form_gives_the_same_floats(cuda_device, monkeypatch, cells, faces, cells_moved):
    _, c = pair(cells, faces)
    fields = [getattr(c, name).data for name in ("u", "v", "w")]
    dt_over_cell = cells_moved / max(float(x.abs().max()) for x in fields)
    monkeypatch.setenv("PLUME_MAC_ELEMENTS", "3")
    expected = march(c.info, fields, dt_over_cell)
    assert all(bool(torch.isfinite(x).all()) for x in expected)
    for elements, segments in ((1, 0), (2, 0), (1, 1), (2, cells[0]), (1, cells[0]), (2, 3)):
        monkeypatch.setenv("PLUME_MAC_ELEMENTS", str(elements))
        monkeypatch.setenv("PLUME_MAC_VELOCITY_SEGS", str(segments))
        for name, got, want in zip("uvw", march(c.info, fields, dt_over_cell), expected):
            assert same(got, want), f"{name}, {elements} elements, {segments} segments"


@pytest.mark.parametrize("elements", [1, 2])
def test_faces_that_are_no_number_spread_the_same(cuda_device, monkeypatch, elements):
    _, c = pair((24, 40, 70), OPEN)
    fields = [getattr(c, name).data.clone() for name in ("u", "v", "w")]
    dt_over_cell = 0.7 / max(float(x.abs().max()) for x in fields)
    fields[0][12, 20, 35] = float("nan")
    fields[1][5, 9, 68] = -float("inf")
    fields[2][20, 30, 35] = float("inf")
    fields[2][2, 0, 0] = 3.0e38
    monkeypatch.setenv("PLUME_MAC_ELEMENTS", "3")
    expected = march(c.info, fields, dt_over_cell)
    monkeypatch.setenv("PLUME_MAC_ELEMENTS", str(elements))
    assert all(same(a, b) for a, b in zip(march(c.info, fields, dt_over_cell), expected))


def test_an_axis_beyond_the_coordinate_split_matches_the_oracle(cuda_device):
    o, c = pair((1, 2, (1 << 22) + 70), OPEN)
    fields = [getattr(c, name).data for name in ("u", "v", "w")]
    dt = 0.5 * c.info.cell_m / max(float(x.abs().max()) for x in fields)
    velocity = tuple(f.data for f in o.velocity_fields())
    out = march(c.info, fields, dt / c.info.cell_m)
    # the coordinates themselves have a rounding of a quarter of a cell here, the same on both sides: traces that agree
    # to an ulp of the velocity land on the same one almost always
    for name, tensor in zip(("u", "v", "w"), out):
        O.advect_maccormack(getattr(o, name), velocity, o, dt)
        scale = float(np.abs(getattr(o, name).next).max())
        off = np.abs(host(tensor).astype(np.float64) - getattr(o, name).next) / scale
        assert float(np.mean(off > 1e-5)) < 1e-3, name
