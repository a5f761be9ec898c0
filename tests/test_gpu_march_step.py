"""A velocity advection by a time step that is infinite or no number ends with an answer, and leaves the next one whole."""

import pytest
import torch

from support import OPEN
from test_gpu_fused_advection import pair
from test_gpu_velocity_march import march, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(24, 40, 70), (128, 128, 128)], ids=lambda c: "x".join(map(str, c)))
@pytest.mark.parametrize("step", [float("inf"), -float("inf"), float("nan")])
def test_a_step_that_is_not_finite(cuda_device, monkeypatch, cells, step):
    _, c = pair(cells, OPEN)
    fields = [getattr(c, name).data for name in ("u", "v", "w")]
    before = march(c.info, fields, 0.3)
    got = march(c.info, fields, step)
    monkeypatch.setenv("PLUME_MAC_ELEMENTS", "3")  # the form that forms every trace by itself
    assert all(same(a, b) for a, b in zip(got, march(c.info, fields, step)))
    monkeypatch.delenv("PLUME_MAC_ELEMENTS")
    assert all(bool(torch.isfinite(x).all()) and same(x, y) for x, y in zip(march(c.info, fields, 0.3), before))
