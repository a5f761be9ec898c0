"""FlowFit asks the driver for the free memory only when its tape does not fit what the caching allocator holds idle."""

import pytest

from plume_b200.workloads import plain_step_recipe

pytestmark = pytest.mark.gpu


def test_the_driver_is_asked_only_for_memory_not_at_hand(cuda_device, monkeypatch):
    import torch

    from plume_b200.adjoint import FlowFit

    fit = FlowFit(plain_step_recipe((16, 20, 16), cycles=2), (4, 4, 4), (6, 2, 6), 3, "cuda:0", checkpoint_every=2)
    asked = []
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: asked.append(a) or (0, 1))
    need = fit.substeps * fit.record_bytes()
    torch.cuda.empty_cache()
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda *a: 5 * need)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda *a: 4 * need + 1)
    assert fit._taped_from() == fit.substeps and len(asked) == 1  # idle is too little, and the driver has nothing free
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda *a: 4 * need)
    assert fit._taped_from() == 0 and len(asked) == 1
