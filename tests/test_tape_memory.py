"""Where FlowFit's tape goes when the allocator's idle memory looks large enough for it and is not: the records are cut
back to what the driver's free memory allows, and a pass that runs out of memory is formed again within that. The
substeps are stand-ins on the host; the device's memory counters are the test's."""

import gc
import weakref
from types import SimpleNamespace

import pytest
import torch

from plume_b200.adjoint import FlowFit

SUBSTEPS, EVERY, RECORD = 16, 4, 100


class Record(dict):
    """A substep's record that can be watched."""


class Fit(FlowFit):
    def __init__(self, tape_bytes=None):
        field = SimpleNamespace(data=torch.zeros(2, 2, 2))
        self.grid = SimpleNamespace(smoke=field, temperature=field, pressure=torch.zeros(2, 2, 2), velocity_fields=lambda: [field] * 3)
        self.adjoint_grid = SimpleNamespace(pressure=torch.zeros(2, 2, 2))
        self.recipe = SimpleNamespace(domain=SimpleNamespace(ambient_k=1.0))
        self.device, self.substeps, self.every, self.tape_bytes = "cpu", SUBSTEPS, EVERY, tape_bytes
        self.confined, self.source_shape = False, (2, 2, 2)
        self.live, self.recorded, self.reversed, self.kept, self.out_of_memory_at = [], [], [], None, []

    def record_bytes(self):
        return RECORD

    def _state(self):
        return len(self.recorded)

    def _load(self, state):
        pass

    def _substep(self, n, source, record=False):
        rec = Record(substep=n)
        if record:
            self.recorded.append(n)
            self.live.append(weakref.ref(rec))
        return rec

    def _thickness(self, target):
        gc.collect()
        self.kept = sorted(r()["substep"] for r in self.live if r() is not None)
        return 1.5, torch.zeros(1), torch.zeros(2, 2, 2)

    def _substep_adjoint(self, n, rec, a_smoke, a_heat, a_vel, grads, grad_source):
        if n in self.out_of_memory_at:
            self.out_of_memory_at.remove(n)
            raise torch.OutOfMemoryError("no memory for the reverse substep")
        assert rec["substep"] == n
        self.reversed.append(n)
        return a_smoke, a_heat, a_vel


@pytest.fixture
def memory(monkeypatch):
    m = SimpleNamespace(reserved=10_000, allocated=10_000 - SUBSTEPS * RECORD, free=0, asked=0)

    def mem_get_info(*_):
        m.asked += 1
        return m.free, 1 << 40

    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda *_: m.reserved)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda *_: m.allocated)
    monkeypatch.setattr(torch.cuda, "mem_get_info", mem_get_info)
    return m


def run(fit):
    return fit.loss_and_grad(torch.zeros(2, 2, 2), torch.zeros(1))


BACKWARD = list(reversed(range(SUBSTEPS)))


def test_idle_memory_that_serves_holds_every_record(memory):
    fit = Fit()
    assert run(fit)[0] == 1.5
    assert fit.kept == list(range(SUBSTEPS)) and fit.recorded == fit.kept and fit.reversed == BACKWARD and memory.asked == 0


@pytest.mark.parametrize("free,kept_from", [(16 * RECORD, 8), (9 * RECORD, 12), (7 * RECORD, 16), (0, 16), (40 * RECORD, 0)])
@pytest.mark.parametrize("grows_at", [0, 5, 15])
def test_idle_memory_that_does_not_serve_leaves_the_drivers_budget(memory, free, kept_from, grows_at):
    memory.free = free

    class Fragmented(Fit):
        def _substep(self, n, source, record=False):
            if record and n == grows_at:
                memory.reserved += RECORD  # the allocator had to take more for this record
            return super()._substep(n, source, record)

    fit = Fragmented()
    assert run(fit)[0] == 1.5
    assert fit.kept == list(range(kept_from, SUBSTEPS)) and memory.asked == 1
    assert fit.reversed == BACKWARD
    recomputed = [n for first in reversed(range(0, kept_from, EVERY)) for n in range(first, first + EVERY)]
    in_forward = [n for n in range(SUBSTEPS) if n <= grows_at or n >= kept_from]
    assert fit.recorded == in_forward + recomputed


@pytest.mark.parametrize("at", [15, 3])
def test_out_of_memory_beside_a_tape_in_idle_memory(memory, at):
    memory.free = 8 * RECORD
    fit = Fit()
    fit.out_of_memory_at = [at]
    assert run(fit)[0] == 1.5
    assert fit.kept == [12, 13, 14, 15] and memory.asked == 1
    assert fit.reversed[-SUBSTEPS:] == BACKWARD


def test_out_of_memory_within_a_budget_is_the_callers(memory):
    memory.allocated, memory.free = memory.reserved, 64 * RECORD  # nothing idle: the driver's budget from the start
    for fit in (Fit(), Fit(tape_bytes=64 * RECORD)):
        fit.out_of_memory_at = [7]
        with pytest.raises(torch.OutOfMemoryError):
            run(fit)
