"""The engine's memory plan (which activations a minibatch keeps) against a stand-in for the device: no GPU."""
from types import SimpleNamespace

import pytest
import torch

from mini_trainer_b200.models.config import get_preset
from mini_trainer_b200.parallel import engine as E


class Device:
    """A 183 GB device with ``free`` bytes free and an allocator that holds ``reserved`` of which ``allocated`` are in use."""

    def __init__(self, monkeypatch, free, reserved=8 << 30, allocated=6 << 30):
        self.free, self.reserved, self.allocated, self.asked, self.now = free, reserved, allocated, 0, 100.0
        total = 183 * 10 ** 9
        monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: SimpleNamespace(total_memory=total))
        monkeypatch.setattr(torch.cuda, "mem_get_info", self.query)
        monkeypatch.setattr(torch.cuda, "memory_reserved", lambda d=None: self.reserved)
        monkeypatch.setattr(torch.cuda, "memory_allocated", lambda d=None: self.allocated)
        monkeypatch.setattr(torch.cuda.memory, "memory_stats_as_nested_dict", lambda d=None: {
            "reserved_bytes": {"all": {"current": self.reserved}}, "allocated_bytes": {"all": {"current": self.allocated}}})
        monkeypatch.setattr("time.monotonic", lambda: self.now)

    def query(self, device=None):
        self.asked += 1
        return self.free, 183 * 10 ** 9


def planner(name, world=1):
    eng = object.__new__(E.ShardedEngine)
    cfg = get_preset(name)
    eng.cfg, eng.device, eng.param_dtype, eng.world, eng.symmetric = cfg, torch.device("cuda"), torch.bfloat16, world, False
    eng.blocks = [None] * cfg.num_hidden_layers
    eng.ops = SimpleNamespace(ce_chunk=8192)
    eng._pbufs = eng._gbufs = []
    eng.activation_budget_bytes, eng._oom_retries, eng._state_bytes, eng._free_reading = None, 0, 6 << 30, None
    return eng


def test_small_minibatch_on_a_full_device_recomputes(monkeypatch):
    """Another process has taken the device: what is free decides, however little the minibatch wants."""
    for name in ("nano-llama", "qwen2.5-1.5b"):
        eng, dev = planner(name), Device(monkeypatch, free=1 << 30, reserved=8 << 30, allocated=8 << 30)
        assert set(eng.plan_checkpointing(600)) <= {2, 3}
        dev.free = 150 << 30
        assert set(eng.plan_checkpointing(600)) == {0}


def test_free_memory_is_read_again(monkeypatch):
    eng, dev = planner("qwen2.5-1.5b"), Device(monkeypatch, free=150 << 30)
    for _ in range(5):
        assert set(eng.plan_checkpointing(600)) == {0}
        dev.now += 0.1
    assert dev.asked == 1                      # far from the limit: one reading serves a second
    dev.free = 1 << 30
    dev.now += 1.0
    assert set(eng.plan_checkpointing(600)) <= {2, 3} and dev.asked == 2
    dev.free = 150 << 30                       # near the limit every minibatch asks
    assert set(eng.plan_checkpointing(600)) == {0} and dev.asked == 3
    dev.reserved = dev.allocated = 152 << 30   # the allocator itself has taken what was free at the reading
    dev.free = 0
    assert set(eng.plan_checkpointing(600)) <= {2, 3} and dev.asked == 4
    dev.free, dev.reserved, dev.allocated = 150 << 30, 8 << 30, 6 << 30
    eng._oom_retries = 1                       # after an out-of-memory error too
    for asked in (5, 6):
        eng.plan_checkpointing(600)
        assert dev.asked == asked


def test_an_older_reading_changes_no_plan(monkeypatch):
    """Whatever is free, the levels planned from a reading of before are those of a reading of now."""
    for tokens in (600, 8000, 64000):
        for free in (0, 2, 5, 8, 12, 20, 40, 80, 150):
            eng, dev = planner("qwen2.5-1.5b"), Device(monkeypatch, free=free << 30)
            first = eng.plan_checkpointing(tokens)
            dev.now += 0.5
            again = eng.plan_checkpointing(tokens)
            eng._free_reading = None
            assert eng.plan_checkpointing(tokens) == first == again
