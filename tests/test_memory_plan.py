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


@pytest.mark.parametrize("tokens", [1, 200, 4096, 64000])
def test_plan_counts_the_rows_that_experts_are_padded_to(tokens):
    """A mixture-of-experts block keeps, and works on, row buffers with each expert's rows padded to 128."""
    from dataclasses import replace
    from mini_trainer_b200.cli.plan import memory_plan
    cfg = replace(get_preset("mixtral-8x7b"), num_local_experts=128, num_experts_per_tok=8, hidden_size=2048, intermediate_size=768, moe_intermediate_size=768)
    f, h, es = cfg.expert_intermediate_size, cfg.hidden_size, 2
    rows = -(-(tokens * 8 + 128 * 127) // 128) * 128      # what the slabs are allocated with
    lvl1, lvl0 = E.kept_bytes(cfg, tokens)
    assert lvl0 - lvl1 >= rows * 2 * f * es + tokens * (h + cfg.qkv_size) * es
    # backward: gathered output gradient, gradient of the activation and of gate/up; then that of gate/up, of the gathered inputs
    # and the gathered inputs themselves; beside the layer's input, output gradient and input gradient
    assert E.working_set_bytes(cfg, tokens) >= rows * es * max(h + 3 * f, 2 * h + 2 * f) + 3 * tokens * h * es + (128 << 20)
    eng = planner("mixtral-8x7b")
    eng.cfg = cfg
    assert eng._kept_bytes(tokens) == (lvl1, lvl0)
    plan = memory_plan(cfg, 8, tokens)
    assert plan["per_block_gb"]["keep_every_gemm_output"] == round(lvl0 / 2 ** 30, 2)


def test_plan_of_a_dense_block_is_what_it_was():
    cfg, t = get_preset("qwen2.5-1.5b"), 6000
    lvl1, lvl0 = E.kept_bytes(cfg, t)
    assert lvl1 == t * (cfg.q_size * 2 + cfg.num_attention_heads * 4)
    assert lvl0 == lvl1 + t * ((cfg.hidden_size + cfg.qkv_size + 2 * cfg.intermediate_size) * 2 + 8)
    assert E.working_set_bytes(cfg, t) == t * 2 * (7 * cfg.hidden_size + cfg.qkv_size + 6 * cfg.intermediate_size) + (128 << 20)
