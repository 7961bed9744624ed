"""The training loop asks the kernels' status word once per step and stops on what it says."""
import json
import os

import pytest

from mini_trainer_b200.data.sampler import get_data_loader
from mini_trainer_b200.data.synthetic import CONFIG_DATA, synthetic_dataset
from mini_trainer_b200.models.config import get_preset
from mini_trainer_b200.ops import get_ops
from mini_trainer_b200.parallel.comm import make_comm
from mini_trainer_b200.parallel.engine import OptimConfig, ShardedEngine
from mini_trainer_b200.trainer import setup_training_components, train


def test_training_stops_when_a_kernel_gave_up(tmp_path, monkeypatch):
    for k in ("RANK", "WORLD_SIZE", "LOCAL_RANK"):
        monkeypatch.delenv(k, raising=False)
    spec, vocab, max_tokens, _ = CONFIG_DATA["tiny-qwen2"]
    cfg = get_preset("nano-llama")
    ops, asked = get_ops("cpu"), []

    def check_status():
        asked.append(1)
        if len(asked) == 2:
            raise RuntimeError("a device-side bounded wait expired (status code 70)")
    ops.check_status = check_status
    eng = ShardedEngine(cfg, "cpu", ops, comm=make_comm("auto"), optim=OptimConfig())
    eng.init_random(seed=1)
    model, opt, sched = setup_training_components(eng, learning_rate=1e-4, num_warmup_steps=2)
    ds = synthetic_dataset(64, spec, min(vocab, cfg.vocab_size), seed=1)
    loader = get_data_loader(dataset=ds, batch_size=2, max_tokens_per_gpu=max_tokens, seed=1, rank=0, world_size=1, prefetch=0)
    with pytest.raises(RuntimeError, match="status code 70"):
        train(model, opt, sched, loader, str(tmp_path), min_samples_per_checkpoint=1000, max_steps=5, log_echo=False)
    assert len(asked) == 2
    steps = [json.loads(l) for l in open(os.path.join(tmp_path, "training_metrics_0.jsonl"))] if os.path.exists(os.path.join(tmp_path, "training_metrics_0.jsonl")) else []
    assert all(s["step"] < 2 for s in steps)      # the step that is not to be used is not reported
