"""The work a training run has this framework do, as cases that can be timed and checked.

Six kinds of call, all through the entry points a program uses:

* ``step``       a whole optimizer step (``ShardedEngine.train_step``) of a small model
* ``block``      forward and backward of one dense decoder block (``decoder.block_forward`` / ``block_backward``)
* ``moe``        forward and backward of the routed experts (``moe.moe_forward`` / ``moe_backward``)
* ``attention``  varlen causal attention, forward and backward (``ops.attention`` / ``attention_bwd``)
* ``head``       final norm, LM head and cross-entropy with their gradients (``decoder.head_forward_backward``)
* ``optimizer``  gradient accumulation, norm and AdamW over one rank's shard (``accumulate`` / ``sumsq`` / ``adamw_step``)

``listed()`` holds one case per use, ``draw(rng)`` another one of the same ranges. Weights, activations and gradients
are bf16 as in training; sample lengths follow from the case, all values from the seed.
"""
from __future__ import annotations

import math
import random

import torch

from mini_trainer_b200.data.sampler import mb_collate_fn
from mini_trainer_b200.models import decoder as D
from mini_trainer_b200.models import layout as L
from mini_trainer_b200.models import moe as M
from mini_trainer_b200.models.config import ModelConfig
from mini_trainer_b200.ops import get_ops
from mini_trainer_b200.parallel.engine import OptimConfig, ShardedEngine

DEV = "cuda"
EPS = 1e-5
THETA = 5e5
LR = 5e-6

_OPS = None


def _ops():
    """The kernel backend: a program makes one and uses it for everything."""
    global _OPS
    if _OPS is None:
        _OPS = get_ops(torch.device(DEV, torch.cuda.current_device()))
    return _OPS


# ------------------------------------------------------------------------------------------ cases
def listed() -> list:
    return [
        # the smallest complete call: a first step on a few short samples, as the smoke run does it
        {"name": "step_small", "kind": "step", "vocab": 4096, "hidden": 512, "inter": 1536, "layers": 2, "hq": 4, "hkv": 1,
         "d": 128, "bias": False, "tied": False, "tokens": 640, "samples": 3},
        # the tiny benchmark model at its full token budget: head_dim 64, q/k/v bias, tied embeddings
        {"name": "step_tiny", "kind": "step", "vocab": 32000, "hidden": 256, "inter": 688, "layers": 2, "hq": 4, "hkv": 2,
         "d": 64, "bias": True, "tied": True, "tokens": 4096, "samples": 12},
        # a block of the 1.5B benchmark model on a minibatch that the packer could not fill
        {"name": "block_1b5", "kind": "block", "family": "qwen2", "hidden": 1536, "inter": 8960, "hq": 12, "hkv": 2, "d": 128,
         "tokens": 5987, "samples": 4, "recompute": False},
        # a block of the headline 8B model on a quarter of its token budget: the largest case
        {"name": "block_8b", "kind": "block", "family": "llama", "hidden": 4096, "inter": 14336, "hq": 32, "hkv": 8, "d": 128,
         "tokens": 16384, "samples": 6, "recompute": False},
        # per-head q/k norm, recomputed in backward as when activations do not fit
        {"name": "block_qknorm", "kind": "block", "family": "qwen3", "hidden": 2048, "inter": 6144, "hq": 16, "hkv": 8, "d": 128,
         "tokens": 4099, "samples": 7, "recompute": True},
        # LayerNorm, biases everywhere and an MLP without a gate
        {"name": "block_layernorm", "kind": "block", "family": "starcoder2", "hidden": 3072, "inter": 12288, "hq": 24, "hkv": 2,
         "d": 128, "tokens": 7001, "samples": 5, "recompute": False},
        # the experts of the 8-expert benchmark model: few large slabs
        {"name": "moe_8x", "kind": "moe", "hidden": 4096, "inter": 14336, "experts": 8, "chosen": 2, "tokens": 4096},
        # many small experts, several per token: many short, uneven slabs
        {"name": "moe_many", "kind": "moe", "hidden": 2048, "inter": 1024, "experts": 64, "chosen": 8, "tokens": 2051},
        # one long document: attention is most of the step
        {"name": "attention_long", "kind": "attention", "hq": 32, "hkv": 8, "d": 128, "tokens": 16384, "samples": 1},
        # many short chat samples, head_dim 64
        {"name": "attention_short", "kind": "attention", "hq": 16, "hkv": 4, "d": 64, "tokens": 12345, "samples": 41},
        # the 151 936-token vocabulary on a minibatch with a masked prompt in every sample
        {"name": "head_1b5", "kind": "head", "hidden": 1536, "vocab": 151936, "tokens": 6000, "counted": 0.62},
        # one rank's state of one 8B block, fp32 moments
        {"name": "optimizer_8b", "kind": "optimizer", "numel": 218112000, "fp32_moments": True},
    ]


def _log(rng, lo: float, hi: float, step: int = 1) -> int:
    return max(step, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step)


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["step", "block", "block", "block", "moe", "moe", "attention", "attention", "head", "optimizer"])
    if kind == "step":
        d = rng.choice([64, 128])
        hkv = rng.choice([1, 2])
        hq = hkv * rng.choice([1, 2, 4])
        tokens = _log(rng, 100, 5000)
        return {"kind": kind, "vocab": _log(rng, 2048, 32000, 8), "hidden": _log(rng, 256, 1024, 8), "inter": _log(rng, 512, 3072, 8),
                "layers": rng.choice([2, 3]), "hq": hq, "hkv": hkv, "d": d, "bias": rng.random() < 0.5, "tied": rng.random() < 0.5,
                "tokens": tokens, "samples": min(rng.randint(1, 13), tokens // 20)}
    if kind == "block":
        family = rng.choice(["llama", "qwen2", "qwen3", "starcoder2"])
        d = 128 if family == "qwen3" else rng.choice([64, 128, 128])
        hkv = rng.choice([2, 4, 8])
        hq = hkv * rng.choice([1, 2, 3, 4])
        hidden = _log(rng, 512, 4096, 8)
        inter = _log(rng, 2 * hidden, 4 * hidden, 8)
        most = 12e12 / (6 * hidden * (3 * inter + 2 * d * (hq + hkv)))
        tokens = _log(rng, 500, min(16384, most))
        return {"kind": kind, "family": family, "hidden": hidden, "inter": inter, "hq": hq, "hkv": hkv, "d": d, "tokens": tokens,
                "samples": rng.randint(1, 12), "recompute": rng.random() < 0.35}
    if kind == "moe":
        experts = rng.choice([4, 8, 16, 32, 64])
        chosen = min(rng.choice([1, 2, 4, 8]), experts // 2)
        hidden = _log(rng, 512, 4096, 8)
        inter = _log(rng, 512, min(14336, 1.5e9 / (3 * hidden * experts)), 8)
        return {"kind": kind, "hidden": hidden, "inter": inter, "experts": experts, "chosen": chosen, "tokens": _log(rng, 300, 4096)}
    if kind == "attention":
        d = rng.choice([64, 128])
        hkv = rng.choice([1, 2, 4, 8])
        samples = _log(rng, 1, 50)
        return {"kind": kind, "hq": hkv * rng.choice([1, 2, 4]), "hkv": hkv, "d": d, "tokens": _log(rng, max(400, 40 * samples), 16384),
                "samples": samples}
    if kind == "head":
        hidden = _log(rng, 512, 4096, 8)
        vocab = _log(rng, 32000, 152064, 8)
        return {"kind": kind, "hidden": hidden, "vocab": vocab, "tokens": _log(rng, 400, min(9000, 9e12 / (6 * hidden * vocab))),
                "counted": round(rng.uniform(0.4, 1.0), 2)}
    return {"kind": kind, "numel": _log(rng, 1e6, 2.1e8, 128), "fp32_moments": rng.random() < 0.6}


# ------------------------------------------------------------------------------------------ inputs
def _lengths(case: dict) -> list:
    """Lengths of the packed samples: lognormal, as chat data is, and fixed by the case."""
    n, t = case["samples"], case["tokens"]
    r = random.Random(1000003 * t + n)
    w = [r.lognormvariate(0.0, 0.8) for _ in range(n)]
    lens = [max(1, int(x / sum(w) * (t - n))) for x in w]
    lens[0] += t - sum(lens)
    return lens


def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(1_000_003 * (seed + 1))


def _bf(gen, *shape, scale=1.0, shift=0.0) -> torch.Tensor:
    return torch.randn(*shape, generator=gen, device=DEV, dtype=torch.float32).mul_(scale).add_(shift).bfloat16()


def _config(case: dict) -> ModelConfig:
    kind = case["kind"]
    family = case.get("family", "qwen2" if case.get("bias") else "llama")
    kw = dict(model_type=family, vocab_size=case.get("vocab", 1024), hidden_size=case["hidden"],
              intermediate_size=case.get("inter", 8 * 128), num_hidden_layers=case.get("layers", 1),
              num_attention_heads=case.get("hq", 1), num_key_value_heads=case.get("hkv", 1), head_dim=case.get("d", 128),
              rope_theta=THETA, rms_norm_eps=EPS, tie_word_embeddings=case.get("tied", False))
    if family == "qwen2":
        kw.update(attention_bias=True)
    if family == "qwen3":
        kw.update(qk_norm=True)
    if family == "starcoder2":
        kw.update(norm_type="layernorm", mlp_gated=False, attention_bias=True, mlp_bias=True, hidden_act="gelu_pytorch_tanh")
    if kind == "moe":
        kw.update(model_type="mixtral", num_local_experts=case["experts"], num_experts_per_tok=case["chosen"])
    return ModelConfig(**kw)


def _weights(flat: torch.Tensor, views: dict, gen) -> None:
    """Trained-looking values: matrices at the usual initial scale, norms near one, small biases."""
    flat.normal_(0.0, 0.02, generator=gen)
    for name, v in views.items():
        if v.dim() == 1 and not name.startswith("b"):
            v.mul_(5.0).add_(1.0)


def _host_batch(case: dict, seed: int) -> dict:
    g = torch.Generator().manual_seed(seed)
    samples = []
    for n in _lengths(case):
        ids = torch.randint(0, case.get("vocab", 1024), (n,), generator=g)
        labels = ids.clone()
        masked = n // 4
        labels[:masked] = -100
        samples.append({"input_ids": ids, "labels": labels, "len": n, "num_loss_counted_tokens": n - masked})
    return mb_collate_fn(samples, sum(s["num_loss_counted_tokens"] for s in samples))


def _block_inputs(case: dict, seed: int) -> dict:
    cfg, gen = _config(case), _gen(seed)
    lay = L.GroupLayout("block0", L.block_entries(cfg), 1)
    flat = torch.empty(lay.padded_numel, dtype=torch.bfloat16, device=DEV)
    views = lay.views(flat)
    _weights(flat, views, gen)
    t, h = case["tokens"], case["hidden"]
    return {"cfg": cfg, "layout": lay, "p": views, "x": _bf(gen, t, h), "dout": _bf(gen, t, h, scale=0.01)}


def _moe_inputs(case: dict, seed: int) -> dict:
    cfg, gen = _config(case), _gen(seed)
    h, f, e, k, t = case["hidden"], case["inter"], case["experts"], case["chosen"], case["tokens"]
    entries = [("router", (e, h))]
    for x in range(e):
        entries += [(f"wgu{x}", (2 * f, h)), (f"wd{x}", (h, f))]
    lay = L.GroupLayout("experts", entries, 1)
    flat = torch.empty(lay.padded_numel, dtype=torch.bfloat16, device=DEV)
    flat.normal_(0.0, 0.02, generator=gen)
    p = lay.views(flat)
    # A trained router separates the experts it chooses from the others, and uses some far more than others: the
    # tokens are noise plus the combination of router rows that gives them such logits.
    pop = torch.rand(e, generator=gen, device=DEV).mul_(3.0).exp_()
    picked = torch.multinomial(pop.expand(t, e), k, generator=gen)
    logits = torch.rand(t, e, generator=gen, device=DEV) * 2 - 2
    logits.scatter_add_(1, picked, 3.0 + torch.rand(t, k, generator=gen, device=DEV))
    r = p["router"].float()
    noise = torch.randn(t, h, generator=gen, device=DEV)
    n2 = noise + torch.linalg.solve(r @ r.t(), (logits - noise @ r.t()).t()).t() @ r
    return {"cfg": cfg, "layout": lay, "p": p, "n2": n2.bfloat16(), "h1": _bf(gen, t, h), "dout": _bf(gen, t, h, scale=0.01)}


def _attention_inputs(case: dict, seed: int) -> dict:
    gen, t, hq, hkv, d = _gen(seed), case["tokens"], case["hq"], case["hkv"], case["d"]
    return {"qkv": _bf(gen, t, (hq + 2 * hkv) * d), "dout": _bf(gen, t, hq * d, scale=0.01)}


def _head_inputs(case: dict, seed: int) -> dict:
    gen, t, h, v = _gen(seed), case["tokens"], case["hidden"], case["vocab"]
    mask = torch.rand(t, generator=torch.Generator().manual_seed(t)) < case["counted"]
    mask[-1] = case["counted"] >= 1.0
    rows = mask.nonzero().flatten().to(DEV)
    return {"x": _bf(gen, t, h), "norm": _bf(gen, h, scale=0.1, shift=1.0), "lm": _bf(gen, v, h, scale=0.02),
            "targets": torch.randint(0, v, (t,), generator=gen, device=DEV), "rows": rows}


def _optimizer_inputs(case: dict, seed: int) -> dict:
    gen, n = _gen(seed), case["numel"]
    sd = torch.float32 if case["fp32_moments"] else torch.bfloat16
    f = lambda scale: torch.randn(n, generator=gen, device=DEV).mul_(scale)   # noqa: E731
    return {"master": f(0.02), "m": f(1e-4).to(sd), "v": f(1e-4).square_().to(sd), "gacc": f(1e-4), "g": f(1e-4).bfloat16(),
            "param": torch.zeros(n, dtype=torch.bfloat16, device=DEV)}


def _step_tensors(case: dict, seed: int) -> dict:
    """Checkpoint tensors of a small model under their Hugging Face names."""
    cfg, gen = _config(case), _gen(seed)
    h, f, d, v = case["hidden"], case["inter"], case["d"], case["vocab"]
    mat = lambda *s: torch.randn(*s, generator=gen, device=DEV).mul_(0.02)   # noqa: E731
    sd = {"model.embed_tokens.weight": mat(v, h)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        for n, rows in (("q", case["hq"] * d), ("k", case["hkv"] * d), ("v", case["hkv"] * d)):
            sd[p + f"self_attn.{n}_proj.weight"] = mat(rows, h)
            if cfg.attention_bias:
                sd[p + f"self_attn.{n}_proj.bias"] = mat(rows)
        sd[p + "self_attn.o_proj.weight"] = mat(h, case["hq"] * d)
        sd[p + "mlp.gate_proj.weight"], sd[p + "mlp.up_proj.weight"] = mat(f, h), mat(f, h)
        sd[p + "mlp.down_proj.weight"] = mat(h, f)
        sd[p + "input_layernorm.weight"], sd[p + "post_attention_layernorm.weight"] = mat(h).mul_(5).add_(1), mat(h).mul_(5).add_(1)
    sd["model.norm.weight"] = mat(h).mul_(5).add_(1)
    if not case["tied"]:
        sd["lm_head.weight"] = mat(v, h)
    return {k: x.bfloat16().float() for k, x in sd.items()}


# ------------------------------------------------------------------------------------------ what a program has in hand
def prepare(case: dict, seed: int) -> dict:
    ops, kind = _ops(), case["kind"]
    if kind == "step":
        eng = ShardedEngine(_config(case), torch.device(DEV, torch.cuda.current_device()), ops, optim=OptimConfig(lr=LR))
        eng.load_hf_tensors(_step_tensors(case, seed).__getitem__)
        return {"kind": kind, "engine": eng, "batch": _host_batch(case, seed)}
    if kind == "block":
        s = _block_inputs(case, seed)
        s["batch"] = D.make_packed_batch(_host_batch(case, seed), DEV)
        s["inv_freq"] = s["cfg"].rope_inv_freq().to(DEV)
        s["g"] = s["layout"].views(torch.zeros(s["layout"].padded_numel, dtype=torch.bfloat16, device=DEV))
        return {"kind": kind, "ops": ops, "recompute": case["recompute"], **s}
    if kind == "moe":
        s = _moe_inputs(case, seed)
        s["gflat"] = torch.zeros(s["layout"].padded_numel, dtype=torch.bfloat16, device=DEV)
        s["g"] = s["layout"].views(s["gflat"])
        return {"kind": kind, "ops": ops, **s}
    if kind == "attention":
        cu = [0]
        for n in _lengths(case):
            cu.append(cu[-1] + n)
        return {"kind": kind, "ops": ops, "cu_host": cu, "cu": torch.tensor(cu, dtype=torch.int32, device=DEV),
                "max_seqlen": max(_lengths(case)), "hq": case["hq"], "hkv": case["hkv"], "d": case["d"], **_attention_inputs(case, seed)}
    if kind == "head":
        s = _head_inputs(case, seed)
        targets = torch.full_like(s["targets"], -100)
        targets[s["rows"]] = s["targets"][s["rows"]]
        t = case["tokens"]
        partial = s["rows"].numel() < t
        cu = torch.tensor([0, t], dtype=torch.int32, device=DEV)
        batch = D.PackedBatch(torch.zeros(t, dtype=torch.int64, device=DEV), targets, torch.arange(t, dtype=torch.int32, device=DEV), cu,
                              [0, t], t, s["rows"] if partial else None, targets[s["rows"]] if partial else None)
        return {"kind": kind, "ops": ops, "cfg": _config(case), "batch": batch, "x": s["x"], "p": {"norm": s["norm"]}, "lm": s["lm"],
                "g": {"norm": torch.zeros_like(s["norm"])}, "dlm": torch.zeros_like(s["lm"]), "scale": 1.0 / s["rows"].numel()}
    return {"kind": kind, "ops": ops, "step": 3, **_optimizer_inputs(case, seed)}


# ------------------------------------------------------------------------------------------ one pass
def run(state: dict):
    s, kind = state, state["kind"]
    if kind == "step":
        eng = s["engine"]
        out = eng.train_step([s["batch"]], LR)
        res = {"loss_sum": out["loss_sum"], "grad_norm": out["grad_norm"]}
        for grp in eng.groups:
            for name, v in grp.layout.views(grp.gacc).items():
                res[f"{grp.layout.name}.{name}.grad"] = v
            for name, v in grp.layout.views(grp.master).items():
                res[f"{grp.layout.name}.{name}"] = v
        return res
    ops = s["ops"]
    if kind == "block":
        cfg, p, x, batch, inv = s["cfg"], s["p"], s["x"], s["batch"], s["inv_freq"]
        out, acts, _ = D.block_forward(ops, cfg, p, x, batch, inv, keep=False if s["recompute"] else "compact")
        if s["recompute"]:
            _, acts, _ = D.block_forward(ops, cfg, p, x, batch, inv, keep=True, need_out=False)
        dx = D.block_backward(ops, cfg, p, s["g"], acts, s["dout"], batch, inv)
        return {"out": out, "dx": dx, "grads": s["g"]}
    if kind == "moe":
        out, st = M.moe_forward(ops, s["cfg"], s["p"], s["n2"], s["h1"], True, False)
        dn2 = M.moe_backward(ops, s["cfg"], s["p"], s["g"], st, s["n2"], s["dout"])
        return {"out": out, "dn2": dn2, "router": s["g"]["router"], "experts": s["gflat"][s["layout"].specs["wgu0"].offset:]}
    if kind == "attention":
        a = (s["cu"], s["cu_host"], s["max_seqlen"], s["hq"], s["hkv"], s["d"])
        out, lse = ops.attention(s["qkv"], *a)
        return {"out": out, "lse": lse, "dqkv": ops.attention_bwd(s["dout"], s["qkv"], out, lse, *a)}
    if kind == "head":
        loss, dx = D.head_forward_backward(ops, s["cfg"], s["p"], s["g"], s["lm"], s["dlm"], False, s["x"], s["batch"], s["scale"])
        return {"loss": loss, "dx": dx, "norm": s["g"]["norm"], "lm_head": s["dlm"]}
    ops.accumulate(s["gacc"], s["g"], True)
    sq = ops.sumsq(s["gacc"])
    coef = torch.clamp(1.0 / (sq.sqrt() + 1e-6), max=1.0)
    s["step"] += 1
    ops.adamw_step(s["master"], s["m"], s["v"], s["gacc"], s["param"], LR, 0.9, 0.95, 1e-8, 0.01, s["step"], coef)
    return {"sq": sq, "gacc": s["gacc"], "master": s["master"], "m": s["m"], "v": s["v"], "param": s["param"]}


# ------------------------------------------------------------------------------------------ cost and accuracy
def _pairs(case: dict) -> float:
    return sum(n * (n + 1) / 2 for n in _lengths(case))


def work(case: dict) -> dict:
    """Bytes: inputs, weights and states read once, outputs and gradients written once. FLOPs: two per multiply-add of the
    matrix products, forward once and backward twice (attention: two products forward, five backward, causal half)."""
    kind, t = case["kind"], case.get("tokens", 0)
    if kind == "optimizer":
        n, sd = case["numel"], 4 if case["fp32_moments"] else 2
        return {"bytes": n * (2 + 2 * 4 + 2 * 4 + 4 * sd + 2), "flops": 20 * n}
    h = case.get("hidden", 0)
    if kind == "attention":
        q, kv = case["hq"] * case["d"], case["hkv"] * case["d"]
        return {"bytes": 2 * t * (2 * (q + 2 * kv) + 2 * q) + 4 * t * case["hq"], "flops": 14 * q * _pairs(case)}
    if kind == "head":
        rows = int(t * case["counted"])
        return {"bytes": 2 * (2 * case["vocab"] * h + 2 * t * h) + 4 * t, "flops": 6 * rows * h * case["vocab"]}
    if kind == "moe":
        f, e, k = case["inter"], case["experts"], case["chosen"]
        return {"bytes": 2 * (2 * e * (3 * h * f + h) + 5 * t * h), "flops": 6 * t * (k * 3 * h * f + e * h)}
    q, kv = case["hq"] * case["d"], case["hkv"] * case["d"]
    mats = 2 if case.get("family") == "starcoder2" else 3
    params = h * (q + 2 * kv) + h * q + mats * h * case["inter"]
    if kind == "block":
        again = 2 if case["recompute"] else 0   # forward products made a second time, all but the last
        flops = 6 * t * params + again * t * (params - h * case["inter"]) + (14 + 2 * again) * q * _pairs(case)
        return {"bytes": 2 * (2 * params + 4 * t * h), "flops": flops}
    n = case["layers"]
    total = n * params + case["vocab"] * h * (1 if case["tied"] else 2)
    flops = 6 * t * n * params + 6 * 0.75 * t * h * case["vocab"] + 14 * n * q * _pairs(case)
    return {"bytes": total * 28.0 + 8 * t, "flops": flops}


def tolerance(case: dict) -> dict:
    # Measured against 64 bits at the listed and at drawn sizes, times about four.
    if case["kind"] == "optimizer":   # fp32 sums; parameters and bf16 moments may round the other way
        return {"rel": 1e-3 if case["fp32_moments"] else 4e-3, "max": 0.02}
    if case["kind"] == "step":        # gradients of a whole small model, in bf16 from end to end
        return {"rel": 0.03, "max": 0.6}
    if case["kind"] == "attention":   # bf16 probabilities and outputs
        return {"rel": 0.01, "max": 0.2}
    if case["kind"] == "head":        # bf16 logits and their gradients
        return {"rel": 0.012, "max": 0.2}
    return {"rel": 0.02, "max": 0.4}


# ------------------------------------------------------------------------------------------ the same in 64 bits
class _Attention64(torch.autograd.Function):
    """Causal attention of packed samples, one head of one sample at a time; also returns the log-sum-exp rows."""

    @staticmethod
    def forward(ctx, q, k, v, lens, scale):
        ctx.save_for_backward(q, k, v)
        ctx.lens, ctx.scale = lens, scale
        out = torch.empty_like(q)
        lse = torch.empty(q.shape[1], q.shape[0], dtype=q.dtype, device=q.device)
        for a, n, h, p, ls in _Attention64._rows(q, k, lens, scale):
            out[a:a + n, h] = p @ v[a:a + n, h * v.shape[1] // q.shape[1]]
            lse[h, a:a + n] = ls
        return out, lse

    @staticmethod
    def _rows(q, k, lens, scale):
        a = 0
        for n in lens:
            tri = torch.ones(n, n, dtype=torch.bool, device=q.device).triu_(1)
            for h in range(q.shape[1]):
                s = (q[a:a + n, h] @ k[a:a + n, h * k.shape[1] // q.shape[1]].t()).mul_(scale).masked_fill_(tri, -math.inf)
                ls = torch.logsumexp(s, 1)
                yield a, n, h, s.sub_(ls[:, None]).exp_(), ls
            a += n

    @staticmethod
    def backward(ctx, dout, _):
        q, k, v = ctx.saved_tensors
        dq, dk, dv = torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
        for a, n, h, p, _ls in _Attention64._rows(q, k, ctx.lens, ctx.scale):
            r, j = slice(a, a + n), h * k.shape[1] // q.shape[1]
            dv[r, j] += p.t() @ dout[r, h]
            dp = dout[r, h] @ v[r, j].t()
            ds = dp.sub_((dp * p).sum(1, keepdim=True)).mul_(p).mul_(ctx.scale)
            dq[r, h] = ds @ k[r, j]
            dk[r, j] += ds.t() @ q[r, h]
        return dq, dk, dv, None, None


def _rms64(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _block64(case: dict, p: dict, x, lens: list):
    t, hq, hkv, d, family = case["tokens"], case["hq"], case["hkv"], case["d"], case.get("family", "llama")
    ln = family == "starcoder2"
    norm = (lambda y, n: torch.nn.functional.layer_norm(y, (y.shape[1],), p[n], p["b" + n], EPS)) if ln else (lambda y, n: _rms64(y, p[n]))
    lin = lambda y, w, b: y @ p[w].t() + (p[b] if b in p else 0.0)   # noqa: E731
    qkv = lin(norm(x, "ln1"), "wqkv", "bqkv").view(t, hq + 2 * hkv, d)
    q, k, v = qkv[:, :hq], qkv[:, hq:hq + hkv], qkv[:, hq + hkv:]
    if "qn" in p:
        q, k = _rms64(q, p["qn"]), _rms64(k, p["kn"])
    inv = (1.0 / THETA ** (torch.arange(0, d, 2, dtype=torch.float64) / d)).float().double().to(DEV)
    ang = torch.cat([torch.arange(n, device=DEV, dtype=torch.float64) for n in lens])[:, None] * inv
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]
    rot = lambda y: torch.cat([y[..., : d // 2] * cos - y[..., d // 2:] * sin, y[..., d // 2:] * cos + y[..., : d // 2] * sin], -1)   # noqa: E731
    o, _ = _Attention64.apply(rot(q), rot(k), v, lens, d ** -0.5)
    h1 = x + lin(o.reshape(t, hq * d), "wo", "bo")
    u = lin(norm(h1, "ln2"), "wgu", "bgu")
    if ln:
        a = torch.nn.functional.gelu(u, approximate="tanh")
    else:
        a = torch.nn.functional.silu(u[:, : u.shape[1] // 2]) * u[:, u.shape[1] // 2:]
    return h1 + lin(a, "wd", "bd")


def _ce64(n, lm, targets, scale):
    """Per-row loss, and the gradients of ``scale * sum(loss)`` for rows and head, a chunk of rows at a time."""
    loss, dn, dlm = [], torch.empty_like(n), torch.zeros_like(lm)
    for a in range(0, n.shape[0], 1024):
        z = n[a:a + 1024] @ lm.t()
        y = targets[a:a + 1024, None]
        lse = torch.logsumexp(z, 1, keepdim=True)
        loss.append((lse - z.gather(1, y))[:, 0])
        z.sub_(lse).exp_().scatter_add_(1, y, torch.full_like(lse, -1.0)).mul_(scale)
        dn[a:a + 1024] = z @ lm
        dlm.addmm_(z.t(), n[a:a + 1024])
    return torch.cat(loss), dn, dlm


def _exact_step(case: dict, seed: int) -> dict:
    sd = {k: v.double().requires_grad_() for k, v in _step_tensors(case, seed).items()}
    mb, lens = _host_batch(case, seed), _lengths(case)
    ids, labels = mb["input_ids"].view(-1).to(DEV), mb["labels"].view(-1).to(DEV)
    targets = torch.full_like(labels, -100)
    targets[:-1] = labels[1:]
    rows = (targets != -100).nonzero().flatten()
    scale = 1.0 / mb["batch_num_loss_counted_tokens"]
    x = sd["model.embed_tokens.weight"][ids]
    blocks = []
    for i in range(case["layers"]):
        g = lambda n: sd[f"model.layers.{i}.{n}"]   # noqa: B023, E731
        p = {"ln1": g("input_layernorm.weight"), "wqkv": torch.cat([g(f"self_attn.{n}_proj.weight") for n in "qkv"]),
             "wo": g("self_attn.o_proj.weight"), "ln2": g("post_attention_layernorm.weight"),
             "wgu": torch.cat([g("mlp.gate_proj.weight"), g("mlp.up_proj.weight")]), "wd": g("mlp.down_proj.weight")}
        if case["bias"]:
            p["bqkv"] = torch.cat([g(f"self_attn.{n}_proj.bias") for n in "qkv"])
        p = {n: w.detach().requires_grad_() for n, w in p.items()}
        blocks.append(p)
        x = _block64(case, p, x, lens)
    n = _rms64(x[rows], sd["model.norm.weight"])
    lm = sd["model.embed_tokens.weight"] if case["tied"] else sd["lm_head.weight"]
    loss, dn, dlm = _ce64(n.detach(), lm.detach(), targets[rows], scale)
    n.backward(dn)
    grads = {"embed": {"embed": sd["model.embed_tokens.weight"].grad + (dlm if case["tied"] else 0.0)}}
    weights = {"embed": {"embed": sd["model.embed_tokens.weight"]}, "head": {"norm": sd["model.norm.weight"]}}
    for i, p in enumerate(blocks):
        grads[f"block{i}"], weights[f"block{i}"] = {k: w.grad for k, w in p.items()}, p
    grads["head"] = {"norm": sd["model.norm.weight"].grad}
    if not case["tied"]:
        grads["head"]["lm_head"], weights["head"]["lm_head"] = dlm, lm
    norm = math.sqrt(sum(float(g.square().sum()) for d in grads.values() for g in d.values()))
    coef = min(1.0, 1.0 / (norm + 1e-6))
    res = {"loss_sum": loss.sum(), "grad_norm": torch.tensor(norm, dtype=torch.float64)}
    for grp, d in grads.items():
        for name, g in d.items():
            u = g * coef   # first step: both bias corrections cancel
            res[f"{grp}.{name}.grad"] = g
            res[f"{grp}.{name}"] = weights[grp][name].detach() - LR * u / (u.abs() + 1e-8)
    return res


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "step":
        return _exact_step(case, seed)
    if kind == "block":
        s = _block_inputs(case, seed)
        p = {n: w.double().requires_grad_() for n, w in s["p"].items()}
        x = s["x"].double().requires_grad_()
        out = _block64(case, p, x, _lengths(case))
        out.backward(s["dout"].double())
        return {"out": out.detach(), "dx": x.grad, "grads": {n: w.grad for n, w in p.items()}}
    if kind == "moe":
        return _exact_moe(case, seed)
    if kind == "attention":
        s = _attention_inputs(case, seed)
        t, hq, hkv, d = case["tokens"], case["hq"], case["hkv"], case["d"]
        qkv = s["qkv"].double().requires_grad_()
        r = qkv.view(t, hq + 2 * hkv, d)
        out, lse = _Attention64.apply(r[:, :hq], r[:, hq:hq + hkv], r[:, hq + hkv:], _lengths(case), d ** -0.5)
        out.backward(s["dout"].double().view(t, hq, d))
        return {"out": out.detach().reshape(t, hq * d), "lse": lse.detach(), "dqkv": qkv.grad}
    if kind == "head":
        s = _head_inputs(case, seed)
        rows = s["rows"]
        x, w = s["x"].double()[rows].requires_grad_(), s["norm"].double().requires_grad_()
        n = _rms64(x, w)
        loss, dn, dlm = _ce64(n.detach(), s["lm"].double(), s["targets"][rows], 1.0 / rows.numel())
        n.backward(dn)
        full, dx = torch.zeros(case["tokens"], dtype=torch.float64, device=DEV), torch.zeros(s["x"].shape, dtype=torch.float64, device=DEV)
        full[rows], dx[rows] = loss, x.grad
        return {"loss": full, "dx": dx, "norm": w.grad, "lm_head": dlm}
    s = {k: v.double() for k, v in _optimizer_inputs(case, seed).items()}
    g = s["gacc"] + s["g"]
    sq = g.square().sum()
    u = g * torch.clamp(1.0 / (sq.sqrt() + 1e-6), max=1.0)
    m, v = 0.9 * s["m"] + 0.1 * u, 0.95 * s["v"] + 0.05 * u * u
    w = s["master"] * (1 - LR * 0.01) - LR / (1 - 0.9 ** 4) * m / (v.sqrt() / math.sqrt(1 - 0.95 ** 4) + 1e-8)
    return {"sq": sq.view(1), "gacc": g, "master": w, "m": m, "v": v, "param": w}


def _exact_moe(case: dict, seed: int) -> dict:
    s = _moe_inputs(case, seed)
    h, f, k, t = case["hidden"], case["inter"], case["chosen"], case["tokens"]
    n2, h1, dout, r = s["n2"].double(), s["h1"].double(), s["dout"].double(), s["p"]["router"].double()
    probs = torch.softmax(n2 @ r.t(), 1)
    topv, topi = probs.topk(k, 1)
    w = topv / topv.sum(1, keepdim=True)
    y, dn2, dw, experts = torch.zeros_like(n2), torch.zeros_like(n2), torch.zeros_like(w), []
    for e in range(case["experts"]):
        tok, slot = (topi == e).nonzero(as_tuple=True)
        wgu, wd = s["p"][f"wgu{e}"].double(), s["p"][f"wd{e}"].double()
        xs, do, we = n2[tok], dout[tok], w[tok, slot][:, None]
        g, u = (xs @ wgu.t()).split(f, 1)
        sig = torch.sigmoid(g)
        a = g * sig * u
        ye = a @ wd.t()
        y.index_add_(0, tok, ye * we)
        dw[tok, slot] = (do * ye).sum(1)
        da = (do * we) @ wd
        dgu = torch.cat([da * u * sig * (1 + g * (1 - sig)), da * g * sig], 1)
        dn2.index_add_(0, tok, dgu @ wgu)
        experts += [(dgu.t() @ xs).view(-1), ((do * we).t() @ a).reshape(-1)]
    dtop = (dw - (dw * w).sum(1, keepdim=True)) / topv.sum(1, keepdim=True)
    dp = torch.zeros_like(probs).scatter_(1, topi, dtop)
    dl = probs * (dp - (dp * probs).sum(1, keepdim=True))
    flat = torch.zeros(s["layout"].padded_numel - s["layout"].specs["wgu0"].offset, dtype=torch.float64, device=DEV)
    base = s["layout"].specs["wgu0"].offset
    for e in range(case["experts"]):
        for name, v in ((f"wgu{e}", experts[2 * e]), (f"wd{e}", experts[2 * e + 1])):
            o = s["layout"].specs[name].offset - base
            flat[o:o + v.numel()] = v
    return {"out": h1 + y, "dn2": dn2 + dl @ r, "router": dl.t() @ n2, "experts": flat}
