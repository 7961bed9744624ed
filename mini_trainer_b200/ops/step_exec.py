"""Host side of ``csrc/step_exec.cu``: forward and backward of a minibatch through a whole small model, queued by one native call.

The schedule is that of ``parallel/engine.py`` for one rank whose blocks all keep their activations; that file is the definition. ``forward_backward``
returns ``None`` for what stays with it: several ranks, models or options the call does not cover, and minibatches whose buffers are large
(``MOST_WORKSPACE``; the device is the bound there) or find no room.
"""
from __future__ import annotations

import ctypes
import os
from ctypes import c_float, c_int, c_longlong, c_void_p

import torch

from ..utils import nvtx
from . import block_exec, gemm_plan

MOST_WORKSPACE = 1 << 30
PARAMS = len(block_exec.NAMES)


class Spec(ctypes.Structure):
    _fields_ = [("block", block_exec.Spec)] + [(n, c_int) for n in ("layers", "V", "R", "tied")] \
        + [(n, c_float) for n in ("logit_alpha", "grad_scale")] + [("form", c_int * 3), ("splits", c_int * 3), ("off", c_longlong * PARAMS)] \
        + [(n, c_longlong) for n in ("off_embed", "off_norm", "off_bnorm", "off_lm")]


class Group(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in ("param", "grad", "acc")] + [("n", c_longlong), ("add", c_int)]


class IO(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in ("embed", "blocks", "head", "inv_freq", "ids", "targets", "rows", "pos", "fwd_plan", "bwd_plan", "loss", "ws", "counters",
                                        "epochs", "part")] + [("part_bytes", c_longlong), ("status", c_void_p)]


def check_layout(lib) -> None:
    sizes = (c_int * 3)()
    lib.mtb200_step_sizes(sizes)
    if list(sizes) != [ctypes.sizeof(t) for t in (Spec, Group, IO)]:
        raise RuntimeError(f"the library lays its step structures out in {list(sizes)} bytes: it is of another version, build it again")


def covers(eng) -> bool:
    """Whether the engine's model and set-up are ones that the call covers, whatever the minibatch."""
    cfg, ops = eng.cfg, eng.ops
    return (hasattr(ops, "step_forward_backward") and eng.world == 1 and not eng.symmetric and eng.param_dtype == torch.bfloat16
            and not cfg.is_moe and not cfg.post_norm and cfg.head_dim in (64, 128) and cfg.norm_weight_offset == 0.0 and cfg.rotary_dim == cfg.head_dim
            and cfg.embedding_multiplier == 1.0 and not (cfg.mlp_gated and cfg.mlp_bias)
            and (cfg.residual_multiplier == 1.0 or not (cfg.o_proj_bias or cfg.mlp_bias)) and len(eng.blocks) <= 256
            and not ops.ce_wants_stats(cfg.vocab_size, cfg.hidden_size)
            and all(g.gacc.numel() <= eng.INLINE_REDUCE for g in eng.groups))


def _ready(eng, batch) -> bool:
    ops = eng.ops
    rows = batch.loss_rows
    R = batch.num_tokens if rows is None else rows.shape[0]
    return (getattr(eng, "osft", None) is None and eng.activation_budget_bytes is None and not eng.poison and not eng._oom_retries and ops.profile is None
            and not nvtx.ENABLED and ops.attention_impl == "native" and not eng.stalls_recorded() and os.environ.get("MTB200_OFFLOAD_BLOCKS", "0") == "0"
            and 0 < batch.num_tokens <= ops.EMB_SCAN and 0 < R <= ops.ce_chunk and batch.input_ids.is_contiguous() and batch.targets.is_contiguous()
            and batch.position_ids.dtype == torch.int32 and not torch.cuda.is_current_stream_capturing())


def _spec(eng, T: int, R: int):
    """``(spec, bytes of partial sums)`` of a minibatch of ``T`` tokens whose head runs on ``R`` rows."""
    ops, cfg = eng.ops, eng.cfg
    tied = cfg.tie_word_embeddings
    block, fwd_part, bwd_part, _ = block_exec._spec(ops, cfg, T)
    lay, head = eng.blocks[0].layout.specs, eng.head.layout.specs
    H, V = cfg.hidden_size, cfg.vocab_size
    s = Spec(block, len(eng.blocks), V, R, int(tied), 1.0 / cfg.logits_scaling)
    s.off[:] = [lay[n].offset if n in lay else -1 for n in block_exec.NAMES]
    s.off_embed, s.off_norm, s.off_bnorm = eng.embed.layout.specs["embed"].offset, head["norm"].offset, head["bnorm"].offset if "bnorm" in head else -1
    s.off_lm = s.off_embed if tied else head["lm_head"].offset
    plans = [ops.product_plan(*m) for m in ((R, V, H, H), (R, H, V, V | H), (V, H, R, V | H))]
    s.form[:], s.splits[:] = [gemm_plan.FORMS[n] for n, _, _ in plans], [k for _, k, _ in plans]
    return s, max(fwd_part, bwd_part, *(b if k > 1 else 0 for _, k, b in plans))


def forward_backward(eng, batch, grad_scale: float):
    """``ShardedEngine.forward_backward``, or ``None``."""
    if not _ready(eng, batch):
        return None
    ops, cfg, rows = eng.ops, eng.cfg, batch.loss_rows
    T = batch.num_tokens
    key = (T, T if rows is None else rows.shape[0], cfg.vocab_size, cfg.hidden_size)
    hit = eng._step_specs.get(key)
    if hit is None:
        if len(eng._step_specs) >= 1024:
            eng._step_specs.clear()
        hit = eng._step_specs[key] = _spec(eng, *key[:2])
    s = Spec.from_buffer_copy(hit[0])
    b = s.block
    cu = batch.cu_seqlens_host
    name, tail, fwd_plan = ops._cached(cu, ("fwd", b.Hq, b.Hkv, b.D)) or ops._plan_attention(cu, b.Hq, b.Hkv, b.D)
    bwd_plan, b.bwd_splits, attn_part, b.bwd_in_order = ops._cached(cu, ("bwd", b.Hq, b.Hkv, b.D)) or ops._plan_attention_bwd(cu, b.Hq, b.Hkv, b.D)
    b.need_out, b.attn_form, b.fwd_items, b.bwd_items = 1, (1 + tail[0] if name == "mtb200_attn_fwd" else 0), fwd_plan.shape[0], bwd_plan.shape[0]
    s.grad_scale = grad_scale
    io = IO()
    io.rows = None if rows is None else rows.data_ptr()
    nbytes = ops.lib.mtb200_step_workspace(ctypes.byref(s), ctypes.byref(io))
    if not 0 <= nbytes <= MOST_WORKSPACE:
        return None
    ws = block_exec._workspace(ops, nbytes)
    if ws is None:
        return None
    for ev in (*eng._root_free.values(), *eng._gbuf_free):   # reductions of an earlier minibatch that went another way
        eng.wait_event(ev)
    group = lambda g, grad: Group(g.shard.data_ptr(), grad.data_ptr(), g.gacc.data_ptr(), g.gacc.numel(), int(g.has_grad))   # noqa: E731
    embed, head = group(eng.embed, eng._eg_full), group(eng.head, eng._hg_full)
    n = len(eng.blocks)
    blocks = (Group * n)(*(group(g, eng._gbufs[i % len(eng._gbufs)]) for i, g in enumerate(eng.blocks)))
    inv = [eng._inv_freq(i, batch) for i in range(n)]
    freqs = (c_void_p * n)(*(None if f is None else f.data_ptr() for f in inv))
    loss = torch.empty(T, dtype=torch.float32, device=ops.device)
    io.embed, io.blocks, io.head, io.inv_freq = (ctypes.addressof(x) for x in (embed, blocks, head, freqs))
    targets = batch.targets if rows is None else batch.loss_targets
    io.ids, io.targets, io.pos = batch.input_ids.data_ptr(), targets.data_ptr(), batch.position_ids.data_ptr()
    io.fwd_plan, io.bwd_plan, io.loss, io.ws, io.status = fwd_plan.data_ptr(), bwd_plan.data_ptr(), loss.data_ptr(), ws.data_ptr(), ops.status.data_ptr()
    st = ops._st()
    part = max(hit[1], attn_part if b.bwd_splits > 1 else 0)
    got = ops._split(st, part) if part else None
    if got is not None:
        counters, first, partials = got
        epochs = (ctypes.c_ulonglong * (13 * n + 4))(first, *(next(ops._epoch) for _ in range(13 * n + 3)))
        io.counters, io.epochs, io.part, io.part_bytes = counters.data_ptr(), ctypes.addressof(epochs), partials.data_ptr(), 4 * partials.numel()
    block_exec._call(ops, "mtb200_step_forward_backward", ctypes.byref(s), ctypes.byref(io), st)
    for g in eng.groups:
        g.has_grad = True
    eng._root_free = {"embed": None, "head": None}
    eng._gbuf_free = [None] * len(eng._gbuf_free)
    return loss
