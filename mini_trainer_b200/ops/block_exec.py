"""Host side of ``csrc/block_exec.cu``: a dense pre-norm decoder block, forward or backward, queued by one native call.

The block is that of ``models/decoder.py`` on the kernels of ``native.py``: the same launches in the same order, without the interpreter
between them. ``forward`` and ``backward`` return ``None`` for what stays with the Python form: other block forms, parameters that are being
gathered, tensors that are not laid out as the native call addresses them, and blocks whose temporaries are large (``MOST_WORKSPACE``; the device
is the bound there) or find no room: the Python form gives each temporary back when it is done with.
"""
from __future__ import annotations

import ctypes
from ctypes import c_char_p, c_float, c_int, c_longlong, c_void_p

import torch

from ..utils import nvtx
from . import gemm_plan

MOST_WORKSPACE = 256 << 20
GEMMS = 12   # G_QKV .. W_QKV of csrc/block_exec.cu
NAMES = ("ln1", "bln1", "wqkv", "bqkv", "qn", "kn", "wo", "bo", "ln2", "bln2", "wgu", "bgu", "wd", "bd")


class Spec(ctypes.Structure):
    _fields_ = [(n, c_int) for n in ("T", "H", "F", "Hq", "Hkv", "D", "gated", "gelu", "layernorm", "qk_norm")] \
        + [(n, c_float) for n in ("eps", "scale", "alpha")] + [("form", c_int * GEMMS), ("splits", c_int * GEMMS), ("act_form", c_int)] \
        + [(n, c_int) for n in ("need_out", "attn_form", "fwd_items", "bwd_items", "bwd_splits", "bwd_in_order")]


class Params(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in NAMES]


class IO(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in ("x", "n1", "qkv", "attn", "h1", "n2", "gu", "act", "out", "qk_pre", "mean1", "rstd1", "lse", "mean2", "rstd2",
                                        "rstd_qk", "pos", "fwd_plan", "bwd_plan", "inv_freq")] \
        + [("have_attn", c_int)] + [(n, c_void_p) for n in ("dout", "dx", "ws", "counters", "epochs", "part")] \
        + [("part_bytes", c_longlong), ("status", c_void_p)]


def check_layout(lib) -> None:
    """The structures are laid out here and in ``csrc/block_exec.h``, the kernels of a product numbered in ``gemm_plan`` and in ``csrc/entries.h``."""
    sizes = (c_int * 3)()
    lib.mtb200_block_sizes(sizes)
    if list(sizes) != [ctypes.sizeof(t) for t in (Spec, Params, IO)]:
        raise RuntimeError(f"the library lays its block structures out in {list(sizes)} bytes: it is of another version, build it again")
    lib.mtb200_gemm_form.restype = c_char_p
    names = [lib.mtb200_gemm_form(i) for i in range(len(gemm_plan.FORMS) + 1)]
    if names != [*(n.encode() for n in gemm_plan.FORMS), None]:
        raise RuntimeError(f"the library numbers the kernels of a product {names}: it is of another version, build it again")


def _ptr(t):
    return None if t is None else t.data_ptr()


def _params(p: dict):
    """Addresses of the block's tensors, or ``None`` when one of them is not a plain bf16 array."""
    out = Params()
    for n in NAMES:
        t = p.get(n)
        if t is not None:
            if t.dtype != torch.bfloat16 or not t.is_contiguous():
                return None
            setattr(out, n, t.data_ptr())
    return out


def _supported(ops, cfg, p: dict, x, batch) -> bool:
    return (ops.profile is None and not nvtx.ENABLED and ops.attention_impl == "native" and cfg.head_dim in (64, 128) and not cfg.is_moe
            and not cfg.post_norm and cfg.norm_weight_offset == 0.0 and cfg.rotary_dim == cfg.head_dim and "_gather" not in p
            and not (cfg.mlp_gated and "bgu" in p) and (cfg.residual_multiplier == 1.0 or not ("bo" in p or "bd" in p))
            and x.dtype == torch.bfloat16 and x.is_contiguous() and x.shape[0] > 0 and batch.position_ids.dtype == torch.int32)


def _spec(ops, cfg, T: int):
    """``(spec, bytes of partial sums forward, backward, workspace bytes by direction)`` of a block on ``T`` tokens."""
    key = (T, cfg.hidden_size, cfg.intermediate_size, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, cfg.mlp_gated, cfg.mlp_act,
           cfg.norm_type, cfg.qk_norm, cfg.rms_norm_eps, cfg.attention_scale, cfg.residual_multiplier)
    hit = ops._block_specs.get(key)
    if hit is None:
        H, F, q, Q = cfg.hidden_size, cfg.intermediate_size, cfg.q_size, cfg.qkv_size
        gu = 2 * F if cfg.mlp_gated else F
        products = [(T, Q, H), (T, H, q), (T, gu, H), (T, H, F), (T, F, H), (T, H, gu), (T, q, H), (T, H, Q), (H, F, T), (gu, H, T), (H, q, T), (Q, H, T)]
        # leading dimensions: forward K and K, input gradients K and N, weight gradients M and N
        pitches = [k for _, _, k in products[:4]] + [n | k for _, n, k in products[4:8]] + [m | n for m, n, _ in products[8:]]
        plans = [ops.product_plan(*m, ld) for m, ld in zip(products, pitches)]
        s = Spec(T, H, F, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, int(cfg.mlp_gated),
                 int((cfg.mlp_act if cfg.mlp_gated else "gelu_tanh") != "silu"), int(cfg.norm_type == "layernorm"), int(cfg.qk_norm), cfg.rms_norm_eps,
                 cfg.attention_scale, cfg.residual_multiplier)
        s.form[:] = [gemm_plan.FORMS[n] for n, _, _ in plans]
        act, _, _ = ops.product_plan(*products[2], pitches[2], act=True)
        s.act_form = gemm_plan.FORMS[act]
        s.splits[:] = [k for _, k, _ in plans]
        part = [b if k > 1 else 0 for _, k, b in plans]
        if len(ops._block_specs) >= 1024:
            ops._block_specs.clear()
        hit = ops._block_specs[key] = (s, max(part[:4]), max(part[4:]), {})
    return hit


def _workspace_bytes(ops, spec, io, bwd: int, sizes: dict) -> int:
    what = (bwd, io.n1 is None, io.n2 is None, io.act is None)
    n = sizes.get(what)
    if n is None:
        n = sizes[what] = ops.lib.mtb200_block_workspace(ctypes.byref(spec), ctypes.byref(io), bwd)
    return n


def _workspace(ops, n: int):
    """The last tensor that a call takes: the Python form needs less than this at a time, and its results as well."""
    try:
        return torch.empty(max(n, 1), dtype=torch.uint8, device=ops.device)
    except torch.OutOfMemoryError:
        return None


def _split(ops, io, stream, nbytes: int):
    """Scratch and epochs of the launches that split; what has to stay alive until they are queued."""
    got = ops._split(stream, nbytes) if nbytes else None
    if got is None:
        return None
    counters, first, part = got
    epochs = (ctypes.c_ulonglong * (GEMMS + 1))(first, *(next(ops._epoch) for _ in range(GEMMS)))
    io.counters, io.epochs, io.part, io.part_bytes = counters.data_ptr(), ctypes.addressof(epochs), part.data_ptr(), 4 * part.numel()
    return counters, epochs, part


def forward(ops, acts_type, cfg, p: dict, x, batch, inv_freq, keep, saved_attn, want_attn, need_out):
    """``decoder.block_forward``, or ``None``."""
    if not _supported(ops, cfg, p, x, batch):
        return None
    prm = _params(p)
    T, H = x.shape
    F, q, Q = cfg.intermediate_size, cfg.q_size, cfg.qkv_size
    if prm is None or (saved_attn is not None and not saved_attn[0].is_contiguous()):
        return None
    base, nbytes, _, sizes = _spec(ops, cfg, T)
    spec = Spec.from_buffer_copy(base)
    bf = lambda *s: torch.empty(s, dtype=torch.bfloat16, device=ops.device)      # noqa: E731
    f32 = lambda *s: torch.empty(s, dtype=torch.float32, device=ops.device)      # noqa: E731
    io = IO()
    io.x, io.status = x.data_ptr(), ops.status.data_ptr()
    ln, full = bool(spec.layernorm), keep is True
    n1 = n2 = act = None
    if full:   # (otherwise they live in the workspace)
        n1, n2, act = bf(T, H), bf(T, H), bf(T, F) if need_out else None
        io.n1, io.n2, io.act = n1.data_ptr(), n2.data_ptr(), _ptr(act)
    ws_bytes = _workspace_bytes(ops, spec, io, 0, sizes)
    if ws_bytes > MOST_WORKSPACE:
        return None
    qkv, h1, gu = bf(T, Q), bf(T, H), bf(T, 2 * F if cfg.mlp_gated else F)
    out = bf(T, H) if need_out else None
    attn, lse = saved_attn if saved_attn is not None else (bf(T, q), f32(spec.Hq, T))
    r1, r2 = f32(T), f32(T)
    m1, m2 = (f32(T), f32(T)) if ln else (None, None)
    pre, rqk = (bf(T, q + cfg.kv_size) if keep else None, f32(T * (spec.Hq + spec.Hkv))) if spec.qk_norm else (None, None)
    ws = _workspace(ops, ws_bytes)
    if ws is None:
        return None
    io.qkv, io.attn, io.h1, io.gu, io.out, io.qk_pre = qkv.data_ptr(), attn.data_ptr(), h1.data_ptr(), gu.data_ptr(), _ptr(out), _ptr(pre)
    io.mean1, io.rstd1, io.lse, io.mean2, io.rstd2, io.rstd_qk = _ptr(m1), r1.data_ptr(), lse.data_ptr(), _ptr(m2), r2.data_ptr(), _ptr(rqk)
    io.pos, io.inv_freq, io.ws = batch.position_ids.data_ptr(), _ptr(inv_freq), ws.data_ptr()
    io.have_attn, spec.need_out = int(saved_attn is not None), int(need_out)
    cu = batch.cu_seqlens_host
    if saved_attn is None:
        name, tail, plan = ops._cached(cu, ("fwd", spec.Hq, spec.Hkv, spec.D)) or ops._plan_attention(cu, spec.Hq, spec.Hkv, spec.D)
        spec.attn_form, spec.fwd_items, io.fwd_plan = (1 + tail[0] if name == "mtb200_attn_fwd" else 0), plan.shape[0], plan.data_ptr()
    st = ops._st()
    alive = _split(ops, io, st, nbytes)
    _call(ops, "mtb200_block_forward", ctypes.byref(spec), ctypes.byref(prm), ctypes.byref(io), st)
    del alive
    acts = None
    if keep:
        acts = acts_type(x, n1, (m1, r1) if ln else r1, qkv, attn, lse, h1, n2, (m2, r2) if ln else r2, gu, act, pre, rqk)
    return out, acts, ((attn, lse) if want_attn else None)


def backward(ops, cfg, p: dict, g: dict, a, dout, batch, inv_freq):
    """``decoder.block_backward``, or ``None``."""
    x = a.x
    if not _supported(ops, cfg, p, x, batch) or dout.dtype != torch.bfloat16 or not dout.is_contiguous():
        return None
    prm, grd = _params(p), _params(g)
    kept = (a.qkv, a.attn, a.h1, a.gu, a.lse)
    if prm is None or grd is None or any(n not in g for n in NAMES if n in p) or not all(t.is_contiguous() for t in kept):
        return None
    base, _, nbytes, sizes = _spec(ops, cfg, x.shape[0])
    spec = Spec.from_buffer_copy(base)
    io = IO()
    io.n1, io.n2, io.act = _ptr(a.n1), _ptr(a.n2), _ptr(a.act)
    ws_bytes = _workspace_bytes(ops, spec, io, 1, sizes)
    if ws_bytes > MOST_WORKSPACE:
        return None
    dx = torch.empty_like(x)
    ws = _workspace(ops, ws_bytes)
    if ws is None:
        return None
    io.x, io.qkv, io.attn, io.h1, io.gu, io.qk_pre = x.data_ptr(), a.qkv.data_ptr(), a.attn.data_ptr(), a.h1.data_ptr(), a.gu.data_ptr(), _ptr(a.qk_pre)
    (m1, r1), (m2, r2) = (a.rstd1, a.rstd2) if spec.layernorm else ((None, a.rstd1), (None, a.rstd2))
    io.mean1, io.rstd1, io.lse, io.mean2, io.rstd2, io.rstd_qk = _ptr(m1), r1.data_ptr(), a.lse.data_ptr(), _ptr(m2), r2.data_ptr(), _ptr(a.rstd_qk)
    io.pos, io.inv_freq, io.ws, io.status = batch.position_ids.data_ptr(), _ptr(inv_freq), ws.data_ptr(), ops.status.data_ptr()
    io.dout, io.dx = dout.data_ptr(), dx.data_ptr()
    cu = batch.cu_seqlens_host
    plan, spec.bwd_splits, attn_bytes, spec.bwd_in_order = ops._cached(cu, ("bwd", spec.Hq, spec.Hkv, spec.D)) or ops._plan_attention_bwd(cu, spec.Hq, spec.Hkv, spec.D)
    spec.bwd_items, io.bwd_plan = plan.shape[0], plan.data_ptr()
    st = ops._st()
    alive = _split(ops, io, st, max(nbytes, attn_bytes if spec.bwd_splits > 1 else 0))
    _call(ops, "mtb200_block_backward", ctypes.byref(spec), ctypes.byref(prm), ctypes.byref(grd), ctypes.byref(io), st)
    del alive
    return dx


def _call(ops, name: str, *args):
    n = c_int(0)
    rc = ops._fn[name](*args[:-1], ctypes.byref(n), args[-1])
    if rc != 0:
        raise RuntimeError(f"{name} failed with code {rc}")
    ops.launches += n.value
