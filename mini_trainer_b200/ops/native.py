"""sm_100a kernel backend: ctypes bindings over ``_native/libmtb200_cuda.so``.

Same method set as ``TorchOps``; tensors are bf16 on a CUDA device, 2-D, row-major. Every call
launches on the current torch CUDA stream. A missing library or a non-zero return code raises —
there is no silent fallback to PyTorch on a GPU machine.

``launches`` counts kernels launched through this backend (reported by the benchmark).
"""
from __future__ import annotations

import ctypes
import itertools
import os
from dataclasses import dataclass
from ctypes import c_float, c_int, c_longlong, c_ulonglong, c_void_p

import torch

from .. import build as _build
from ..utils import nvtx
from . import attention_plan, block_exec, gemm_plan, step_exec

_LIB = None
_raw_stream = torch._C._cuda_getCurrentRawStream if hasattr(torch._C, "_cuda_getCurrentRawStream") else \
    (lambda index: torch.cuda.current_stream(index).cuda_stream)


def load_library():
    global _LIB
    if _LIB is not None:
        return _LIB
    path = _build.CUDA_LIB
    if not path.exists() or os.environ.get("MTB200_REBUILD"):
        _build.build_cuda()
    if not path.exists():
        raise RuntimeError(f"native CUDA library {path} is missing and could not be built (nvcc not found)")
    lib = ctypes.CDLL(str(path))
    for name in dir(_Sig):
        if name.startswith("mtb200_") and hasattr(lib, name):
            fn = getattr(lib, name)
            fn.restype = c_int
            fn.argtypes = getattr(_Sig, name)
    lib.mtb200_block_workspace.restype = c_longlong
    lib.mtb200_step_workspace.restype = c_longlong
    block_exec.check_layout(lib)
    step_exec.check_layout(lib)
    _LIB = lib
    return lib


P, I, L, F, U = c_void_p, c_int, c_longlong, c_float, c_ulonglong


class _Sig:
    mtb200_gemm_bf16 = [P, L, I, P, L, I, P, L, I, P, L, P, I, I, I, F, I, P, U, P, L, P, P, P]
    mtb200_gemm2_bf16 = [P, L, I, P, L, I, P, L, I, P, L, P, I, I, I, F, I, P, U, P, L, P, P, P]
    mtb200_gemm2_wide_bf16 = mtb200_gemm_n64_bf16 = mtb200_gemm_n128_bf16 = mtb200_gemm2_bf16
    mtb200_gemm2_pairs = []
    mtb200_gemm_act = [P, L, P, P, P, P, I, I, I, I, I, I, P, P]
    mtb200_rmsnorm_fwd = [P, P, P, P, F, I, I, P, P]
    mtb200_norm_bwd_blocks = [I, I]
    mtb200_rmsnorm_bwd = [P, P, P, P, P, P, P, P, I, I, P, P]
    mtb200_layernorm_fwd = [P, P, P, P, P, P, F, I, I, P, P]
    mtb200_layernorm_bwd = [P, P, P, P, P, P, P, P, P, P, I, I, P, P]
    mtb200_rope = [P, P, P, I, L, I, I, I, P]
    mtb200_head_rmsnorm_fwd = [P, P, P, P, P, P, P, F, I, L, I, I, I, P]
    mtb200_head_rmsnorm_bwd_blocks = [I, I]
    mtb200_head_rmsnorm_bwd = [P, P, P, P, P, P, P, P, P, P, I, L, L, I, I, I, P]
    mtb200_swiglu_fwd = [P, P, L, I, P]
    mtb200_swiglu_bwd = [P, P, P, L, I, P]
    mtb200_swiglu_bwd_act = [P, P, P, L, I, P]
    mtb200_geglu_fwd = [P, P, L, I, P]
    mtb200_geglu_bwd = [P, P, P, L, I, P]
    mtb200_geglu_bwd_act = [P, P, P, L, I, P]
    mtb200_gelu_fwd = [P, P, L, P]
    mtb200_gelu_bwd = [P, P, P, L, P]
    mtb200_gelu_bwd_act = [P, P, P, L, P]
    mtb200_embedding_fwd = [P, P, P, I, I, I, P, P]
    mtb200_embedding_bwd = [P, P, P, P, I, I, I, P, P]
    mtb200_embedding_bwd_scan = [P, P, P, I, I, I, P, P]
    mtb200_scatter_rows = [P, P, P, P, P, I, I, I, P, P]
    mtb200_ce_fwd_bwd = [P, L, I, P, P, P, P, L, I, I, F, L, P]
    mtb200_colsum = [P, L, P, P, I, I, P]
    mtb200_accumulate = [P, P, L, I, I, P]
    mtb200_f32_to_bf16 = [P, P, L, I, P]
    mtb200_sumsq = [P, L, P, P]
    mtb200_adamw = [P, P, P, I, P, P, L, F, F, F, F, F, I, P, P]
    mtb200_sumsq_groups = [P, I, P, P]
    mtb200_adamw_groups = [P, I, I, P, F, P, F, F, F, F, F, I, P]
    mtb200_block_workspace = [P, P, I]
    mtb200_block_forward = [P, P, P, P, P]
    mtb200_block_backward = [P, P, P, P, P, P]
    mtb200_step_workspace = [P, P]
    mtb200_step_forward_backward = [P, P, P, P]
    mtb200_gemm_grouped = [P, L, P, L, P, L, P, I, I, I, I, I, I, P, P, I, L, P, P]
    mtb200_moe_route = [P, I, I, I, I, P, P, P, P]
    mtb200_moe_plan = [P, I, I, I, P, P, P, P, P, P]
    mtb200_moe_gather = [P, P, P, I, I, I, I, F, P, P]
    mtb200_moe_glu_bwd = [P, P, P, P, P, I, I, I, I, P, P, P]
    mtb200_moe_combine = [P, P, P, P, P, F, I, I, I, P, P]
    mtb200_moe_route_bwd = [P, P, P, P, I, I, I, I, P, P]
    mtb200_attn_fwd_one = [P, L, P, L, P, P, I, I, I, I, I, F, P, P]
    mtb200_attn_fwd = [P, L, P, L, P, P, I, I, I, I, I, I, F, P, P]
    mtb200_attn_bwd = [P, L, P, L, P, L, P, L, P, P, P, P, I, I, I, I, I, I, P, U, P, L, F, I, P, P]


_GLU = {"silu": "mtb200_swiglu", "gelu_tanh": "mtb200_geglu"}
_ACT = {"silu": 0, "gelu_tanh": 1}   # of csrc/gemm_act.cuh
_GEMM_TAGS = (("gemm_nt", "gemm_nn"), ("gemm_tt", "gemm_tn"))   # [A stored [K, M]][B stored [K, N]]
_SPLIT_COUNTERS = 4096          # csrc/gemm_epilogue.cuh
_SPLIT_FLOATS = 32 << 20        # most that the partials of a launch take: 128 MB
_SPLIT_UNITS = 4 * _SPLIT_FLOATS // gemm_plan.UNIT_BYTES   # = 1024 of 128 x 256
_EMB_SCAN = 8192                # tokens up to which the embedding gradient goes without a sort (at most EMB_SCAN of csrc/elementwise.cu)
NATIVE_HEAD_DIMS = (64, 128)   # head dimensions of the hand-written attention kernels


_GROUP_ALIGN = 128   # GROUP_ALIGN and GROUP_MAX of csrc/gemm_epilogue.cuh
_GROUP_MAX = 256


@dataclass
class ExpertSlabs:
    """Rows of a mixture-of-experts layer grouped by expert (see csrc/moe.cu); all on the device."""
    starts: torch.Tensor    # [E + 1] int32 first row of each expert's slab
    counts: torch.Tensor    # [E] int32 rows of each expert
    pair_of: torch.Tensor   # [cap] int32 (token, slot) pair of a row, -1 in padding
    row_of: torch.Tensor    # [T * k] int32 row of a pair
    cap: int                # height of the row buffers
    k: int                  # experts per token

    def __post_init__(self):
        self.experts = self.counts.shape[0]


def _ptr(t):
    return None if t is None else t.data_ptr()


def _launch(name, *args):
    rc = getattr(_LIB, name)(*args)
    if rc != 0:
        raise RuntimeError(f"{name} failed with code {rc}")


def route_topk(logits, k: int, renorm: bool, call=_launch):
    """``(probs, topi, w)`` of a router's logits ``[T, E]``: fp32 softmax, the ``k`` largest of each row and their weights. ``None`` for what the
    kernel does not take (other types and devices, more than 256 experts or 32 chosen ones), and while no ``NativeOps`` has been made."""
    T, E = logits.shape
    if _LIB is None or logits.dtype != torch.bfloat16 or not logits.is_cuda or not logits.is_contiguous() or E > _GROUP_MAX or not 0 < k <= min(E, 32):
        return None
    probs = torch.empty(T, E, dtype=torch.float32, device=logits.device)
    topi = torch.empty(T, k, dtype=torch.int64, device=logits.device)
    w = torch.empty(T, k, dtype=torch.float32, device=logits.device)
    call("mtb200_moe_route", logits.data_ptr(), T, E, k, int(renorm), probs.data_ptr(), topi.data_ptr(), w.data_ptr(), _raw_stream(logits.device.index))
    return probs, topi, w


class NativeOps:
    name = "native"

    def __init__(self, device, ce_chunk: int = 8192, attention: str | None = None):
        self.device = torch.device(device)
        if self.device.type != "cuda":
            raise RuntimeError("NativeOps needs a CUDA device")
        self.lib = load_library()
        self._fn = {name: getattr(self.lib, name) for name in dir(_Sig) if name.startswith("mtb200_") and hasattr(self.lib, name)}
        self._index = self.device.index if self.device.index is not None else torch.cuda.current_device()
        self.ce_chunk = ce_chunk
        self.attention_impl = attention or os.environ.get("MTB200_ATTENTION", "native")
        self.status = torch.zeros(1, dtype=torch.int32, device=self.device)
        # GEMM kernel and splits by size: gemm_plan. The CTA-pair kernel (cta_group::2) with 256 x 256 tiles draws more power: in a step made of long
        # GEMMs, which runs at the 1000 W cap, it lowers the clock of EVERY kernel by 12-16 % and the step gets slower (8B model, 64 000-token
        # minibatches: 9.77 s per step with one CTA, 10.36 with pairs). So a product of more than 1 TFLOP (about 0.8 ms) takes wide tiles, which move
        # less (gemm_plan.wide), or single CTAs. MTB200_GEMM2=0 / 1 forces one kernel for all of them (1: also for the fused gathers).
        self.use_gemm2 = os.environ.get("MTB200_GEMM2") == "1"
        self.pair_max_flops = 0.0 if os.environ.get("MTB200_GEMM2") == "0" else 1e12
        self.launches = 0
        self.profile = [] if os.environ.get("MTB200_PROFILE") else None
        self._scratch = {}
        self._gemm_ws = {}   # stream handle -> arrival counters of split launches
        self._gemm_plans = {}   # sizes of a product, or of a grouped one -> entry point and splits, or mode
        self._epoch = itertools.count(1)   # of the launches that may split
        self._attn_plan_cache = {}
        self._block_specs = {}   # sizes of a block -> its products' plans
        self._pairs = None
        self.sms = torch.cuda.get_device_properties(self._index).multi_processor_count

    # -- plumbing ---------------------------------------------------------------------
    def _st(self):
        return _raw_stream(self._index)   # handle of the device's current torch stream, without a Stream object around it

    def _call(self, name, *args, n=1, tag=None):
        if self.profile is None and not nvtx.ENABLED:
            rc = self._fn[name](*args)
            if rc != 0:
                raise RuntimeError(f"{name} failed with code {rc}")
            self.launches += n
            return
        if self.profile is not None:
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
        if nvtx.ENABLED:
            nvtx.push(tag or name)
        rc = self._fn[name](*args)
        if nvtx.ENABLED:
            nvtx.pop()
        if rc != 0:
            raise RuntimeError(f"{name} failed with code {rc}")
        self.launches += n
        if self.profile is not None:
            e1.record()
            self.profile.append((tag or name, e0, e1))

    def profile_summary(self) -> dict:
        """Device time per op (ms) since profiling was switched on (``MTB200_PROFILE=1``)."""
        torch.cuda.synchronize(self.device)
        out = {}
        for name, e0, e1 in self.profile or []:
            out[name] = out.get(name, 0.0) + e0.elapsed_time(e1)
        self.profile = [] if self.profile is not None else None
        return dict(sorted(out.items(), key=lambda kv: -kv[1]))

    def _buf(self, key, numel, dtype):
        b = self._scratch.get(key)
        if b is None or b.numel() < numel or b.dtype != dtype:
            b = torch.empty(numel, dtype=dtype, device=self.device)
            self._scratch[key] = b
        return b[:numel]

    def _ev(self):
        if self.profile is None:
            return None
        e = torch.cuda.Event(enable_timing=True)
        e.record()
        return e

    def _ev_end(self, name, e0):
        if e0 is not None:
            e1 = torch.cuda.Event(enable_timing=True)
            e1.record()
            self.profile.append((name, e0, e1))

    def check_status(self):
        """Raises if any kernel recorded an expired bounded wait (one host sync)."""
        code = int(self.status.item())
        if code:
            self.status.zero_()
            what = {60: "a token id outside the embedding table", 61: "an attention work item outside the packed batch",
                    62: "a chosen expert outside the model's experts"}.get(
                code, "a device-side bounded wait expired")
            raise RuntimeError(f"{what} (status code {code})")

    # -- GEMM -------------------------------------------------------------------------
    def cta_pairs(self) -> int:
        """CTA pairs the device can run at once; 0 where clusters of two cannot be scheduled, and everything runs on single CTAs."""
        if self._pairs is None:
            self._pairs = self._fn["mtb200_gemm2_pairs"]()
        return self._pairs

    def _split_workspace(self, stream):
        """Arrival counters of a stream's split launches (32 KB). Launches of one stream run one after the other, those of different
        streams may overlap, so each stream has its own (the last eight streams do; dropped ones go back to their stream's
        pool, behind the launches that use them). ``None`` under capture: a graph may be replayed beside anything, so its
        launches never split."""
        if torch.cuda.is_current_stream_capturing():
            return None
        ws = self._gemm_ws.get(stream)
        if ws is None:
            if len(self._gemm_ws) >= 8:
                self._gemm_ws.pop(next(iter(self._gemm_ws), None), None)
            ws = torch.zeros(_SPLIT_COUNTERS, dtype=torch.int64, device=self.device)
            self._gemm_ws[stream] = ws
        return ws

    def _split(self, stream, nbytes):
        """``(counters, epoch, partials)`` of a split launch, or ``None`` where it has to run whole. The partials are scratch of this call:
        taken from the allocator (in powers of two, at most 128 MB) and given back behind the launch, so nothing is held
        between calls, and without memory for them the launch simply does not split."""
        ws = self._split_workspace(stream)
        if ws is None:
            return None
        try:
            part = torch.empty(max(1 << 18, 1 << (nbytes // 4 - 1).bit_length()), dtype=torch.float32, device=self.device)
        except torch.OutOfMemoryError:
            return None
        return ws, next(self._epoch), part

    def _plan_gemm(self, M, N, K, two_cta, ragged=False, act=False):
        """``(entry point, splits, bytes of partials)`` of a product, from its sizes and whether rows of an operand start off 32 bytes. ``act``: with an
        epilogue that only tiles of 256 columns have (activation, statistics)."""
        pairs, one = self.cta_pairs(), True
        wide = narrow = None
        if two_cta if two_cta is not None else self.use_gemm2:
            one = False
        elif two_cta is not None or self.pair_max_flops <= 0:
            pairs = 0
        else:
            narrow = None if act else gemm_plan.narrow(M, N, K, self.sms, pairs, _SPLIT_UNITS, _SPLIT_COUNTERS // 4)
            wide = gemm_plan.wide(M, N, K, ragged, self.sms, pairs, _SPLIT_UNITS, _SPLIT_COUNTERS // 4)
            if 2.0 * M * N * K > self.pair_max_flops:
                pairs = 0
        if narrow:
            tile, splits = narrow
            plan = (f"mtb200_gemm_n{tile}_bf16", splits, -(-M // 128) * -(-N // tile) * splits * 128 * tile * 4)
        elif wide:
            plan = ("mtb200_gemm2_wide_bf16", wide, gemm_plan.partial_bytes(M, N, True, wide))
        else:
            pair, splits = gemm_plan.choose(M, N, K, self.sms, pairs, one, _SPLIT_UNITS, _SPLIT_COUNTERS // 4)
            plan = ("mtb200_gemm2_bf16" if pair else "mtb200_gemm_bf16", splits, gemm_plan.partial_bytes(M, N, pair, splits))
        if len(self._gemm_plans) >= 4096:
            self._gemm_plans.clear()
        self._gemm_plans[(M, N, K, two_cta, ragged, act)] = plan
        return plan

    def product_plan(self, M, N, K, pitches, act=False):
        """``_plan_gemm`` of a product whose operands have these leading dimensions (or-ed)."""
        ragged = pitches & 15 != 0
        return self._gemm_plans.get((M, N, K, None, ragged, act)) or self._plan_gemm(M, N, K, None, ragged, act)

    def gemm(self, a, a_mn, b, b_mn, out, M, N, K, residual=None, bias=None, tag=None, two_cta=None, alpha=1.0, stats=None):
        """out[M,N] = alpha*A*B (+bias) (+residual). ``a_mn``/``b_mn``: operand stored [K, rows].
        ``stats`` [M, ceil(N / 256), 2] fp32 receives the softmax statistics of the (bf16) output rows per 256 columns.
        ``two_cta``: force (True) or forbid (False) the cta_group::2 kernel; default by problem size. Without CTA pairs on the
        device the one-CTA kernel runs in any case."""
        out_f32 = out.dtype == torch.float32
        assert a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16
        assert residual is None or residual.dtype == out.dtype
        ragged, act = (a.stride(0) | b.stride(0)) & 15 != 0, stats is not None
        name, splits, nbytes = self._gemm_plans.get((M, N, K, two_cta, ragged, act)) or self._plan_gemm(M, N, K, two_cta, ragged, act)
        st = self._st()
        split = self._split(st, nbytes) if splits > 1 else None
        ws, epoch, part = split or (None, 0, None)
        self._call(name, a.data_ptr(), a.stride(0), int(a_mn), b.data_ptr(), b.stride(0), int(b_mn),
                   out.data_ptr(), out.stride(0), int(out_f32), _ptr(residual),
                   residual.stride(0) if residual is not None else 0, _ptr(bias), M, N, K, float(alpha), splits if split else 1,
                   _ptr(ws), epoch, _ptr(part), 4 * part.numel() if split else 0, _ptr(stats), self.status.data_ptr(), st,
                   tag=tag or _GEMM_TAGS[bool(a_mn)][bool(b_mn)])
        return out

    # -- embedding --------------------------------------------------------------------
    def embedding(self, weight, ids):
        T, H = ids.shape[0], weight.shape[1]
        out = torch.empty(T, H, dtype=weight.dtype, device=self.device)
        self._call("mtb200_embedding_fwd", weight.data_ptr(), ids.data_ptr(), out.data_ptr(), T, H, weight.shape[0],
                   self.status.data_ptr(), self._st())
        return out

    def embedding_bwd(self, dweight, ids, dx):
        """dweight[ids] += dx, deterministic: one block sums the rows of an id in fp32, in token order. Few tokens are searched for equal ids
        as they are, more are grouped by a stable sort."""
        if ids.shape[0] <= _EMB_SCAN:
            ids = ids.contiguous()
            self._call("mtb200_embedding_bwd_scan", dweight.data_ptr(), ids.data_ptr(), dx.data_ptr(), ids.shape[0], dweight.shape[1],
                       dweight.shape[0], self.status.data_ptr(), self._st())
            return
        sorted_ids, order = torch.sort(ids, stable=True)
        self._call("mtb200_embedding_bwd", dweight.data_ptr(), sorted_ids.data_ptr(), order.data_ptr(), dx.data_ptr(),
                   ids.shape[0], dweight.shape[1], dweight.shape[0], self.status.data_ptr(), self._st())

    def scatter_rows(self, rows, src, vec, T):
        """``(out [T, H], v [T])``: zero but in ``rows``, where they are ``src`` and ``vec`` (fp32)."""
        R, H = src.shape
        out = torch.empty(T, H, dtype=src.dtype, device=self.device)
        v = torch.empty(T, dtype=torch.float32, device=self.device)
        self._call("mtb200_scatter_rows", rows.data_ptr(), src.data_ptr(), out.data_ptr(), vec.data_ptr(), v.data_ptr(), R, H, T,
                   self.status.data_ptr(), self._st(), n=2)
        return out, v

    # -- rmsnorm ----------------------------------------------------------------------
    def rmsnorm(self, x, w, eps):
        T, H = x.shape
        y = torch.empty_like(x)
        rstd = torch.empty(T, dtype=torch.float32, device=self.device)
        self._call("mtb200_rmsnorm_fwd", x.data_ptr(), w.data_ptr(), y.data_ptr(), rstd.data_ptr(), eps, T, H,
                   self.status.data_ptr(), self._st())
        return y, rstd

    def rmsnorm_bwd(self, dy, x, rstd, w, dw_out, add_to=None):
        T, H = x.shape
        dx = torch.empty_like(x)
        blocks = self.lib.mtb200_norm_bwd_blocks(T, H)
        part = self._buf("rms_part", blocks * H, torch.float32)
        self._call("mtb200_rmsnorm_bwd", dy.data_ptr(), x.data_ptr(), rstd.data_ptr(), w.data_ptr(), _ptr(add_to),
                   dx.data_ptr(), part.data_ptr(), dw_out.data_ptr(), T, H, self.status.data_ptr(), self._st(), n=2)
        return dx

    # -- layernorm (Starcoder2) -----------------------------------------------------------
    def layernorm(self, x, w, b, eps):
        """``((x - mean) * rstd) * w + b``; returns ``(y, (mean, rstd))`` with fp32 row statistics."""
        T, H = x.shape
        y = torch.empty_like(x)
        mean = torch.empty(T, dtype=torch.float32, device=self.device)
        rstd = torch.empty(T, dtype=torch.float32, device=self.device)
        self._call("mtb200_layernorm_fwd", x.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), mean.data_ptr(),
                   rstd.data_ptr(), eps, T, H, self.status.data_ptr(), self._st())
        return y, (mean, rstd)

    def layernorm_bwd(self, dy, x, stats, w, dw_out, db_out, add_to=None):
        T, H = x.shape
        dx = torch.empty_like(x)
        blocks = self.lib.mtb200_norm_bwd_blocks(T, H)
        part = self._buf("layernorm_dw", blocks * 2 * H, torch.float32)
        self._call("mtb200_layernorm_bwd", dy.data_ptr(), x.data_ptr(), stats[0].data_ptr(), stats[1].data_ptr(), w.data_ptr(),
                   _ptr(add_to), dx.data_ptr(), part.data_ptr(), dw_out.data_ptr(), db_out.data_ptr(), T, H, self.status.data_ptr(),
                   self._st(), n=2)
        return dx

    # -- linear -----------------------------------------------------------------------
    def linear(self, x, w, bias=None, residual=None, gather=None, alpha=1.0, out=None):
        """``alpha * x @ w.T (+bias) (+residual)``. ``gather = (GatherPlan, stage)`` runs the projection with the all-gather of its parameter
        group fused into the same kernel (symmetric-memory backend only). ``out``: write into this ``[T, N]`` view (rows of a
        larger buffer) instead of a new tensor."""
        T, K = x.shape
        N = w.shape[0]
        if out is None:
            out = torch.empty(T, N, dtype=x.dtype, device=self.device)
        if gather is not None:
            assert residual is None and alpha == 1.0
            ev = self._ev()
            gather[0].launch(self, x, w, bias, out, gather[1])
            self._ev_end("gemm_nt_allgather", ev)
            return out
        return self.gemm(x, False, w, False, out, T, N, K, residual=residual, bias=bias, alpha=alpha)

    def linear_dgrad(self, dy, w, alpha=1.0, out=None):
        T, N = dy.shape
        K = w.shape[1]
        if out is None:
            out = torch.empty(T, K, dtype=dy.dtype, device=self.device)
        return self.gemm(dy, False, w, True, out, T, K, N, alpha=alpha)

    def linear_act(self, x, w, fn="silu", gated=True, bias=None):
        """``(pre, act)`` of ``pre = x @ w.T (+bias)`` in one launch: ``pre`` [T, 2F] = [gate | up] and ``fn(gate) * up`` where the MLP is ``gated``, else
        ``pre`` [T, F] and ``fn(pre)``. A bias only without a gate."""
        T, K = x.shape
        N = w.shape[0]
        F, code = N // 2 if gated else N, _ACT[fn]
        assert x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16
        name, _, _ = self.product_plan(T, N, K, x.stride(0) | K, act=True)
        splits = self.product_plan(T, N, K, x.stride(0) | K)[1]
        # Two launches where one cannot address the weight, and for a product that splits its reduction: 700 x 2048 x 8192 32 us, 43 whole with the
        # activation inside (level at reductions of 4096: 512 x 2048 24.6 and 24.9). No kernel is SiLU alone.
        plain = w.is_contiguous() and K % 8 == 0 and F % 8 == 0
        alone = gated or fn == "gelu_tanh"
        if not plain or (splits > 1 and alone):
            pre = self.linear(x, w, bias)
            return pre, (torch.nn.functional.silu(pre) if not alone else self.swiglu(pre, fn) if gated else self.gelu(pre))
        pre = torch.empty(T, N, dtype=x.dtype, device=self.device)
        act = torch.empty(T, F, dtype=x.dtype, device=self.device)
        self._call("mtb200_gemm_act", x.data_ptr(), x.stride(0), w.data_ptr(), pre.data_ptr(), act.data_ptr(), _ptr(bias), 1 if gated else 2, code,
                   T, F, K, gemm_plan.FORMS[name], self.status.data_ptr(), self._st(), tag="gemm_nt_act")
        return pre, act

    def linear_wgrad(self, dy, x, dw_out, dbias_out=None, alpha=1.0):
        T, N = dy.shape
        K = x.shape[1]
        self.gemm(dy, True, x, True, dw_out, N, K, T, alpha=alpha)
        if dbias_out is not None:
            scratch = self._buf("colsum", 32 * N, torch.float32)
            self._call("mtb200_colsum", dy.data_ptr(), dy.stride(0), dbias_out.data_ptr(), scratch.data_ptr(), T, N,
                       self._st(), n=2)

    # -- rope -------------------------------------------------------------------------
    def rope_(self, qkv, position_ids, inv_freq, n_q_heads, n_kv_heads, head_dim, inverse=False, rot_dim=None):
        if rot_dim is not None and rot_dim != head_dim:
            # A partial rotary embedding (Phi-4-mini) pairs dimension i with i + rot_dim / 2 and leaves the tail of the head
            # alone; the kernel pairs i with i + head_dim / 2. Such models take the PyTorch-op form of the rotation.
            from .torch_ref import TorchOps
            return TorchOps.rope_(self, qkv, position_ids, inv_freq, n_q_heads, n_kv_heads, head_dim, inverse, rot_dim)
        assert position_ids.dtype == torch.int32
        self._call("mtb200_rope", qkv.data_ptr(), position_ids.data_ptr(), inv_freq.data_ptr(), qkv.shape[0],
                   qkv.stride(0), n_q_heads + n_kv_heads, head_dim, int(inverse), self._st())
        return qkv

    # -- per-head RMSNorm of q and k (Qwen3) -----------------------------------------------
    def head_rmsnorm_(self, qkv, wq, wk, eps, n_q_heads, n_kv_heads, head_dim):
        """Normalises every q head (weight ``wq``) and k head (``wk``) of ``qkv`` over ``head_dim``, in place;
        returns the reciprocal RMS per (token, head), ``[T * (n_q + n_kv)]`` fp32."""
        return self.qk_norm_rope_(qkv, wq, wk, eps, n_q_heads, n_kv_heads, head_dim, None, None, keep=False)[1]

    def qk_norm_rope_(self, qkv, wq, wk, eps, n_q_heads, n_kv_heads, head_dim, position_ids, inv_freq, keep=True):
        """``head_rmsnorm_`` and then ``rope_`` (unless ``inv_freq`` is ``None``) in one pass. Returns ``(pre, rstd)``; ``pre``, the
        q|k heads as they came, is only made when ``keep``."""
        T, nh = qkv.shape[0], n_q_heads + n_kv_heads
        assert inv_freq is None or position_ids.dtype == torch.int32
        rstd = torch.empty(T * nh, dtype=torch.float32, device=self.device)
        pre = torch.empty(T, nh * head_dim, dtype=qkv.dtype, device=self.device) if keep else None
        self._call("mtb200_head_rmsnorm_fwd", qkv.data_ptr(), wq.data_ptr(), wk.data_ptr(), _ptr(pre), rstd.data_ptr(),
                   None if inv_freq is None else position_ids.data_ptr(), _ptr(inv_freq), eps, T, qkv.stride(0), n_q_heads, nh,
                   head_dim, self._st())
        return pre, rstd

    def head_rmsnorm_bwd_(self, dqkv, pre, rstd, wq, wk, dwq_out, dwk_out, n_q_heads, n_kv_heads, head_dim):
        """In place on the q and k columns of ``dqkv``: gradient of the normalised heads in, gradient of the projection
        output out. ``pre``: the q|k heads before the norm, ``[T, (n_q + n_kv) * head_dim]``."""
        return self.qk_norm_rope_bwd_(dqkv, pre, rstd, wq, wk, dwq_out, dwk_out, n_q_heads, n_kv_heads, head_dim, None, None)

    def qk_norm_rope_bwd_(self, dqkv, pre, rstd, wq, wk, dwq_out, dwk_out, n_q_heads, n_kv_heads, head_dim, position_ids, inv_freq):
        """The inverse rotation (unless ``inv_freq`` is ``None``) and then ``head_rmsnorm_bwd_`` in one pass."""
        T, nh = dqkv.shape[0], n_q_heads + n_kv_heads
        assert inv_freq is None or position_ids.dtype == torch.int32
        blocks = self.lib.mtb200_head_rmsnorm_bwd_blocks(T, nh)
        part = self._buf("head_rmsnorm_dw", blocks * 2 * head_dim, torch.float32)
        self._call("mtb200_head_rmsnorm_bwd", dqkv.data_ptr(), pre.data_ptr(), rstd.data_ptr(), wq.data_ptr(), wk.data_ptr(),
                   part.data_ptr(), dwq_out.data_ptr(), dwk_out.data_ptr(), None if inv_freq is None else position_ids.data_ptr(),
                   _ptr(inv_freq), T, dqkv.stride(0), pre.stride(0), n_q_heads, nh, head_dim, self._st(), n=2)
        return dqkv

    # -- attention --------------------------------------------------------------------
    def _cached(self, cu_host, what: tuple):
        """What ``_keep`` has kept for this minibatch (its list of sequence starts, as it reads now), or ``None``."""
        hit = self._attn_plan_cache.get((id(cu_host),) + what)
        return hit[2] if hit is not None and hit[0] is cu_host and hit[1] == tuple(cu_host) else None

    def _keep(self, cu_host, what: tuple, value):
        if len(self._attn_plan_cache) > 16:
            self._attn_plan_cache.clear()
        self._attn_plan_cache[(id(cu_host),) + what] = (cu_host, tuple(cu_host), value)
        return value

    def _attn_plan(self, cu_host, block, most_work_last_block: bool):
        """Work table for the attention kernels: one row (seq_start, seq_len, block_start) per
        ``block`` rows of every sequence, most work first (forward: late query blocks see the most
        keys; backward: early key blocks are seen by the most queries). Built once per minibatch
        and reused by every layer."""
        what = (block, most_work_last_block)
        table = self._cached(cu_host, what)
        return self._keep(cu_host, what, self._attn_table(cu_host, block, most_work_last_block)) if table is None else table

    def _plan_attention(self, cu_host, hq, hkv, d):
        """``(entry point, its row_pairs argument, work table)`` of a minibatch's forward. A work item is one 128-row block of a head; or, in
        pairs, a block of two heads of a kv head, or two blocks of a head where heads do not pair up."""
        if attention_plan.forward_in_pairs(attention_plan.blocks_per_sequence(cu_host), hq, hkv, d, self.sms):
            row_pairs = (hq // hkv) % 2
            plan = ("mtb200_attn_fwd", (row_pairs,), self._attn_plan(cu_host, 256 if row_pairs else 128, True))
        else:
            plan = ("mtb200_attn_fwd_one", (), self._attn_plan(cu_host, 128, True))
        return self._keep(cu_host, ("fwd", hq, hkv, d), plan)

    def _plan_attention_bwd(self, cu_host, hq, hkv, d):
        """``(work table, CTAs per key block, bytes of their partials, launched in order)`` of a minibatch's backward."""
        table = self._attn_plan(cu_host, 128, False)
        units = table.shape[0] * hkv   # per unit: 8 counters and, for every CTA that shares it, dK and dV of 128 rows in fp32
        most = 1 if units * 8 > _SPLIT_COUNTERS else min(hq // hkv, _SPLIT_FLOATS // max(1, units * 2 * 128 * d))
        splits = attention_plan.backward_splits(attention_plan.blocks_per_sequence(cu_host), hq, hkv, self.sms, most)
        in_order = attention_plan.backward_in_order(attention_plan.blocks_per_sequence(cu_host), hq, hkv, d, splits)
        return self._keep(cu_host, ("bwd", hq, hkv, d), (table, splits, splits * units * 2 * 128 * d * 4, int(in_order)))

    def _attn_table(self, cu_host, block, most_work_last_block: bool):
        items = []
        for a, b in zip(cu_host[:-1], cu_host[1:]):
            n = b - a
            for s0 in range(0, n, block):
                work = s0 if most_work_last_block else n - s0
                items.append((work, a, n, s0))
        items.sort(key=lambda it: -it[0])
        table = torch.tensor([it[1:] for it in items], dtype=torch.int32)
        if table.numel() > 8192 or torch.cuda.is_current_stream_capturing():
            table = table.pin_memory()   # (the driver stages small copies, which is faster than pinning memory for them)
        return table.to(self.device, non_blocking=True)

    def attention(self, qkv, cu_seqlens, cu_host, max_seqlen, hq, hkv, d, scale=None):
        T = qkv.shape[0]
        scale = d ** -0.5 if scale is None else float(scale)
        if self.attention_impl == "flash_attn" or d not in NATIVE_HEAD_DIMS:
            return self._fa_fwd(qkv, cu_seqlens, max_seqlen, hq, hkv, d, scale)
        out = torch.empty(T, hq * d, dtype=qkv.dtype, device=self.device)
        lse = torch.empty(hq, T, dtype=torch.float32, device=self.device)
        name, tail, plan = self._cached(cu_host, ("fwd", hq, hkv, d)) or self._plan_attention(cu_host, hq, hkv, d)
        self._call(name, qkv.data_ptr(), qkv.stride(0), out.data_ptr(), out.stride(0), lse.data_ptr(),
                   plan.data_ptr(), plan.shape[0], T, hq, hkv, d, *tail, scale, self.status.data_ptr(), self._st(), tag="mtb200_attn_fwd")
        return out, lse

    def attention_bwd(self, dout, qkv, out, lse, cu_seqlens, cu_host, max_seqlen, hq, hkv, d, scale=None):
        T = qkv.shape[0]
        scale = d ** -0.5 if scale is None else float(scale)
        if self.attention_impl == "flash_attn" or d not in NATIVE_HEAD_DIMS:
            return self._fa_bwd(dout, qkv, out, lse, cu_seqlens, max_seqlen, hq, hkv, d, scale)
        dqkv = torch.empty_like(qkv)
        plan, splits, nbytes, in_order = self._cached(cu_host, ("bwd", hq, hkv, d)) or self._plan_attention_bwd(cu_host, hq, hkv, d)
        scratch = torch.empty(hq * T * (d + 1), dtype=torch.float32, device=self.device)   # dQ's accumulator [T, hq * d] and delta [hq, T]: one allocation
        dq_acc = scratch.data_ptr()
        st = self._st()
        split = self._split(st, nbytes) if splits > 1 else None
        ws, epoch, part = split or (None, 0, None)
        self._call("mtb200_attn_bwd", qkv.data_ptr(), qkv.stride(0), out.data_ptr(), out.stride(0), dout.data_ptr(),
                   dout.stride(0), dqkv.data_ptr(), dqkv.stride(0), lse.data_ptr(), dq_acc + 4 * hq * T * d, dq_acc,
                   plan.data_ptr(), plan.shape[0], T, hq, hkv, d, splits if split else 1, _ptr(ws), epoch, _ptr(part), 4 * part.numel() if split else 0, scale,
                   in_order, self.status.data_ptr(), st, n=3)
        return dqkv

    # Library attention (flash-attn 2): selectable for A/B comparisons, and the path of head dimensions the
    # tcgen05 kernels are not built for (Gemma's 256: S plus a 256-column output accumulator would fill tensor memory
    # with no second S buffer to overlap softmax and MMA, so it needs a kernel of its own design).
    def _fa_fwd(self, qkv, cu, max_seqlen, hq, hkv, d, scale):
        from flash_attn.flash_attn_interface import _flash_attn_varlen_forward
        T = qkv.shape[0]
        q = qkv[:, : hq * d].view(T, hq, d)
        k = qkv[:, hq * d: (hq + hkv) * d].view(T, hkv, d)
        v = qkv[:, (hq + hkv) * d:].view(T, hkv, d)
        ev = self._ev()
        out, lse, _, _ = _flash_attn_varlen_forward(q, k, v, cu, cu, max_seqlen, max_seqlen, 0.0, scale, causal=True)
        self._ev_end("flash_attn_fwd", ev)
        return out.reshape(T, hq * d), lse

    def _fa_bwd(self, dout, qkv, out, lse, cu, max_seqlen, hq, hkv, d, scale):
        from flash_attn.flash_attn_interface import _flash_attn_varlen_backward
        T = qkv.shape[0]
        q = qkv[:, : hq * d].view(T, hq, d)
        k = qkv[:, hq * d: (hq + hkv) * d].view(T, hkv, d)
        v = qkv[:, (hq + hkv) * d:].view(T, hkv, d)
        dqkv = torch.empty_like(qkv)
        dq = dqkv[:, : hq * d].view(T, hq, d)
        dk = dqkv[:, hq * d: (hq + hkv) * d].view(T, hkv, d)
        dv = dqkv[:, (hq + hkv) * d:].view(T, hkv, d)
        ev = self._ev()
        _flash_attn_varlen_backward(dout.view(T, hq, d), q, k, v, out.view(T, hq, d), lse, dq, dk, dv, cu, cu,
                                    max_seqlen, max_seqlen, 0.0, scale, True, -1, -1, 0.0, None, False)
        self._ev_end("flash_attn_bwd", ev)
        return dqkv

    # -- a whole decoder block (block_exec.py) ---------------------------------------------
    EMB_SCAN = _EMB_SCAN

    def step_forward_backward(self, eng, batch, grad_scale):
        return step_exec.forward_backward(eng, batch, grad_scale)

    def block_forward(self, acts_type, cfg, p, x, batch, inv_freq, keep, saved_attn, want_attn, need_out):
        return block_exec.forward(self, acts_type, cfg, p, x, batch, inv_freq, keep, saved_attn, want_attn, need_out)

    def block_backward(self, cfg, p, g, acts, dout, batch, inv_freq):
        return block_exec.backward(self, cfg, p, g, acts, dout, batch, inv_freq)

    # -- swiglu -----------------------------------------------------------------------
    def swiglu(self, gate_up, act="silu"):
        """``act(gate) * up`` over ``[gate | up]``: SiLU (SwiGLU) or the tanh-approximated GELU (GeGLU)."""
        T, F2 = gate_up.shape
        out = torch.empty(T, F2 // 2, dtype=gate_up.dtype, device=self.device)
        self._call(_GLU[act] + "_fwd", gate_up.data_ptr(), out.data_ptr(), T, F2 // 2, self._st())
        return out

    def swiglu_bwd(self, dact, gate_up, act="silu"):
        T, F2 = gate_up.shape
        dgu = torch.empty_like(gate_up)
        self._call(_GLU[act] + "_bwd", dact.data_ptr(), gate_up.data_ptr(), dgu.data_ptr(), T, F2 // 2, self._st())
        return dgu

    def swiglu_bwd_act(self, dact, gate_up, act="silu"):
        """Returns ``(dgate_up, act)``; ``act`` (the forward output) is written over ``dact``."""
        T, F2 = gate_up.shape
        dgu = torch.empty_like(gate_up)
        self._call(_GLU[act] + "_bwd_act", dact.data_ptr(), gate_up.data_ptr(), dgu.data_ptr(), T, F2 // 2, self._st())
        return dgu, dact

    # -- mixture of experts: grouped projections over expert slabs ----------------------------
    @staticmethod
    def expert_stack(p: dict, name: str, E: int):
        """``(first matrix, elements between two experts)`` when the matrices ``name0 .. name{E-1}`` of ``p`` sit at equal
        distances in memory, as in a block's flat buffer; ``None`` when one grouped launch cannot address them."""
        ws = [p[f"{name}{e}"] for e in range(E)]
        a = ws[0]
        if E > _GROUP_MAX or any(w.dtype != torch.bfloat16 or not w.is_contiguous() or w.shape != a.shape for w in ws) \
                or a.data_ptr() % 16 or a.shape[0] % 8 or a.shape[1] % 8:
            return None
        step = ws[1].data_ptr() - a.data_ptr() if E > 1 else a.numel() * 2
        if step <= 0 or step % 16 or any(w.data_ptr() - a.data_ptr() != e * step for e, w in enumerate(ws)):
            return None
        return a, step // 2

    def expert_slabs(self, topi, E: int) -> ExpertSlabs:
        """Groups the (token, slot) pairs of ``topi`` [T, k] by expert. No host read: the buffers are sized for the worst case."""
        T, k = topi.shape
        n = T * k
        cap = -(-(n + E * (_GROUP_ALIGN - 1)) // _GROUP_ALIGN) * _GROUP_ALIGN
        buf = torch.empty(2 * E + 1 + cap + n, dtype=torch.int32, device=self.device)
        starts, counts, pair_of, row_of = buf.split([E + 1, E, cap, n])
        topi = topi.contiguous()
        self._call("mtb200_moe_plan", topi.data_ptr(), n, E, cap, starts.data_ptr(), counts.data_ptr(), pair_of.data_ptr(),
                   row_of.data_ptr(), self.status.data_ptr(), self._st())
        return ExpertSlabs(starts, counts, pair_of, row_of, cap, k)

    def gather_rows(self, src, sl: ExpertSlabs, scale: float = 1.0):
        """Rows of ``src`` [T, H] in slab order, zeros between the slabs."""
        H = src.shape[1]
        out = torch.empty(sl.cap, H, dtype=src.dtype, device=self.device)
        self._call("mtb200_moe_gather", src.contiguous().data_ptr(), sl.pair_of.data_ptr(), sl.starts.data_ptr(), sl.experts, sl.k,
                   sl.cap, H, float(scale), out.data_ptr(), self._st())
        return out

    def _plan_grouped(self, key):
        """``mode`` of a grouped product's entry point, with its kernel, from its sizes and whether rows of an operand start off 32 bytes."""
        mode, cap, E, M, N, K, off_a, off_b = key
        rows = cap - (_GROUP_ALIGN - 1) * E   # of all experts, to within a tile
        wide = rows > 0 and self.pair_max_flops > 0 and self.cta_pairs() > 0 and gemm_plan.grouped_wide(
            mode == 2, rows, E, 2.0 * rows * N * (M if mode == 2 else K), K, off_a != 0 or off_b != 0,
            gemm_plan.grouped_ratio(mode == 2, rows, E, M, N, K, off_a != 0, off_b != 0, self.sms, self.cta_pairs()))
        if len(self._gemm_plans) >= 4096:
            self._gemm_plans.clear()
        self._gemm_plans[key] = mode + 4 * wide
        return mode + 4 * wide

    def _grouped(self, mode, a, b, ldb, out, ldd, sl, M, N, K, stride, act=None, fn="silu"):
        lda, cap, E = a.stride(0), sl.cap, sl.experts
        key = (mode, cap, E, M, N, K, lda & 15, ldb & 15)   # asked six times a layer, which the host bounds where experts are small
        form = self._gemm_plans.get(key)
        if form is None:
            form = self._plan_grouped(key)
        self._call("mtb200_gemm_grouped", a.data_ptr(), lda, b.data_ptr(), ldb, out.data_ptr(), ldd, _ptr(act), _ACT[fn], form, cap, M, N, K,
                   sl.starts.data_ptr(), sl.counts.data_ptr(), E, stride, self.status.data_ptr(), self._st(),
                   tag="gemm_grouped_" + ("nt", "nn", "tn", "nt_act")[mode])
        return out

    def grouped_linear(self, x, stack, sl: ExpertSlabs):
        """``x_e @ W_e.T`` for every slab; ``stack``: see ``expert_stack``, matrices ``[N, K]``."""
        w, stride = stack
        N, K = w.shape
        out = torch.empty(sl.cap, N, dtype=x.dtype, device=self.device)
        return self._grouped(0, x, w, K, out, N, sl, sl.cap, N, K, stride)

    def grouped_linear_act(self, x, stack, sl: ExpertSlabs, fn="silu"):
        """``(pre, fn(gate) * up)`` of ``pre = [gate | up] = x_e @ W_e.T`` for every slab, in one launch."""
        w, stride = stack
        N, K = w.shape
        pre = torch.empty(sl.cap, N, dtype=x.dtype, device=self.device)
        act = torch.empty(sl.cap, N // 2, dtype=x.dtype, device=self.device)
        return self._grouped(3, x, w, K, pre, N, sl, sl.cap, N, K, stride, act, fn), act

    def grouped_dgrad(self, dy, stack, sl: ExpertSlabs):
        """``dy_e @ W_e`` for every slab."""
        w, stride = stack
        N, K = w.shape
        out = torch.empty(sl.cap, K, dtype=dy.dtype, device=self.device)
        return self._grouped(1, dy, w, K, out, K, sl, sl.cap, K, N, stride)

    def grouped_wgrad(self, dy, x, stack, sl: ExpertSlabs):
        """``dW_e = dy_e.T @ x_e`` into the stacked gradient matrices; zeros for an expert without rows."""
        g, stride = stack
        N, K = g.shape
        self._grouped(2, dy, x, x.stride(0), g, K, sl, N, K, 0, stride)

    def expert_glu_bwd(self, du, gu, w, sl: ExpertSlabs, act="silu"):
        """``(dgu, weighted activation (over du), dw)`` from ``du``, the gradient of the activation before the expert weight."""
        F = du.shape[1]
        dgu = torch.empty_like(gu)
        dw = torch.zeros_like(w)
        self._call("mtb200_moe_glu_bwd", du.data_ptr(), gu.data_ptr(), w.data_ptr(), sl.pair_of.data_ptr(), sl.starts.data_ptr(),
                   sl.experts, sl.cap, F, int(act != "silu"), dgu.data_ptr(), dw.data_ptr(), self._st())
        return dgu, du, dw

    def combine_rows(self, rows, sl: ExpertSlabs, base, w=None, add=None, scale=1.0):
        """``base + scale * (sum over a token's slots of w * row + add)``, summed in fp32; ``w`` [T, k] and ``add`` [T, H] fp32."""
        T, H = base.shape
        out = torch.empty_like(base)
        self._call("mtb200_moe_combine", rows.data_ptr(), sl.row_of.data_ptr(), _ptr(w), _ptr(add), base.contiguous().data_ptr(), float(scale), T,
                   sl.k, H, out.data_ptr(), self._st())
        return out

    def route_topk(self, logits, k: int, renorm: bool):
        """``(probs, topi, w)`` of router logits in one launch, or ``None``: see ``route_topk`` above."""
        return route_topk(logits, k, renorm, self._call)

    def route_bwd(self, probs, topi, w, dw, renorm: bool, dtype):
        """Gradient of the router logits ``[T, E]``."""
        T, E = probs.shape
        out = torch.empty(T, E, dtype=dtype, device=self.device)
        self._call("mtb200_moe_route_bwd", probs.data_ptr(), topi.data_ptr(), w.data_ptr(), dw.data_ptr(), int(renorm), T, E, topi.shape[1],
                   out.data_ptr(), self._st())
        return out

    # -- plain GELU (tanh approximation) of a not gated MLP ----------------------------------
    def gelu(self, x):
        y = torch.empty_like(x)
        self._call("mtb200_gelu_fwd", x.data_ptr(), y.data_ptr(), x.numel(), self._st())
        return y

    def gelu_bwd(self, dy, x):
        dx = torch.empty_like(x)
        self._call("mtb200_gelu_bwd", dy.data_ptr(), x.data_ptr(), dx.data_ptr(), x.numel(), self._st())
        return dx

    def gelu_bwd_act(self, dy, x):
        """Returns ``(dx, act)``; ``act`` (the forward output) is written over ``dy``."""
        dx = torch.empty_like(x)
        self._call("mtb200_gelu_bwd_act", dy.data_ptr(), x.data_ptr(), dx.data_ptr(), x.numel(), self._st())
        return dx, dy

    # -- fused linear + cross-entropy ---------------------------------------------------
    @staticmethod
    def ce_wants_stats(V: int, H: int) -> bool:
        # The statistics save the cross-entropy a read of the row, which only costs where a row does not stay on the SM, and take the
        # epilogue 3 us per tile, which only hides behind longer reductions. Logits and gradient together, with and without: 3720 x 151936 x 1536 1505
        # and 1777 us, 8000 x 32000 x 2048 899 and 1002, x 1536 744 and 821, but x 1024 702 and 622; 8000 x 512 x 64 50 and 15.
        return V > 16384 and H >= 1536

    def linear_ce(self, x, w, targets, grad_scale, dw_out, accumulate_dw=False, ignore_index=-100, logit_scale=1.0):
        """Per-token CE of ``logit_scale * x @ w.T``. Chunked over tokens (8192 rows): bf16 logits chunk
        by the tcgen05 GEMM (fp32 accumulation, one rounding: what the reference's fused linear-CE holds
        too), whose epilogue also leaves softmax statistics where that pays -> loss and the bf16 gradient written over the logits -> dX
        chunk and dW accumulation, again on the tcgen05 GEMM. Only ``[chunk, V]`` logits ever exist.
        dW is accumulated in fp32 over the chunks and rounded to bf16 once."""
        T, H = x.shape
        V = w.shape[0]
        loss = torch.empty(T, dtype=torch.float32, device=self.device)
        dx = torch.empty_like(x)
        ck = min(self.ce_chunk, T)
        logits = self._buf("ce_logits", ck * V, torch.bfloat16).view(ck, V)
        stats = self._buf("ce_stats", ck * -(-V // 256) * 2, torch.float32) if self.ce_wants_stats(V, H) else None
        # one chunk: its weight gradient is the whole sum, rounded (or added to what is there) in the GEMM's epilogue
        whole = T <= ck and dw_out.is_contiguous()
        dw = dw_out.view(V, H) if whole else None
        dw32 = None if whole else self._buf("ce_dw", V * H, torch.float32).view(V, H)
        first = True
        for a in range(0, T, ck):
            n = min(ck, T - a)
            self.gemm(x[a:a + n], False, w, False, logits, n, V, H, alpha=logit_scale, stats=stats)
            self._call("mtb200_ce_fwd_bwd", logits.data_ptr(), V, 1, _ptr(stats), targets[a:a + n].data_ptr(),
                       loss[a:a + n].data_ptr(), logits.data_ptr(), V, n, V, float(grad_scale), ignore_index, self._st())
            self.gemm(logits, False, w, True, dx[a:a + n], n, H, V, alpha=logit_scale)
            if whole:
                self.gemm(logits, True, x, True, dw, V, H, n, residual=dw if accumulate_dw else None, alpha=logit_scale)
            else:
                self.gemm(logits, True, x[a:a + n], True, dw32, V, H, n, residual=None if first else dw32, alpha=logit_scale)
            first = False
        if not whole:
            self._call("mtb200_f32_to_bf16", dw_out.data_ptr(), dw32.data_ptr(), V * H, int(accumulate_dw), self._st())
        return loss, dx

    # -- optimizer --------------------------------------------------------------------
    def sumsq(self, g):
        out = torch.zeros(1, dtype=torch.float32, device=self.device)
        self._call("mtb200_sumsq", g.data_ptr(), g.numel(), out.data_ptr(), self._st())
        return out

    def add_sumsq(self, g, out):
        """``out += sum(g ** 2)`` (``out``: one fp32 element on the device)."""
        self._call("mtb200_sumsq", g.data_ptr(), g.numel(), out.data_ptr(), self._st())

    @staticmethod
    def group_table(groups):
        """Addresses and sizes of parameter groups ``(master, m, v, gradient, working copy)``, for one call of ``add_sumsq_groups`` or
        ``adamw_groups``."""
        rows = [x for g in groups for x in (*(t.data_ptr() for t in g), g[0].numel())]
        return (c_longlong * len(rows))(*rows), len(groups)

    def add_sumsq_groups(self, table, out):
        """``add_sumsq`` of the gradients of all groups, in one launch."""
        self._call("mtb200_sumsq_groups", *table, out.data_ptr(), self._st())

    def adamw_groups(self, table, fp32_moments, sumsq, max_norm, lr, beta1, beta2, eps, weight_decay, step):
        """``adamw_step`` of all groups in one launch, with the gradients scaled by ``min(1, max_norm / (norm + 1e-6))`` (``max_norm`` 0: as they
        are). Returns the norm, ``sqrt(sumsq)``, 0-dim."""
        norm = torch.empty((), dtype=torch.float32, device=self.device)
        self._call("mtb200_adamw_groups", *table, int(fp32_moments), sumsq.data_ptr(), max_norm, norm.data_ptr(), lr, beta1, beta2, eps, weight_decay,
                   step, self._st())
        return norm

    def accumulate(self, acc, src, accumulate: bool):
        """acc(fp32) = (acc if accumulate else 0) + src (bf16 or fp32)."""
        self._call("mtb200_accumulate", acc.data_ptr(), src.data_ptr(), acc.numel(), int(src.dtype == torch.float32),
                   int(accumulate), self._st())

    def adamw_step(self, master, m, v, grad, param_out, lr, beta1, beta2, eps, weight_decay, step, grad_coef):
        if not torch.is_tensor(grad_coef):
            grad_coef = torch.full((1,), float(grad_coef), dtype=torch.float32, device=self.device)
        grad_coef = grad_coef.reshape(1).float()
        self._call("mtb200_adamw", master.data_ptr(), m.data_ptr(), v.data_ptr(), int(m.dtype == torch.float32),
                   grad.data_ptr(), param_out.data_ptr(), master.numel(), lr, beta1, beta2, eps, weight_decay, step,
                   grad_coef.data_ptr(), self._st())
