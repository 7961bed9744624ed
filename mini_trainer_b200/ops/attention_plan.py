"""Which form of the attention kernels a packed batch runs on, from the lengths of its sequences alone.

A launch is a list of units (CTAs, or pairs of query tiles of a persistent CTA) of known length, dealt to the SMs longest first.
``finish_time`` bounds when the last one is done; the forms and splits are compared by it. The unit times of the forward are measured
on a B200 (microseconds; 630 batches of one to 300 sequences of 16 to 16384 tokens, 1 to 32 heads): over these the choice costs 0.2 % on
average against the better form, always pairs would cost 19 % (at most 90 %), always one tile 14 % (at most 125 %).
"""
from __future__ import annotations

BLOCK = 128   # rows of a query block, keys of a key block

# Forward, per head_dim. one: launch, a CTA, a key tile of it. two: launch; a pair of heads, a key tile of both; a pair of row
# blocks, a key tile of both; a row block without partner, a key tile of it.
_ONE = {64: (1.87, 4.1, 0.84), 128: (1.88, 5.55, 0.94)}
_TWO = {64: (3.98, 2.81, 1.65, 3.4, 1.75, 1.89, 1.61), 128: (3.32, 5.27, 1.72, 4.83, 1.66, 3.47, 1.66)}

# Backward, in iterations (one query block of one head, 1.5 us at head_dim 64 and 2.7 at 128): a CTA's start and end (loads of K and V,
# stores of dK and dV), and what a partial sum of dK and dV adds to it.
_BWD_CTA, _BWD_PARTIAL = 5.0, 2.0


def finish_time(units: list, workers: int) -> float:
    """Lower bound, and in practice about the value, of the finish time of ``units`` [(time, count)] on ``workers``: the longest
    unit, the mean load, and k units on one worker as soon as there are more than (k - 1) * workers of at least that length."""
    units = sorted(units, reverse=True)
    t = max(units[0][0], sum(c * n for c, n in units) / workers)
    seen, k = 0, 2
    for c, n in units:
        seen += n
        while k <= 8 and seen > (k - 1) * workers:
            t = max(t, k * c)
            k += 1
    return t


def blocks_per_sequence(cu_host) -> list:
    return [-(-(b - a) // BLOCK) for a, b in zip(cu_host[:-1], cu_host[1:]) if b > a]


def _with_at_least(blocks: list) -> list:
    """``out[n]``: sequences of at least ``n`` blocks (``out[0]`` unused)."""
    out = [0] * (max(blocks) + 2)
    for b in blocks:
        out[b] += 1
    for n in range(len(out) - 2, 0, -1):
        out[n] += out[n + 1]
    return out


def forward_in_pairs(blocks: list, hq: int, hkv: int, d: int, sms: int) -> bool:
    """Forward: pairs of query tiles (``attention_fwd.cu``) or one tile per CTA (``attention_fwd_one.cu``). A unit with ``n`` key
    tiles exists once per sequence of at least ``n`` blocks."""
    if not blocks:
        return True
    if sum(blocks) * hq <= sms:   # one tile per CTA is done after the longest tile, and pairs take longer over theirs
        return False
    return _forward_in_pairs(blocks, hq, hkv, d, sms)


def _forward_in_pairs(blocks: list, hq: int, hkv: int, d: int, sms: int) -> bool:
    at = _with_at_least(blocks)
    longest = len(at) - 2
    launch, a, b = _ONE[d]
    one = launch + finish_time([(a + b * n, at[n] * hq) for n in range(1, longest + 1)], sms)
    launch, a, b, ra, rb, la, lb = _TWO[d]
    if (hq // hkv) % 2 == 0:
        units = [(a + b * n, at[n] * hq // 2) for n in range(1, longest + 1)]
    else:
        units = [(ra + rb * n, at[n] * hq) for n in range(2, longest + 1, 2)]
        units += [(la + lb * n, (at[n] - at[n + 1]) * hq) for n in range(1, longest + 1, 2) if at[n] > at[n + 1]]
    return launch + finish_time(units, sms) <= one


def backward_splits(blocks: list, hq: int, hkv: int, sms: int, most: int) -> int:
    """Backward: CTAs (at most ``most``) that share the query heads of a key block. A key block of a kv head is one CTA's work; with few
    kv heads and a short batch that leaves SMs idle and the longest CTA decides (5987 tokens, 12/2 heads: 437 -> 137 us with
    the heads divided). But every CTA loads K and V again and adds a partial sum, so short samples are not divided
    (16 of 128 tokens, 32/8 heads of 128: 47 us whole, 86 when divided until there were two CTAs per SM)."""
    group = hq // hkv
    if not blocks or group == 1 or most <= 1:
        return 1
    if sum(blocks) * hq <= sms and most >= group:   # however divided, everything runs at once: the longest CTA decides
        return group if _BWD_PARTIAL < (group - 1) * max(blocks) else 1
    return _backward_splits(blocks, hq, hkv, sms, most)


def _backward_splits(blocks: list, hq: int, hkv: int, sms: int, most: int) -> int:
    at = _with_at_least(blocks)
    longest, group, units = len(at) - 2, hq // hkv, sum(blocks) * hkv
    best, splits = float("inf"), 1
    for s in range(1, min(group, most) + 1):
        if s > 1 and units * (s - 1) >= 2 * sms:   # two CTAs per SM already
            break
        cta = _BWD_CTA + (_BWD_PARTIAL if s > 1 else 0.0)
        t = finish_time([(cta + group / s * n, at[n] * hkv * s) for n in range(1, longest + 1)], sms)
        t = max(t, cta + -(-group // s) * longest)
        if t < best:
            best, splits = t, s
    return splits


# Iterations of a CTA, on average, from which the backward is launched behind its predecessor's end and not under its tail (csrc/attention_bwd.cu). 85 batches at head_dim 128
# (16/4, 32/8, 12/2, 16/16 and 8/1 heads, one to 148 sequences), early over in order, with the forward and with a product in front of it: from 20 on 0.99 to 1.15, 1.03 on
# average (8 of 2048 tokens, 16/4: 675 and 586 us; one of 4096, 32/8: 601 and 569), below 12 0.95 to 1.04, 0.99 (37 of 128, 12/2: 53 and 54), between them
# 0.97 to 1.05. At head_dim 64 early is the faster or level throughout (0.95 to 1.00 in 13 batches).
IN_ORDER_ITERATIONS = 20


def backward_in_order(blocks: list, hq: int, hkv: int, d: int, splits: int) -> bool:
    """Backward: whether CTAs go round the chip in order, or come early to whatever SMs are free."""
    return d == 128 and sum(b * (b + 1) for b in blocks) * (hq // hkv) >= 2 * IN_ORDER_ITERATIONS * splits * sum(blocks) > 0
