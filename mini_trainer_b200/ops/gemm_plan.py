"""Which GEMM kernel a product runs on, and in how many splits of its reduction, from its sizes alone.

Both kernels are persistent: the tiles (128 x 256 on one CTA, 256 x 256 on a CTA pair), times the splits, are dealt to the SMs or pairs in
turn, so a launch takes as many rounds as the busiest worker has items. A pair loads less per product and is faster per k-block, but it
has half as many workers with twice the tile: 4736 x 1024 is one round of 148 tiles on single CTAs and two rounds on 74 pairs (K = 4096:
29 and 47 us). Splitting shortens an item and costs the partial sums. The times below (microseconds) are fitted to about 3000 launches of 320
products on a B200, M 128 to 40000, N 64 to 17920, K 200 to 152000, all three layouts: the choice costs 1 % over the best kernel and split
on average, where pairs for everything of 64 tiles with the earlier split rule cost 6 % (and up to 46 % over the one-CTA kernel of the time before pairs).
"""
from __future__ import annotations

BK = 64
MAX_SPLITS = 16
UNIT_BYTES = 128 * 256 * 4      # partial of 128 rows x 256 columns: one per tile and split of a single CTA, two of a pair
# launch; a k-block, the rest of an item, and the least an item takes (its epilogue); a split launch, a partial
_ONE = (1.7, 0.45, 4.8, 7.0, 4.2, 1.32)
_PAIR = (2.5, 0.33, 5.0, 7.4, 3.9, 1.47)


def partial_bytes(M: int, N: int, pair: bool, splits: int) -> int:
    """Scratch of a split launch."""
    return -(-N // 256) * (2 * -(-M // 256) if pair else -(-M // 128)) * splits * UNIT_BYTES


def _best_split(tiles: int, units: int, kblocks: int, workers: int, max_units: int, t: tuple):
    launch, block, item, least, split, partial = t
    best = launch + -(-tiles // workers) * max(kblocks * block + item, least)
    splits = 1
    for s in range(2, MAX_SPLITS + 1):
        if units * s > max_units or kblocks < 4 * s or tiles * (s - 1) >= 3 * workers:
            break
        c = launch + -(-tiles * s // workers) * max(-(-kblocks // s) * block + item, least) + split + partial * s
        if c < best:
            best, splits = c, s
    return best, splits


def choose(M: int, N: int, K: int, sms: int, pairs: int, one: bool, max_units: int, max_counted: int) -> tuple:
    """``(two_cta, splits)`` for an ``M x N x K`` product. ``pairs``: CTA pairs that may be used (0: none); ``one``: single CTAs may be.
    ``max_units``: partials the scratch may hold, ``max_counted``: 128-row units it has counters for."""
    kblocks, cols = -(-K // BK), -(-N // 256)
    t1, t2 = -(-M // 128) * cols, -(-M // 256) * cols
    best = None
    if one or pairs <= 0:
        best = _best_split(t1, t1, kblocks, sms, max_units if t1 <= max_counted else 0, _ONE) + (False,)
    if pairs > 0:
        p = _best_split(t2, 2 * t2, kblocks, pairs, max_units if 2 * t2 <= max_counted else 0, _PAIR) + (True,)
        if best is None or p[0] < best[0]:
            best = p
    return best[2], best[1]
