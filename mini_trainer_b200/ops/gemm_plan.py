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


# The kernels of a product, numbered as in csrc/entries.h: single CTAs, CTA pairs, pairs with wide tiles, single CTAs with narrow ones.
FORMS = {"mtb200_gemm_bf16": 0, "mtb200_gemm2_bf16": 1, "mtb200_gemm2_wide_bf16": 2, "mtb200_gemm_n64_bf16": 3, "mtb200_gemm_n128_bf16": 4}


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


# Tiles of 128 x 64 and 128 x 128, each on an SM of its own: launch, a k-block, a split launch, a partial. Fitted to 240 and 350 launches of 150 products of
# 64 to 11500 rows and columns. Of 150 products 108 are narrow by this rule, 1.36 times as fast on average, one 8 % slower.
_NARROW = {64: (3.6, 0.256, 2.3, 0.34), 128: (4.0, 0.292, 3.4, 0.63)}


def narrow(M: int, N: int, K: int, sms: int, pairs: int, max_units: int, max_counted: int):
    """``(columns of a tile, splits)`` where narrow tiles are the faster form, else ``None``: a product that has at most one of them per SM."""
    kblocks, rows, best = -(-K // BK), -(-M // 128), None
    for tile, (launch, block, split, partial) in _NARROW.items():
        tiles = rows * -(-N // tile)
        for s in range(1, MAX_SPLITS + 1):
            if tiles * s > sms or (s > 1 and (kblocks < 3 * s or tiles > max_counted or tiles * s * tile > max_units * 256)):
                break
            c = launch + -(-kblocks // s) * block + (split + partial * s if s > 1 else 0.0)
            if best is None or c < best[0]:
                best = (c, tile, s)
    if best is None:
        return None
    t1, t2 = rows * -(-N // 256), -(-M // 256) * -(-N // 256)
    other = _best_split(t1, t1, kblocks, sms, max_units if t1 <= max_counted else 0, _ONE)[0]
    if pairs > 0:
        other = min(other, _best_split(t2, 2 * t2, kblocks, pairs, max_units if 2 * t2 <= max_counted else 0, _PAIR)[0])
    return best[1:] if best[0] < 0.9 * other else None


# Wide tiles (256 x 512 on a CTA pair) move a quarter less from L2 to the SMs than pairs with 256 x 256. Fitted to 180 products of 0.02 to 1.4 TFLOP,
# each in a loop of its own of 0.1 s and more, where the clock is already held down by power: a fixed part (launches overlap), a k-block, the rest
# of an item, a split launch, a partial. Pairs and single CTAs twice: rows that start on 32-byte sectors, and rows that do not (a pitch that is no multiple of 16
# elements), which cost L2 a request more per 128 bytes; there wide tiles are the faster form by 6 % on average (4285 x 37920 x 3864 1213 -> 1016 us),
# elsewhere only where the reduction is long enough to hide a wide tile's ends (7001 x 3072 x 12288 458 -> 431 us, but 4099 x 12288 x 2048 179 -> 187).
_WIDE = (-2.0, 0.85, 4.1, 11.0, 2.9)
_PAIR_LOOP = ((-4.0, 0.445, 1.6, 5.8, 3.6), (-5.8, 0.51, 2.0, 4.6, 3.4))
_ONE_LOOP = ((-6.7, 0.467, 2.1, 10.5, 1.8), (-7.5, 0.69, 1.7, 0.1, 3.1))
WIDE_RAGGED_FLOPS, WIDE_FLOPS, WIDE_K = 3e10, 1e11, 4096
LONG_FLOPS = 1e12


def _loop_cost(tiles: int, kblocks: int, units: int, max_units: int, workers: int, t: tuple, halves: bool) -> tuple:
    fixed, block, item, split, partial = t
    rest = tiles % workers
    tail = 0.5 if halves and 2 * rest <= workers else 1   # a last round that half the pairs have a wide tile for is given out as half tiles
    best, splits = tiles // workers * (kblocks * block + item) + (kblocks * block * tail + item if rest else 0), 1
    for s in range(2, MAX_SPLITS + 1):
        if units * s > max_units or kblocks < 4 * s or tiles * (s - 1) >= 5 * workers:
            break
        c = -(-tiles * s // workers) * (-(-kblocks // s) * block + item) + split + partial * s
        if c < best:
            best, splits = c, s
    return best + fixed, splits


def wide(M: int, N: int, K: int, ragged: bool, sms: int, pairs: int, max_units: int, max_counted: int) -> int:
    """Splits of the product on wide tiles, or 0 where the other kernels are the faster. ``ragged``: rows of an operand do not start on 32 bytes.
    Products of more than ``LONG_FLOPS`` run at the power cap, where what is moved costs clock: there wide tiles give 1300 to 1410 TFLOP/s, pairs 1170 to
    1375 and single CTAs 1180 to 1325 (16384 tokens of an 8B model), and may be estimated up to 10 % above the others: of 28 such products with an estimate between
    1.0 and 1.1 of the best other one (2160 to 64648 rows, 1 to 8 TFLOP, loops of 0.25 s), they were 1.14 times as fast as single CTAs (0.99 to 1.46)."""
    flops, kblocks, rows, cols = 2.0 * M * N * K, -(-K // BK), -(-M // 256), -(-N // 256)
    if pairs <= 0 or not (flops > LONG_FLOPS or flops >= WIDE_FLOPS and K >= WIDE_K or ragged and flops >= WIDE_RAGGED_FLOPS):
        return 0
    units = 2 * rows * cols
    most = max_units if units <= max_counted else 0
    cost, splits = _loop_cost(rows * -(-N // 512), kblocks, units, most, pairs, _WIDE, True)
    other, _ = _loop_cost(rows * cols, kblocks, units, most, pairs, _PAIR_LOOP[ragged], False)
    ones = -(-M // 128) * cols
    other = min(other, _loop_cost(ones, kblocks, ones, max_units if ones <= max_counted else 0, sms, _ONE_LOOP[ragged], False)[0])
    return splits if cost <= other * (1.1 if flops > LONG_FLOPS else 1.0) else 0


# Grouped products, as above: a k-block on single CTAs, in a weight gradient and else, what rows of A and of B that start off 32 bytes add to it, the rest of an item;
# a k-block and the rest of an item on wide tiles. Fitted to 900 products of 160 drawn expert layers of 20 GFLOP and more, each in both forms (root mean square 8 to 12 %).
_GROUPED_ONE, _GROUPED_WIDE = (0.43, 0.46, 0.08, 0.13, 2.2), (0.84, 4.5)


def grouped_ratio(reduce: bool, rows: int, experts: int, M: int, N: int, K: int, off_a: bool, off_b: bool, sms: int, pairs: int) -> float:
    """Estimated time of a grouped product on wide tiles over that on single CTAs. What decides is how many rounds the tiles take, and only the device knows
    how the rows divide: a slab is taken to end anywhere in its last tile, so that the experts have ``rows`` / tile + half a tile each."""
    tall, cols = rows / experts, -(-N // 256)
    kblocks = tall / BK + 0.5 if reduce else -(-K // BK)
    gradient, other, add_a, add_b, item = _GROUPED_ONE
    block = (gradient if reduce else other) + add_a * off_a + add_b * off_b
    wide_block, wide_item = _GROUPED_WIDE
    low, high = (experts * -(-M // t) if reduce else max(experts * (tall / t + 0.5), experts) for t in (128, 256))
    rounds = low * cols / sms
    one = (rounds + 0.5 if rounds >= 6 else -(-rounds // 1)) * (kblocks * block + item)   # (many rounds even out)
    wide = high * -(-N // 512)
    there = high * cols / (2 * wide)   # of the tiles' columns, those that are there
    full, rest = divmod(wide, pairs)
    tail = 0.0 if rest < 0.5 else 0.5 if 2 * rest <= pairs else 1.0   # given out as half tiles
    if wide >= 6 * pairs:
        full, tail = wide / pairs + 0.25, 0.0
    return (full * (kblocks * wide_block * there + wide_item) + (kblocks * wide_block * tail + wide_item if tail else 0.0)) / one


def grouped_wide(reduce: bool, rows: int, experts: int, flops: float, K: int, ragged: bool, ratio: float = 0.0) -> bool:
    """Wide tiles for a grouped product of ``rows`` rows over all experts (``reduce``: a weight gradient), or 128 x 256 tiles on single CTAs. A tile of 256
    rows may find 128 in a slab's last one, so slabs have to be tall. Rows that start off 32 bytes are 1.1 to 1.7 times as fast
    wide (749 tokens x 4 of 16 experts of 2376 x 7528: 414 -> 366, 282 -> 178, 228 -> 180, 550 -> 316 us), others 0.6 to 1.05 unless the launch is long enough
    for the power cap (8 of 4096 x 14336, 4096 tokens x 2: layer 8200 -> 7780 us). But a product that is a round of single CTAs and as many, longer, rounds of
    pairs loses (402 tokens x 4 of 8 experts of 1944 x 6080: 107 -> 142 us, the layer 696 -> 721), so the estimate (``ratio``) may not be far above 1. The
    line is drawn by whole layers, 21 of them with some of their products either way, since their loops are at the power cap and a product's own is not: narrow
    were faster those with a product of 1.17 and more (by 8 to 51 us), wide those whose estimates end at 1.10 (by up to 76 us)."""
    tall = rows / experts
    if ratio > GROUPED_MOST:
        return False
    if flops >= GROUPED_LONG_FLOPS:
        return tall >= 768
    return ragged and flops >= 2e10 and (tall >= 330 if reduce else tall >= 160 and K >= 1024)


GROUPED_MOST = 1.13
GROUPED_LONG_FLOPS = 8e11
