"""Host side of the native backend (choice of kernels, workspaces, plans) with stand-ins for the library's launches: no GPU."""
import itertools

import pytest
import torch


def make_ops(**fakes):
    """A ``NativeOps`` on CPU tensors whose library calls are recorded instead of launched."""
    from mini_trainer_b200.ops import native
    ops = object.__new__(native.NativeOps)
    ops.device = torch.device("cpu")
    ops._index, ops.launches, ops.profile = 0, 0, None
    ops.use_gemm2, ops.pair_max_flops, ops.sms = False, 1e12, 148
    ops.status = torch.zeros(1, dtype=torch.int32)
    ops._scratch, ops._gemm_ws, ops._attn_plan_cache, ops._gemm_plans, ops._pairs = {}, {}, {}, {}, None
    ops._epoch = itertools.count(1)
    ops.calls = []
    fakes.setdefault("mtb200_gemm2_pairs", lambda: 74)

    class Fns(dict):
        def __missing__(self, name):
            return lambda *a: ops.calls.append((name, a)) or 0
    ops._fn = Fns(fakes)
    ops._st = lambda: 0
    ops._split_workspace = lambda st: None

    def _call(name, *args, n=1, tag=None):
        assert len(args) == len(getattr(native._Sig, name))
        ops.calls.append((name, args))
    ops._call = _call
    return ops


def gemm(ops, M, N, K, **kw):
    a, b, out = torch.empty(M, K, dtype=torch.bfloat16), torch.empty(N, K, dtype=torch.bfloat16), torch.empty(M, N, dtype=torch.bfloat16)
    ops.gemm(a, False, b, False, out, M, N, K, **kw)
    return ops.calls[-1][0]


@pytest.mark.parametrize("pairs", [0, 74])
def test_gemm_runs_on_single_ctas_where_pairs_cannot_be_scheduled(pairs):
    ops = make_ops(mtb200_gemm2_pairs=lambda: pairs)
    want = "mtb200_gemm2_bf16" if pairs else "mtb200_gemm_bf16"
    assert gemm(ops, 8192, 2048, 2048) == want
    assert gemm(ops, 512, 512, 64, two_cta=True) == want
    assert gemm(ops, 512, 512, 64, two_cta=False) == "mtb200_gemm_bf16"


# (lengths, query heads, kv heads, head_dim, pairs): launches with fewer pairs than SMs, and batches of many units; each of these is
# at least 5 % faster in its form
@pytest.mark.parametrize("lens,hq,hkv,d,pairs", [([2048], 16, 4, 64, False), ([16384], 2, 1, 128, False), ([8192], 4, 4, 64, False), ([64], 32, 8, 64, False),
                                                 ([4000, 5200, 3100, 5900], 1, 1, 64, False), ([1024], 14, 2, 128, False),
                                                 ([300] * 41, 16, 4, 64, True), ([16384], 32, 8, 128, True), ([128] * 100, 32, 8, 128, True),
                                                 ([100] * 300, 28, 4, 64, True), ([2048], 32, 8, 128, True), ([5000] * 4, 9, 3, 128, True)])
def test_attention_forward_form(lens, hq, hkv, d, pairs):
    from mini_trainer_b200.ops import attention_plan as A
    blocks = [-(-n // 128) for n in lens]
    assert A.forward_in_pairs(blocks, hq, hkv, d, 148) == pairs
    # both forms do the same tiles: the choice is asked for every batch, so it has to accept any of them
    assert A.forward_in_pairs([], hq, hkv, d, 148)


def test_attention_finish_time_is_a_lower_bound():
    from mini_trainer_b200.ops.attention_plan import finish_time
    import heapq
    import random
    rng = random.Random(0)
    for _ in range(200):
        units = [(rng.uniform(1, 50), rng.randint(1, 60)) for _ in range(rng.randint(1, 12))]
        load = [0.0] * 37
        for c, n in sorted(units, reverse=True):
            for _ in range(n):
                heapq.heappush(load, heapq.heappop(load) + c)
        t = finish_time(units, 37)
        assert t <= max(load) * (1 + 1e-9) and max(load) <= 2 * t   # a list schedule ends within mean + longest


def test_attention_forward_launches_the_chosen_form():
    ops = make_ops()
    ops.sms, ops.attention_impl = 148, "native"
    ops._attn_table = lambda cu, block, last: torch.zeros(block, 3, dtype=torch.int32)
    for lens, hq, hkv, name, block in (([2048], 16, 4, "mtb200_attn_fwd_one", 128), ([300] * 41, 16, 4, "mtb200_attn_fwd", 128),
                                       ([300] * 41, 27, 3, "mtb200_attn_fwd", 256)):
        cu = [0]
        for n in lens:
            cu.append(cu[-1] + n)
        qkv = torch.empty(cu[-1], (hq + 2 * hkv) * 64, dtype=torch.bfloat16)
        for _ in range(2):   # the second layer finds the choice and the table
            out, lse = ops.attention(qkv, None, cu, max(lens), hq, hkv, 64)
            assert ops.calls[-1][0] == name and ops.calls[-1][1][6] == block
            assert out.shape == (cu[-1], hq * 64) and lse.shape == (hq, cu[-1])


def test_attention_plan_follows_a_list_that_is_filled_again():
    ops = make_ops()
    ops.sms, ops.attention_impl = 148, "native"
    ops._attn_table = lambda cu, block, last: torch.tensor([[a, b - a, 0] for a, b in zip(cu[:-1], cu[1:])], dtype=torch.int32)
    cu, hq, hkv, d = [0, 128, 2048], 16, 4, 64
    qkv, o = torch.empty(2048, 24 * d, dtype=torch.bfloat16), torch.empty(2048, hq * d, dtype=torch.bfloat16)
    for lens in ([128, 1920], [1000, 1048], [2048], [64] * 32):
        cu[:] = [0]
        for n in lens:
            cu.append(cu[-1] + n)
        for _ in range(2):
            ops.attention(qkv, None, cu, max(lens), hq, hkv, d)
            assert ops._cached(cu, ("fwd", hq, hkv, d))[2][:, 1].tolist() == lens
            ops.attention_bwd(o, qkv, o, torch.empty(hq, 2048), None, cu, max(lens), hq, hkv, d)
            assert ops._cached(cu, ("bwd", hq, hkv, d))[0][:, 1].tolist() == lens


# (lengths, query heads, kv heads, range of CTAs per key block): nothing to divide, short samples, short batches, full ones
@pytest.mark.parametrize("lens,hq,hkv,lo,hi", [([2048], 8, 8, 1, 1), ([128] * 16, 32, 8, 1, 1), ([110] * 100, 4, 1, 1, 1), ([16384], 32, 8, 1, 1),
                                               ([1024], 12, 2, 6, 6), ([2048], 14, 2, 7, 7), ([8192], 24, 2, 2, 3), ([4096], 16, 4, 2, 2),
                                               ([900, 1400, 700, 1100, 600, 1300, 1000, 800], 12, 2, 2, 3)])
def test_attention_backward_splits(lens, hq, hkv, lo, hi):
    from mini_trainer_b200.ops import attention_plan as A
    blocks = [-(-n // 128) for n in lens]
    assert lo <= A.backward_splits(blocks, hq, hkv, 148, 64) <= hi
    assert A.backward_splits(blocks, hq, hkv, 148, 1) == 1 and A.backward_splits([], hq, hkv, 148, 64) == 1
    for most in (2, 3):
        assert A.backward_splits(blocks, hq, hkv, 148, most) <= most


# (lengths, query heads, kv heads, CTAs per key block, in order): lengths that are whole blocks and that are not, many short samples, divided heads
@pytest.mark.parametrize("lens,hq,hkv,splits,want", [([4096], 32, 8, 1, True), ([4313], 32, 8, 1, True), ([1024] * 37, 16, 4, 1, False), ([1100] * 37, 16, 4, 1, True),
                                                     ([2048] * 8, 16, 4, 1, True), ([128] * 148, 16, 4, 1, False), ([1500], 12, 2, 6, False), ([4096], 12, 2, 3, True),
                                                     ([3000], 16, 16, 1, False), ([5000], 16, 16, 1, True), ([], 8, 2, 1, False)])
def test_attention_backward_in_order(lens, hq, hkv, splits, want):
    from mini_trainer_b200.ops import attention_plan as A
    blocks = [-(-n // 128) for n in lens]
    assert A.backward_in_order(blocks, hq, hkv, 128, splits) == want and not A.backward_in_order(blocks, hq, hkv, 64, splits)
    mean = sum((b - j) * hq / hkv / splits for b in blocks for j in range(b)) / max(1, sum(blocks))
    assert (mean >= 20) == want
    ops = make_ops()
    ops.attention_impl = "native"
    ops._attn_table = lambda cu, block, last: torch.zeros(sum(-(-(b - a) // block) for a, b in zip(cu[:-1], cu[1:])), 3, dtype=torch.int32)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    if lens:
        plan = ops._plan_attention_bwd(cu, hq, hkv, 128)
        qkv, o = torch.empty(cu[-1], (hq + 2 * hkv) * 128, dtype=torch.bfloat16), torch.empty(cu[-1], hq * 128, dtype=torch.bfloat16)
        ops.attention_bwd(o, qkv, o, torch.empty(hq, cu[-1]), None, cu, max(lens), hq, hkv, 128)
        assert ops.calls[-1][1][23] == plan[3] == int(A.backward_in_order(blocks, hq, hkv, 128, plan[1]))


def test_attention_backward_divides_only_what_the_workspace_holds():
    ops = make_ops()
    ops.sms, ops.attention_impl = 148, "native"
    ops._attn_table = lambda cu, block, last: torch.zeros(sum(-(-(b - a) // block) for a, b in zip(cu[:-1], cu[1:])), 3, dtype=torch.int32)
    ws = torch.zeros(8)
    for lens, have, want in (([1024], True, True), ([1024], False, False), ([110] * 100, True, False), ([2000] * 80, True, False)):
        cu = [0]
        for n in lens:
            cu.append(cu[-1] + n)
        ops._split_workspace = lambda st: ws if have else None
        hq, hkv, d, T = 8, 2, 64, cu[-1]
        qkv, o = torch.empty(T, 12 * d, dtype=torch.bfloat16), torch.empty(T, hq * d, dtype=torch.bfloat16)
        ops.attention_bwd(o, qkv, o, torch.empty(hq, T), None, cu, max(lens), hq, hkv, d)
        args = ops.calls[-1][1]
        splits, units = args[17], args[12] * hkv
        assert (splits > 1) == want and (args[18] is not None) == want and (args[20] is not None) == want
        if want:
            assert units * 8 <= 4096 and splits * units * 2 * 128 * d * 4 <= args[21] <= 128 << 20


# (M, N, K, pair, whole): a round that only single CTAs fill evenly; two rounds where pairs are the faster per k-block; a few tiles with a
# long reduction; one tile; more than 1 TFLOP. Each is at least 5 % faster than on the other kernel or with the other answer to splitting.
@pytest.mark.parametrize("M,N,K,pair,whole", [(4736, 1024, 4096, False, True), (3700, 1280, 5120, False, True), (5987, 17920, 1536, True, True), (8192, 2048, 2048, True, True),
                                              (4096, 2048, 4099, True, True), (128, 256, 4096, None, False), (896, 896, 6000, None, False), (128, 256, 64, None, True),
                                              (3720, 1536, 151936, False, False), (16384, 4096, 14336, False, True)])
def test_gemm_choice(M, N, K, pair, whole):
    ops = make_ops()
    ws = torch.zeros(1)
    ops._split_workspace = lambda st: ws
    a, b, out = (torch.empty(1, dtype=torch.bfloat16).expand(8, 8) for _ in range(3))
    ops.gemm(a, False, b, False, out, M, N, K)
    name, args = ops.calls[-1]
    assert pair is None or (name == "mtb200_gemm2_bf16") == pair
    assert (args[16] == 1) == whole and (args[17] is None) == whole and (args[19] is None) == whole
    assert whole or args[20] >= (1 + (args[16] > 1)) * 128 * 256 * 4
    ops._split_workspace = lambda st: None      # as under capture
    ops.gemm(a, False, b, False, out, M, N, K)
    assert ops.calls[-1][0] == name and ops.calls[-1][1][16] == 1
    for two in (False, True):
        ops.gemm(a, False, b, False, out, M, N, K, two_cta=two)
        assert ops.calls[-1][0] == ("mtb200_gemm2_bf16" if two else "mtb200_gemm_bf16")


def test_gemm_choice_keeps_within_the_workspace():
    from mini_trainer_b200.ops import gemm_plan as G
    import random
    rng = random.Random(1)
    for _ in range(500):
        M, N, K = (int(2 ** rng.uniform(0, 16)) for _ in range(3))
        units, counted = rng.choice([(1024, 1024), (8, 4), (0, 0)])
        for pairs, one in ((0, True), (74, True), (74, False), (0, False)):
            two, s = G.choose(M, N, K, 148, pairs, one, units, counted)
            u = -(-N // 256) * (2 * -(-M // 256) if two else -(-M // 128))
            assert two is False or pairs > 0
            assert two is True or one or pairs == 0
            assert s == 1 or (u <= counted and u * s <= units and 4 * s <= -(-K // 64))


def test_split_launch_runs_whole_without_memory_for_its_partials(monkeypatch):
    ops = make_ops()
    ops._split_workspace = lambda st: torch.zeros(1)
    real, taken = torch.empty, []

    def empty(*shape, **kw):
        if kw.get("dtype") == torch.float32 and len(shape) == 1:
            taken.append(shape[0])
            raise torch.OutOfMemoryError("no memory")
        return real(*shape, **kw)
    monkeypatch.setattr(torch, "empty", empty)
    gemm(ops, 128, 256, 4096)
    assert taken and ops.calls[-1][1][16] == 1 and ops.calls[-1][1][17] is None
    taken.clear()
    gemm(ops, 128, 256, 256)      # nothing to split: nothing asked for
    assert not taken and ops.calls[-1][1][16] == 1


def test_linear_ce_takes_a_flat_weight_gradient():
    """``dw_out`` is written as V x H whatever its shape, in one chunk of tokens as in several."""
    ops = make_ops()
    T, H, V = 24, 64, 512
    x, w, t = torch.empty(T, H, dtype=torch.bfloat16), torch.empty(V, H, dtype=torch.bfloat16), torch.zeros(T, dtype=torch.int64)
    for chunk in (64, 8):
        ops.ce_chunk = chunk
        for dw in (torch.empty(V, H, dtype=torch.bfloat16), torch.empty(V * H, dtype=torch.bfloat16)):
            for acc in (False, True):
                ops.calls.clear()
                ops.linear_ce(x, w, t, 1.0, dw, accumulate_dw=acc)
                name, args = [c for c in ops.calls if c[1][0] == dw.data_ptr() or (len(c[1]) > 6 and c[1][6] == dw.data_ptr())][-1]
                if chunk >= T:
                    assert name.startswith("mtb200_gemm") and args[7] == H and args[12:15] == (V, H, T)
                    assert (args[9] == dw.data_ptr() and args[10] == H) if acc else args[9] is None
                else:
                    assert name == "mtb200_f32_to_bf16" and args[2:4] == (V * H, int(acc))


def test_attention_choices_agree_with_the_full_estimate():
    """What a small batch is answered without the estimate is what the estimate says."""
    from mini_trainer_b200.ops import attention_plan as A
    import random
    rng = random.Random(2)
    for _ in range(400):
        blocks = [rng.randint(1, 6) for _ in range(rng.randint(1, 6))]
        hkv = rng.choice((1, 2, 4))
        hq = hkv * rng.randint(1, 8)
        for sms in (148, 40):
            assert A.backward_splits(blocks, hq, hkv, sms, 64) == A._backward_splits(blocks, hq, hkv, sms, 64)
            for d in (64, 128):
                assert A.forward_in_pairs(blocks, hq, hkv, d, sms) == A._forward_in_pairs(blocks, hq, hkv, d, sms)


# (M, N, K, rows that start off 32 bytes, splits on wide tiles, 0: another kernel): each at least 3 % faster that way in a loop of its own
@pytest.mark.parametrize("M,N,K,ragged,splits", [(16384, 4096, 28672, False, 1), (28672, 4096, 16384, False, 1), (7001, 3072, 12288, False, 1), (5987, 1536, 17920, False, 1),
                                                 (4285, 37920, 3864, True, 1), (2534, 2520, 5768, True, 1), (4090, 14832, 1912, True, 1),
                                                 (5987, 17920, 1536, False, 0), (10324, 1728, 2112, False, 0), (5587, 3328, 7872, False, 0), (2457, 1760, 5264, True, 0), (1384, 3216, 7946, True, 0)])
def test_gemm_wide_tiles_choice(M, N, K, ragged, splits):
    from mini_trainer_b200.ops import gemm_plan as G
    assert G.wide(M, N, K, ragged, 148, 74, 1024, 1024) == splits
    assert G.wide(M, N, K, ragged, 148, 0, 1024, 1024) == 0
    for units, counted in ((1024, 1024), (64, 1024), (1024, 4)):
        s = G.wide(M, N, K, ragged, 148, 74, units, counted)
        u = 2 * -(-M // 256) * -(-N // 256)
        assert s <= 1 or (u <= counted and u * s <= units and 4 * s <= -(-K // 64))
    ops = make_ops()
    ops.use_gemm2 = True        # one kernel for all of them
    assert ops._plan_gemm(M, N, K, None, ragged)[0] == "mtb200_gemm2_bf16"
    ops.use_gemm2, ops.pair_max_flops = False, 0.0
    assert ops._plan_gemm(M, N, K, None, ragged)[0] == "mtb200_gemm_bf16"


@pytest.mark.parametrize("reduce,rows,E,flops,K,ragged,want", [(False, 8192, 8, 1.9e12, 4096, False, True), (True, 8192, 8, 1.9e12, 4096, False, True), (False, 16384, 64, 1.4e11, 2048, False, False),
                                                               (False, 2996, 16, 2.1e11, 2376, True, True), (True, 2996, 16, 2.1e11, 0, True, False), (True, 7936, 16, 1.4e11, 0, True, True),
                                                               (False, 2996, 16, 2.1e11, 712, True, False), (False, 1000, 32, 1e11, 2376, True, False), (False, 1310, 4, 1.5e10, 2456, True, False)])
def test_grouped_products_choice(reduce, rows, E, flops, K, ragged, want):
    from mini_trainer_b200.ops import gemm_plan as G
    assert G.grouped_wide(reduce, rows, E, flops, K, ragged) == want


# (reduce, rows, E, M, N, K, rows of A and of B off 32 bytes, wide): a round of single CTAs and as many of pairs; two rounds and one; many rounds; tiles of which half
# is past the last column; a weight gradient with little more; long ones
@pytest.mark.parametrize("reduce,rows,E,M,N,K,off_a,off_b,want", [(False, 1672, 8, 2688, 1944, 12160, False, True, False), (False, 2576, 16, 4608, 1248, 4088, True, True, False),
                                                                  (False, 4752, 16, 6656, 584, 17760, False, True, False), (False, 1286, 4, 1792, 2888, 18256, False, True, False),
                                                                  (True, 6532, 4, 2456, 768, 0, True, False, False), (False, 3336, 8, 4352, 3704, 5456, False, True, True),
                                                                  (False, 1668, 4, 2176, 3608, 2552, True, True, True), (False, 32016, 16, 34048, 632, 19744, False, True, True),
                                                                  (False, 5508, 4, 6016, 904, 3600, False, True, True), (True, 1668, 4, 7216, 2552, 0, False, True, True),
                                                                  (True, 10376, 8, 8448, 536, 0, False, True, True), (False, 3460, 4, 4096, 3544, 12144, False, True, True),
                                                                  (False, 7176, 8, 8192, 28672, 4096, False, False, True), (True, 7176, 8, 28672, 4096, 0, False, False, True)])
def test_grouped_products_take_wide_tiles_where_their_rounds_come_out_shorter(reduce, rows, E, M, N, K, off_a, off_b, want):
    ops = make_ops()
    cap = rows + 127 * E
    key = (2 if reduce else 1, cap, E, M, N, K, 8 * off_a, 8 * off_b)
    assert ops._plan_grouped(key) == key[0] + 4 * want
    ops._gemm_plans.clear()
    ops._pairs = 0           # no clusters of two CTAs
    assert ops._plan_grouped(key) == key[0]


def test_grouped_product_is_planned_once_per_size(monkeypatch):
    from mini_trainer_b200.ops import gemm_plan, native
    asked = []
    monkeypatch.setattr(gemm_plan, "grouped_wide", lambda reduce, rows, E, flops, K, ragged, ratio: asked.append((reduce, rows, E, flops, K, ragged)) or ragged)
    ops = make_ops()
    i32 = lambda n: torch.zeros(n, dtype=torch.int32)   # noqa: E731
    for _ in range(3):
        sl = native.ExpertSlabs(i32(5), i32(4), None, None, 1024, 2)
        x, w = torch.empty(1024, 64, dtype=torch.bfloat16), torch.empty(96, 64, dtype=torch.bfloat16)
        ops.grouped_linear(x, (w, 96 * 64), sl)
        ops.grouped_linear_act(x, (w, 96 * 64), sl)
        ops.grouped_dgrad(torch.empty(1024, 104, dtype=torch.bfloat16)[:, :96], (w, 96 * 64), sl)   # rows that start off 32 bytes
        ops.grouped_wgrad(torch.empty(1024, 96, dtype=torch.bfloat16), x, (w, 96 * 64), sl)
    assert [a[1][8] for a in ops.calls] == [0, 3, 5, 2] * 3
    rows = 1024 - 4 * 127
    assert asked == [(False, rows, 4, 2.0 * rows * 96 * 64, 64, False)] * 2 + [(False, rows, 4, 2.0 * rows * 64 * 96, 96, True),
                                                                              (True, rows, 4, 2.0 * rows * 64 * 96, 0, False)]
    ops.pair_max_flops = 0.0        # one kernel for all of them
    ops._gemm_plans.clear()
    ops.grouped_dgrad(torch.empty(1024, 104, dtype=torch.bfloat16)[:, :96], (w, 96 * 64), sl)
    assert ops.calls[-1][1][8] == 1


# each at least 10 % faster in this form than in tiles of 256 columns, or (None) in those
@pytest.mark.parametrize("M,N,K,want", [(640, 512, 3072, (64, 3)), (640, 512, 512, (64, 1)), (3072, 512, 640, (128, 1)), (1200, 1024, 768, (128, 1)), (1249, 1296, 616, (128, 1)),
                                        (1262, 3272, 512, None), (4096, 1376, 256, None), (1200, 4096, 768, None), (16384, 4096, 4096, None)])
def test_gemm_narrow_tiles_choice(M, N, K, want):
    from mini_trainer_b200.ops import gemm_plan as G
    assert G.narrow(M, N, K, 148, 74, 1024, 1024) == want
    for units, counted in ((1024, 1024), (8, 1024), (1024, 4)):
        got = G.narrow(M, N, K, 148, 74, units, counted)
        if got is not None:
            tile, s = got
            tiles = -(-M // 128) * -(-N // tile)
            assert tiles * s <= 148 and (s == 1 or (tiles <= counted and tiles * s * tile <= units * 256 and 3 * s <= -(-K // 64)))
    ops = make_ops()
    assert (ops.product_plan(M, N, K, 0)[0] in ("mtb200_gemm_n64_bf16", "mtb200_gemm_n128_bf16")) == (want is not None)
    assert ops.product_plan(M, N, K, 0, act=True)[0] in ("mtb200_gemm_bf16", "mtb200_gemm2_bf16", "mtb200_gemm2_wide_bf16")
    ops.use_gemm2 = True
    assert ops._plan_gemm(M, N, K, None)[0] == "mtb200_gemm2_bf16"


@pytest.mark.parametrize("source", ["attention_fwd", "attention_fwd_one", "attention_bwd"])
def test_attention_kernels_hold_their_rows_in_registers(source, tmp_path):
    """A softmax thread's scores and probabilities: what the compiler spills is stored and read again for every key tile."""
    import re
    import subprocess
    from mini_trainer_b200 import build
    nvcc = build._nvcc()
    if nvcc is None:
        pytest.skip("needs nvcc")
    r = subprocess.run([nvcc, *build.NVCC_FLAGS, "-Xptxas", "-v", "-c", str(build.CSRC / f"{source}.cu"), "-o", str(tmp_path / "x.o")], capture_output=True, text=True, check=True)
    spills = [int(n) for n in re.findall(r"(\d+) bytes spill", r.stdout + r.stderr)]
    assert len(spills) >= 4 and not any(spills)
