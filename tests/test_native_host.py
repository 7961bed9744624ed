"""Host side of the native backend (choice of kernels, workspaces, plans) with stand-ins for the library's launches: no GPU."""
import pytest
import torch


def make_ops(**fakes):
    """A ``NativeOps`` on CPU tensors whose library calls are recorded instead of launched."""
    from mini_trainer_b200.ops import native
    ops = object.__new__(native.NativeOps)
    ops.device = torch.device("cpu")
    ops._index, ops.launches, ops.profile = 0, 0, None
    ops.use_gemm2, ops.pair_max_flops = False, 1e12
    ops.status = torch.zeros(1, dtype=torch.int32)
    ops._scratch, ops._gemm_ws, ops._attn_plan_cache, ops._pairs = {}, {}, {}, None
    ops.calls = []

    class Fns(dict):
        def __missing__(self, name):
            return lambda *a: ops.calls.append((name, a)) or 0
    ops._fn = Fns(fakes)
    ops._st = lambda: 0
    ops._split_workspace = lambda st: None
    return ops


def gemm(ops, M, N, K, **kw):
    a, b, out = torch.empty(M, K, dtype=torch.bfloat16), torch.empty(N, K, dtype=torch.bfloat16), torch.empty(M, N, dtype=torch.bfloat16)
    ops.gemm(a, False, b, False, out, M, N, K, **kw)
    return ops.calls[-1][0]


@pytest.mark.parametrize("pairs", [0, 74])
def test_gemm_runs_on_single_ctas_where_pairs_cannot_be_scheduled(pairs):
    ops = make_ops(mtb200_gemm2_pairs=lambda: pairs)
    want = "mtb200_gemm2_bf16" if pairs else "mtb200_gemm_bf16"
    assert gemm(ops, 4096, 2048, 64) == want
    assert gemm(ops, 512, 512, 64, two_cta=True) == want
    assert gemm(ops, 512, 512, 64, two_cta=False) == "mtb200_gemm_bf16"
