"""Every sm_100a kernel against a plain PyTorch fp32 reference of the same op."""
import pytest
import torch

from mini_trainer_b200.ops.torch_ref import TorchOps

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from mini_trainer_b200.ops.native import NativeOps
    return NativeOps("cuda:0")


REF = TorchOps()


def rel_err(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / (b.norm() + 1e-12)).item()


def max_err(a, b, rtol=2e-2):
    """Largest elementwise error beyond ``rtol * |reference|``, in units of the reference's RMS value: a
    handful of wrong elements in a large output barely moves the Frobenius norm but shows up here."""
    a, b = a.float(), b.float()
    excess = ((a - b).abs() - rtol * b.abs()).clamp_min(0.0)
    return (excess.max() / (b.pow(2).mean().sqrt() + 1e-12)).item()


def bf(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).bfloat16()


GEMM_SHAPES = [(128, 256, 64), (128, 256, 128), (256, 512, 256), (300, 520, 200), (5, 64, 72), (1000, 1024, 4096),
               (777, 2048, 1000), (4096, 6144, 4096), (129, 264, 8)]


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
def test_gemm_forward_layout(ops, M, N, K):
    torch.manual_seed(M + N + K)
    x, w = bf(M, K), bf(N, K, scale=0.05)
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ops.gemm(x, False, w, False, out, M, N, K)
    ref = x.float() @ w.float().t()
    assert rel_err(out, ref) < 6e-3 and max_err(out, ref) < 5e-2
    ops.check_status()


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
def test_gemm_dgrad_layout(ops, M, N, K):
    # out[M, N] = A[M, K] @ B[K, N]  (B stored [K, N]: MN-major)
    torch.manual_seed(1 + M + N + K)
    a, b = bf(M, K), bf(K, N, scale=0.05)
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ops.gemm(a, False, b, True, out, M, N, K)
    assert rel_err(out, a.float() @ b.float()) < 6e-3 and max_err(out, a.float() @ b.float()) < 5e-2
    ops.check_status()


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
def test_gemm_wgrad_layout(ops, M, N, K):
    # out[M, N] = A[K, M]^T @ B[K, N]  (both MN-major)
    torch.manual_seed(2 + M + N + K)
    if M % 8:
        pytest.skip("leading dimension of an MN-major A must be a multiple of 8")
    a, b = bf(K, M), bf(K, N, scale=0.05)
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ops.gemm(a, True, b, True, out, M, N, K)
    assert rel_err(out, a.float().t() @ b.float()) < 6e-3 and max_err(out, a.float().t() @ b.float()) < 5e-2
    ops.check_status()


def test_gemm_epilogues(ops):
    M, N, K = 384, 776, 320
    x, w, bias, res = bf(M, K), bf(N, K, scale=0.05), bf(N), bf(M, N)
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ops.gemm(x, False, w, False, out, M, N, K, residual=res, bias=bias)
    ref = x.float() @ w.float().t() + bias.float() + res.float()
    assert rel_err(out, ref) < 6e-3
    o32 = torch.empty(M, N, dtype=torch.float32, device="cuda")
    ops.gemm(x, False, w, False, o32, M, N, K)
    assert rel_err(o32, x.float() @ w.float().t()) < 1e-5 + 1e-3
    ops.gemm(x, False, w, False, o32, M, N, K, residual=o32)   # accumulate in place
    assert rel_err(o32, 2 * (x.float() @ w.float().t())) < 2e-3
    # alpha scales the product before bias and residual are added
    ops.gemm(x, False, w, False, out, M, N, K, residual=res, bias=bias, alpha=0.25)
    assert rel_err(out, 0.25 * (x.float() @ w.float().t()) + bias.float() + res.float()) < 6e-3
    ops.check_status()


@pytest.mark.parametrize("two_cta", [False, True])
def test_gemm_strided_views(ops, two_cta):
    """Outputs, residuals and operands that are column or row slices of wider buffers, which is how
    the engine calls the kernel (dx[a:a+n], q/k/v column blocks of the fused qkv activation)."""
    M, N, K = 384, 520, 320
    xw = bf(M, K + 64)
    x = xw[:, 32:32 + K]                       # operand with a leading dimension larger than K
    w = bf(N, K, scale=0.05)
    ref = x.float() @ w.float().t()
    wide = torch.full((M, N + 64), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.gemm(x, False, w, False, wide[:, 32:32 + N], M, N, K, two_cta=two_cta)
    assert rel_err(wide[:, 32:32 + N], ref) < 6e-3 and max_err(wide[:, 32:32 + N], ref) < 5e-2
    assert (wide[:, :32] == 7.0).all() and (wide[:, 32 + N:] == 7.0).all()      # nothing outside the view is touched
    tall = torch.full((M + 100, N), 7.0, dtype=torch.bfloat16, device="cuda")
    rw = bf(M, N + 8)
    ops.gemm(x, False, w, False, tall[50:50 + M], M, N, K, residual=rw[:, 8:], two_cta=two_cta)
    assert rel_err(tall[50:50 + M], ref + rw[:, 8:].float()) < 6e-3
    assert (tall[:50] == 7.0).all() and (tall[50 + M:] == 7.0).all()
    ops.check_status()


def test_linear_ops_match_reference(ops):
    T, K, N = 333, 256, 520
    x, w, b, r = bf(T, K), bf(N, K, scale=0.05), bf(N), bf(T, N)
    assert rel_err(ops.linear(x, w, b, r), REF.linear(x.float(), w.float(), b.float(), r.float())) < 6e-3
    dy = bf(T, N)
    assert rel_err(ops.linear_dgrad(dy, w), dy.float() @ w.float()) < 6e-3
    dw, db = torch.empty_like(w), torch.empty_like(b)
    ops.linear_wgrad(dy, x, dw, db)
    assert rel_err(dw, dy.float().t() @ x.float()) < 6e-3
    assert rel_err(db, dy.float().sum(0)) < 6e-3


@pytest.mark.parametrize("T,H", [(1, 256), (37, 1536), (500, 4096), (64, 8192), (300, 3584)])
def test_rmsnorm(ops, T, H):
    x, w, dy, res = bf(T, H), (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16(), bf(T, H), bf(T, H)
    y, rstd = ops.rmsnorm(x, w, 1e-5)
    yr, rr = REF.rmsnorm(x, w, 1e-5)
    assert rel_err(y, yr) < 4e-3 and rel_err(rstd, rr) < 1e-5
    dw, dwr = torch.empty_like(w), torch.empty(H, dtype=torch.float32, device="cuda")
    dx = ops.rmsnorm_bwd(dy, x, rstd, w, dw, add_to=res)
    dxr = REF.rmsnorm_bwd(dy.float(), x.float(), rr, w.float(), dwr, add_to=res.float())
    assert rel_err(dx, dxr) < 6e-3 and rel_err(dw, dwr) < 1e-2
    dx2 = ops.rmsnorm_bwd(dy, x, rstd, w, dw)
    assert rel_err(dx2, REF.rmsnorm_bwd(dy.float(), x.float(), rr, w.float(), dwr)) < 6e-3


@pytest.mark.parametrize("D,hq,hkv", [(128, 4, 1), (64, 4, 2), (128, 28, 4)])
def test_rope_forward_and_inverse(ops, D, hq, hkv):
    from mini_trainer_b200.models.config import ModelConfig
    T = 257
    cfg = ModelConfig(vocab_size=8, hidden_size=hq * D, intermediate_size=8, num_hidden_layers=1,
                      num_attention_heads=hq, num_key_value_heads=hkv, head_dim=D, rope_theta=5e5)
    inv = cfg.rope_inv_freq().cuda()
    pos = torch.randint(0, 60000, (T,), device="cuda", dtype=torch.int32)
    qkv = bf(T, (hq + 2 * hkv) * D)
    orig = qkv.clone()
    ref = REF.rope_(qkv.float().clone(), pos, inv, hq, hkv, D)
    ops.rope_(qkv, pos, inv, hq, hkv, D)
    assert rel_err(qkv, ref) < 4e-3
    assert torch.equal(qkv[:, (hq + hkv) * D:], orig[:, (hq + hkv) * D:])  # v untouched
    ops.rope_(qkv, pos, inv, hq, hkv, D, inverse=True)
    assert rel_err(qkv, orig) < 8e-3


@pytest.mark.parametrize("T,H", [(77, 512), (33, 3072), (9, 6144), (130, 200)])
def test_layernorm_forward_and_backward(ops, T, H):
    """LayerNorm with bias (Starcoder2): statistics, output, input gradient (+ residual gradient), weight and bias
    gradients; partial sums without atomics (run twice: bitwise equal)."""
    x, dy, res = bf(T, H, scale=2.0) + 0.5, bf(T, H), bf(T, H)
    w, b = (1.0 + 0.3 * torch.randn(H, device="cuda")).bfloat16(), (0.3 * torch.randn(H, device="cuda")).bfloat16()
    y, stats = ops.layernorm(x, w, b, 1e-5)
    y_ref, stats_ref = REF.layernorm(x.float(), w.float(), b.float(), 1e-5)
    assert rel_err(y, y_ref) < 4e-3 and max_err(y, y_ref) < 5e-2
    assert rel_err(stats[0], stats_ref[0]) < 1e-4 and rel_err(stats[1], stats_ref[1]) < 1e-4
    gw_ref, gb_ref = torch.empty(H, device="cuda"), torch.empty(H, device="cuda")
    dx_ref = REF.layernorm_bwd(dy.float(), x.float(), stats_ref, w.float(), gw_ref, gb_ref, add_to=res.float())
    outs = []
    for _ in range(2):
        gw, gb = torch.empty(H, dtype=torch.bfloat16, device="cuda"), torch.empty(H, dtype=torch.bfloat16, device="cuda")
        dx = ops.layernorm_bwd(dy, x, stats, w, gw, gb, add_to=res)
        outs.append((dx, gw, gb))
    dx, gw, gb = outs[0]
    assert rel_err(dx, dx_ref) < 5e-3 and max_err(dx, dx_ref) < 5e-2
    assert rel_err(gw, gw_ref) < 6e-3 and rel_err(gb, gb_ref) < 6e-3
    assert all(torch.equal(a, c) for a, c in zip(outs[0], outs[1]))
    ops.check_status()


def test_geglu_and_gelu(ops):
    """The tanh-approximated GELU as the gate of a gated MLP (Gemma) and as a plain activation (Starcoder2)."""
    T, F = 123, 688
    gu, da = bf(T, 2 * F), bf(T, F)
    assert rel_err(ops.swiglu(gu, "gelu_tanh"), REF.swiglu(gu.float(), "gelu_tanh")) < 4e-3
    assert rel_err(ops.swiglu_bwd(da, gu, "gelu_tanh"), REF.swiglu_bwd(da.float(), gu.float(), "gelu_tanh")) < 5e-3
    assert max_err(ops.swiglu_bwd(da, gu, "gelu_tanh"), REF.swiglu_bwd(da.float(), gu.float(), "gelu_tanh")) < 5e-2
    act_ref, dgu_ref = ops.swiglu(gu, "gelu_tanh"), ops.swiglu_bwd(da, gu, "gelu_tanh")
    buf = da.clone()
    dgu, act = ops.swiglu_bwd_act(buf, gu, "gelu_tanh")
    assert act.data_ptr() == buf.data_ptr() and torch.equal(act, act_ref) and torch.equal(dgu, dgu_ref)
    x, dy = bf(T, F, scale=2.0), bf(T, F)
    assert rel_err(ops.gelu(x), REF.gelu(x.float())) < 4e-3 and max_err(ops.gelu(x), REF.gelu(x.float())) < 5e-2
    assert rel_err(ops.gelu_bwd(dy, x), REF.gelu_bwd(dy.float(), x.float())) < 5e-3
    ops.check_status()


@pytest.mark.parametrize("D,hq,hkv,T", [(128, 4, 1, 257), (64, 4, 2, 33), (256, 2, 1, 100), (128, 28, 4, 1031)])
def test_head_rmsnorm_forward_and_backward(ops, D, hq, hkv, T):
    """Per-head RMSNorm of the q and k heads inside the fused qkv rows (Qwen3), in place, v untouched; backward in place
    on the gradient with the pre-norm heads as input, weight gradients without atomics (run twice: bitwise equal)."""
    nh = hq + hkv
    qkv = bf(T, (hq + 2 * hkv) * D)
    wq, wk = (1.0 + 0.3 * torch.randn(D, device="cuda")).bfloat16(), (1.0 + 0.3 * torch.randn(D, device="cuda")).bfloat16()
    orig = qkv.clone()
    pre = qkv[:, : nh * D].clone()
    ref = qkv.float().clone()
    rstd_ref = REF.head_rmsnorm_(ref, wq.float(), wk.float(), 1e-6, hq, hkv, D)
    rstd = ops.head_rmsnorm_(qkv, wq, wk, 1e-6, hq, hkv, D)
    assert rel_err(qkv, ref) < 4e-3 and max_err(qkv, ref) < 5e-2 and rel_err(rstd, rstd_ref) < 1e-5
    assert torch.equal(qkv[:, nh * D:], orig[:, nh * D:])
    dy = bf(T, (hq + 2 * hkv) * D)
    dref = dy.float().clone()
    gq_ref, gk_ref = torch.empty(D, device="cuda"), torch.empty(D, device="cuda")
    REF.head_rmsnorm_bwd_(dref, pre.float(), rstd_ref, wq.float(), wk.float(), gq_ref, gk_ref, hq, hkv, D)
    outs = []
    for _ in range(2):
        d = dy.clone()
        gq, gk = torch.empty(D, dtype=torch.bfloat16, device="cuda"), torch.empty(D, dtype=torch.bfloat16, device="cuda")
        ops.head_rmsnorm_bwd_(d, pre, rstd, wq, wk, gq, gk, hq, hkv, D)
        outs.append((d, gq, gk))
    d, gq, gk = outs[0]
    assert rel_err(d, dref) < 5e-3 and max_err(d, dref) < 5e-2
    assert torch.equal(d[:, nh * D:], dy[:, nh * D:])
    assert rel_err(gq, gq_ref) < 6e-3 and rel_err(gk, gk_ref) < 6e-3
    assert all(torch.equal(a, b) for a, b in zip(outs[0], outs[1]))
    ops.check_status()


def test_swiglu(ops):
    T, F = 123, 688
    gu, da = bf(T, 2 * F), bf(T, F)
    assert rel_err(ops.swiglu(gu), REF.swiglu(gu.float())) < 4e-3
    assert rel_err(ops.swiglu_bwd(da, gu), REF.swiglu_bwd(da.float(), gu.float())) < 5e-3
    # fused form: the gradient and the forward output (written over the incoming gradient) in one pass
    act_ref, dgu_ref = ops.swiglu(gu), ops.swiglu_bwd(da, gu)
    buf = da.clone()
    dgu, act = ops.swiglu_bwd_act(buf, gu)
    assert act.data_ptr() == buf.data_ptr() and torch.equal(act, act_ref) and torch.equal(dgu, dgu_ref)


def test_embedding(ops):
    V, H, T = 1000, 256, 4000
    w = bf(V, H)
    ids = torch.randint(0, 50, (T,), device="cuda")  # many collisions
    assert torch.equal(ops.embedding(w, ids), w[ids])
    dx = bf(T, H, scale=0.01)
    base = bf(V, H, scale=0.01)   # what the buffer already holds (the LM-head gradient when embeddings are tied)
    dw = base.clone()
    ops.embedding_bwd(dw, ids, dx)
    ref = base.float().index_add_(0, ids, dx.float())
    assert rel_err(dw, ref) < 3e-3  # fp32 sum of ~80 addends per row, one bf16 rounding
    assert torch.equal(dw[50:], base[50:])   # rows of ids that do not occur are untouched
    dw2 = base.clone()
    ops.embedding_bwd(dw2, ids, dx)
    assert torch.equal(dw, dw2)   # no atomics: bitwise reproducible


@pytest.mark.parametrize("T,H,V", [(300, 256, 32000), (70, 512, 4104)])
def test_linear_ce(ops, T, H, V):
    torch.manual_seed(0)
    x, w = bf(T, H), bf(V, H, scale=0.05)
    tg = torch.randint(0, V, (T,), device="cuda")
    tg[::3] = -100
    dw, dwr = torch.zeros(V, H, dtype=torch.bfloat16, device="cuda"), torch.zeros(V, H, device="cuda")
    ops.ce_chunk = 128
    loss, dx = ops.linear_ce(x, w, tg, 0.01, dw)
    ref = TorchOps(ce_chunk=128)
    lr, dxr = ref.linear_ce(x.float(), w.float(), tg, 0.01, dwr)
    assert rel_err(loss, lr) < 1e-3
    assert (loss[::3] == 0).all()
    assert rel_err(dx, dxr) < 1e-2 and rel_err(dw, dwr) < 1e-2
    dw2 = dw.clone()
    ops.linear_ce(x, w, tg, 0.01, dw2, accumulate_dw=True)
    assert rel_err(dw2, 2 * dwr) < 1e-2


def test_optimizer_kernels(ops):
    n = 128 * 1000
    for sdt in (torch.float32, torch.bfloat16):
        master = torch.randn(n, device="cuda")
        m, v = torch.randn(n, device="cuda").mul(0.01).to(sdt), torch.rand(n, device="cuda").mul(0.001).to(sdt)
        g = torch.randn(n, device="cuda")
        p = torch.empty(n, dtype=torch.bfloat16, device="cuda")
        rm, rmm, rv, rp = master.clone(), m.clone(), v.clone(), torch.empty(n, device="cuda")
        coef = torch.tensor(0.5, device="cuda")
        ops.adamw_step(master, m, v, g, p, 1e-3, 0.9, 0.95, 1e-8, 0.01, 3, coef)
        REF.adamw_step(rm, rmm, rv, g, rp, 1e-3, 0.9, 0.95, 1e-8, 0.01, 3, coef)
        assert rel_err(master, rm) < 1e-5 and rel_err(m, rmm) < 1e-2 and rel_err(v, rv) < 1e-2
        assert torch.equal(p, master.bfloat16())
    g = torch.randn(n, device="cuda")
    assert abs(ops.sumsq(g).item() - g.pow(2).sum().item()) < 1e-3 * n
    acc, src = torch.randn(n, device="cuda"), bf(n)
    ref = acc + src.float()
    ops.accumulate(acc, src, True)
    assert torch.allclose(acc, ref)
    ops.accumulate(acc, src, False)
    assert torch.equal(acc, src.float())


ATTN_CASES = [(128, 4, 1, [300, 17, 129, 1, 640]), (64, 4, 2, [128, 256, 5]), (128, 8, 2, [1000]), (128, 4, 4, [127, 128, 129]),
              # the GQA ratios of the benchmark models (1.5B: 6, 7B: 7, 70B: 8) and sequences of many key tiles
              (128, 6, 1, [4097, 200]), (128, 7, 1, [513, 2050]), (128, 8, 1, [3000])]


def _cu(lens):
    cu_host = [0]
    for n in lens:
        cu_host.append(cu_host[-1] + n)
    return cu_host, torch.tensor(cu_host, dtype=torch.int32, device="cuda")


def _attn_ref_one_head(q, k, v, do=None):
    """fp32 causal attention of ONE head of ONE sequence in query chunks: (out, lse[, dq, dk, dv])."""
    n, d = q.shape
    scale = d ** -0.5
    out = torch.empty_like(q)
    lse = torch.empty(n, device=q.device)
    dq = torch.zeros_like(q) if do is not None else None
    dk = torch.zeros_like(k) if do is not None else None
    dv = torch.zeros_like(v) if do is not None else None
    for a in range(0, n, 2048):
        b = min(n, a + 2048)
        s = (q[a:b] @ k[:b].t()) * scale
        s = s.masked_fill(torch.arange(b, device=q.device)[None, :] > torch.arange(a, b, device=q.device)[:, None], float("-inf"))
        l = torch.logsumexp(s, -1)
        p = torch.exp(s - l[:, None])
        out[a:b] = p @ v[:b]
        lse[a:b] = l
        if do is not None:
            dp = do[a:b] @ v[:b].t()
            delta = (do[a:b] * out[a:b]).sum(-1, keepdim=True)
            ds = p * (dp - delta) * scale
            dq[a:b] = ds @ k[:b]
            dk[:b] += ds.t() @ q[a:b]
            dv[:b] += p.t() @ do[a:b]
    return out, lse, dq, dk, dv


@pytest.mark.parametrize("n,hq,hkv", [(16384, 8, 1), (65536, 2, 1)])
def test_attention_long_sequences(ops, n, hq, hkv):
    """Sequences as long as the benchmark's (hundreds of key tiles per query block: the S/P double
    buffers and the rescale path run many times) against an fp32 reference computed head by head."""
    D = 128
    torch.manual_seed(n)
    qkv = bf(n, (hq + 2 * hkv) * D)
    dout = bf(n, hq * D)
    cu_host, cu = _cu([n])
    out, lse = ops.attention(qkv, cu, cu_host, n, hq, hkv, D)
    out2, lse2 = ops.attention(qkv, cu, cu_host, n, hq, hkv, D)
    assert torch.equal(out, out2) and torch.equal(lse, lse2)          # forward has no order-dependent accumulation
    dqkv = ops.attention_bwd(dout, qkv, out, lse, cu, cu_host, n, hq, hkv, D)
    ops.check_status()
    g = hq // hkv
    for h in (0, hq - 1):
        hk = h // g
        q = qkv[:, h * D:(h + 1) * D].float()
        k = qkv[:, (hq + hk) * D:(hq + hk + 1) * D].float()
        v = qkv[:, (hq + hkv + hk) * D:(hq + hkv + hk + 1) * D].float()
        ro, rl, rdq, _, _ = _attn_ref_one_head(q, k, v, dout[:, h * D:(h + 1) * D].float())
        assert rel_err(out[:, h * D:(h + 1) * D], ro) < 1e-2 and max_err(out[:, h * D:(h + 1) * D], ro) < 0.1
        assert (lse[h] - rl).abs().max() < 2e-2
        assert rel_err(dqkv[:, h * D:(h + 1) * D], rdq) < 2e-2
    # dK / dV of kv head 0 sum over its whole query-head group
    rdk = torch.zeros(n, D, device="cuda")
    rdv = torch.zeros(n, D, device="cuda")
    k = qkv[:, hq * D:(hq + 1) * D].float()
    v = qkv[:, (hq + hkv) * D:(hq + hkv + 1) * D].float()
    for h in range(g):
        _, _, _, dk, dv = _attn_ref_one_head(qkv[:, h * D:(h + 1) * D].float(), k, v, dout[:, h * D:(h + 1) * D].float())
        rdk += dk
        rdv += dv
    assert rel_err(dqkv[:, hq * D:(hq + 1) * D], rdk) < 2e-2 and rel_err(dqkv[:, (hq + hkv) * D:(hq + hkv + 1) * D], rdv) < 2e-2


@pytest.mark.parametrize("D,hq,hkv,lens", ATTN_CASES)
def test_attention_forward(ops, D, hq, hkv, lens):
    torch.manual_seed(sum(lens))
    T = sum(lens)
    qkv = bf(T, (hq + 2 * hkv) * D)
    cu_host = [0]
    for n in lens:
        cu_host.append(cu_host[-1] + n)
    cu = torch.tensor(cu_host, dtype=torch.int32, device="cuda")
    out, lse = ops.attention(qkv, cu, cu_host, max(lens), hq, hkv, D)
    ro, rl = REF.attention(qkv.float(), cu, cu_host, max(lens), hq, hkv, D)
    ops.check_status()
    assert rel_err(lse, rl) < 2e-3 and (lse - rl).abs().max() < 2e-2
    assert rel_err(out, ro) < 1e-2 and max_err(out, ro) < 0.1
    out2, lse2 = ops.attention(qkv, cu, cu_host, max(lens), hq, hkv, D)
    assert torch.equal(out, out2) and torch.equal(lse, lse2)   # run twice: bitwise identical


@pytest.mark.parametrize("D,hq,hkv,lens", ATTN_CASES)
def test_attention_backward(ops, D, hq, hkv, lens):
    if not hasattr(ops.lib, "mtb200_attn_bwd"):
        pytest.skip("attention backward kernel not built")
    torch.manual_seed(1 + sum(lens))
    T = sum(lens)
    qkv = bf(T, (hq + 2 * hkv) * D)
    dout = bf(T, hq * D)
    cu_host = [0]
    for n in lens:
        cu_host.append(cu_host[-1] + n)
    cu = torch.tensor(cu_host, dtype=torch.int32, device="cuda")
    out, lse = ops.attention(qkv, cu, cu_host, max(lens), hq, hkv, D)
    dqkv = ops.attention_bwd(dout, qkv, out, lse, cu, cu_host, max(lens), hq, hkv, D)
    ro, rl = REF.attention(qkv.float(), cu, cu_host, max(lens), hq, hkv, D)
    rd = REF.attention_bwd(dout.float(), qkv.float(), ro, rl, cu, cu_host, max(lens), hq, hkv, D)
    ops.check_status()
    q_end, k_end = hq * D, (hq + hkv) * D
    assert rel_err(dqkv[:, :q_end], rd[:, :q_end]) < 2e-2 and max_err(dqkv[:, :q_end], rd[:, :q_end]) < 0.25
    assert rel_err(dqkv[:, q_end:k_end], rd[:, q_end:k_end]) < 2e-2 and max_err(dqkv[:, q_end:k_end], rd[:, q_end:k_end]) < 0.25
    assert rel_err(dqkv[:, k_end:], rd[:, k_end:]) < 2e-2 and max_err(dqkv[:, k_end:], rd[:, k_end:]) < 0.25


def test_bounded_wait_expires_with_status_and_context_stays_usable(ops):
    """A wait on a flag that nothing sets must run out, record {code, peer} and return."""
    import ctypes
    lib = ops.lib
    fn = lib.mtb200_symm_wait
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_uint, ctypes.c_uint, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    flags = torch.zeros(16, dtype=torch.int32, device="cuda")
    flags[0] = 5                                   # "peer 0" already signalled epoch 5, "peer 1" never does
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = fn(flags.data_ptr(), 2, 5, 2000, 42, status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    code = int(status.item())
    assert code & 0xff == 42 and code >> 8 == 1
    x = torch.ones(1024, device="cuda")
    assert x.sum().item() == 1024                  # the context is still healthy


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (512, 512, 256), (300, 520, 200), (1000, 1024, 4096), (4096, 6144, 4096), (264, 264, 72)])
@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
def test_gemm_two_cta(ops, M, N, K, layout):
    """cta_group::2 kernel (256x256 tiles per CTA pair) against the fp32 reference, all three layouts."""
    torch.manual_seed(3 + M + N + K)
    if layout == "tn" and M % 8:
        pytest.skip("leading dimension of an MN-major A must be a multiple of 8")
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    if layout == "nt":
        a, b = bf(M, K), bf(N, K, scale=0.05)
        ref = a.float() @ b.float().t()
        ops.gemm(a, False, b, False, out, M, N, K, two_cta=True)
    elif layout == "nn":
        a, b = bf(M, K), bf(K, N, scale=0.05)
        ref = a.float() @ b.float()
        ops.gemm(a, False, b, True, out, M, N, K, two_cta=True)
    else:
        a, b = bf(K, M), bf(K, N, scale=0.05)
        ref = a.float().t() @ b.float()
        ops.gemm(a, True, b, True, out, M, N, K, two_cta=True)
    torch.cuda.synchronize()
    ops.check_status()
    assert rel_err(out, ref) < 6e-3
    res, bias = bf(M, N), bf(N)
    if layout == "nt":
        ops.gemm(a, False, b, False, out, M, N, K, residual=res, bias=bias, two_cta=True)
        assert rel_err(out, ref + res.float() + bias.float()) < 6e-3
    # fp32 output accumulated in place (the form the linear+CE weight gradient uses), scaled product
    o32 = torch.zeros(M, N, dtype=torch.float32, device="cuda")
    for _ in range(2):
        ops.gemm(a, layout == "tn", b, layout != "nt", o32, M, N, K, residual=o32, two_cta=True, alpha=0.5)
    assert rel_err(o32, ref) < 2e-3 and max_err(o32, ref) < 2e-2
    ops.check_status()


def test_osft_projection_on_tcgen05_gemm(ops):
    """G - U(U^T G) and G - (G V^T) V on the tcgen05 GEMM against float64 PyTorch."""
    from mini_trainer_b200.parallel import osft as O
    torch.manual_seed(0)
    w = torch.randn(512, 1024, device="cuda", dtype=torch.float64)
    u_hi, s_hi, v_hi, u_lo, s_lo, v_lo = O.svd_split(w, 0.5)
    du = torch.randn(512, u_lo.shape[1], device="cuda", dtype=torch.float64)
    dv = torch.randn(v_lo.shape[0], 1024, device="cuda", dtype=torch.float64)
    ref_u, ref_v = O.project_orthogonal(du, dv, u_hi, v_hi)
    got_u, got_v = O.project_orthogonal_tcgen05(ops, du.float(), dv.float(), u_hi.float(), v_hi.float())
    ops.check_status()
    assert rel_err(got_u, ref_u) < 1e-2 and rel_err(got_v, ref_v) < 1e-2
    # what is left inside the frozen subspace is at bf16 rounding level
    assert (u_hi.float().t() @ got_u).norm() < 2e-2 * du.float().norm()
    assert (got_v @ v_hi.float().t()).norm() < 2e-2 * dv.float().norm()


def test_out_of_range_inputs_are_reported_not_dereferenced(ops):
    """Bounds checks that record a status code and skip the access: a token id outside the embedding
    table, an attention work item outside the packed batch. The context stays usable."""
    w = bf(100, 64)
    ids = torch.tensor([3, 100, 7, -1], device="cuda")
    out = ops.embedding(w, ids)
    torch.cuda.synchronize()
    assert torch.equal(out[0], w[3]) and torch.equal(out[2], w[7]) and (out[1] == 0).all() and (out[3] == 0).all()
    with pytest.raises(RuntimeError, match="token id outside"):
        ops.check_status()
    dw = torch.zeros(100, 64, dtype=torch.bfloat16, device="cuda")
    ops.embedding_bwd(dw, ids, bf(4, 64))
    with pytest.raises(RuntimeError, match="token id outside"):
        ops.check_status()
    assert dw[3].abs().sum() > 0 and dw[7].abs().sum() > 0
    # an attention plan that claims a sequence longer than the batch
    T, hq, hkv, D = 256, 2, 1, 128
    qkv = bf(T, (hq + 2 * hkv) * D)
    cu_host = [0, 300]
    cu = torch.tensor(cu_host, dtype=torch.int32, device="cuda")
    ops.attention(qkv, cu, cu_host, 300, hq, hkv, D)
    with pytest.raises(RuntimeError, match="attention work item"):
        ops.check_status()
    ops.check_status()     # cleared; and the device still works
    assert torch.ones(8, device="cuda").sum().item() == 8


def _moe_layer(T, H, F, E, k, popular, seed=0, act="silu"):
    """A routed layer in one flat buffer: ``(cfg, p, g, n2, h1, dout)``; only the first ``popular`` experts are ever chosen."""
    from mini_trainer_b200.models import layout as L
    from mini_trainer_b200.models.config import ModelConfig
    torch.manual_seed(seed)
    cfg = ModelConfig(model_type="mixtral", vocab_size=64, hidden_size=H, intermediate_size=F, num_hidden_layers=1, num_attention_heads=1,
                      num_key_value_heads=1, head_dim=64, num_local_experts=E, num_experts_per_tok=k,
                      hidden_act="gelu_pytorch_tanh" if act != "silu" else "silu")
    entries = [("router", (E, H))]
    for e in range(E):
        entries += [(f"wgu{e}", (2 * F, H)), (f"wd{e}", (H, F))]
    lay = L.GroupLayout("x", entries, 1)
    p = lay.views(bf(lay.padded_numel, scale=0.05))
    g = lay.views(torch.full((lay.padded_numel,), float("nan"), dtype=torch.bfloat16, device="cuda"))
    n2 = bf(T, H)
    if popular < E:   # the other experts' logits lie far below
        d = torch.randn(H, device="cuda")
        d /= d.norm()
        n2 = (n2.float() + 6 * d).bfloat16()
        p["router"][popular:] = (p["router"][popular:].float() - 10 * d).bfloat16()
    return cfg, p, g, n2, bf(T, H), bf(T, H)


# one token; slabs of exactly one and two row tiles; sizes off every tile edge; idle experts; a reduction shorter than one k-block;
# more experts than a warp has lanes
@pytest.mark.parametrize("T,H,F,E,k,popular,act", [(1, 64, 72, 4, 2, 4, "silu"), (128, 128, 64, 2, 2, 2, "silu"), (256, 264, 200, 3, 1, 1, "silu"),
                                                   (777, 520, 328, 8, 2, 5, "silu"), (300, 256, 136, 40, 8, 40, "gelu"),
                                                   (2051, 512, 256, 64, 4, 33, "silu")])
def test_grouped_experts_match_loop_over_experts(ops, T, H, F, E, k, popular, act):
    from mini_trainer_b200.models import moe as M
    cfg, p, g, n2, h1, dout = _moe_layer(T, H, F, E, k, popular, act=act)
    assert ops.expert_stack(p, "wgu", E) is not None
    loose = {n: w.clone() for n, w in p.items()}           # separate tensors: the loop over experts
    gl = {n: torch.full_like(w, float("nan")) for n, w in loose.items()}
    res = {}
    try:
        for name, pp, gg in (("grouped", p, g), ("loop", loose, gl)):
            if name == "loop":
                ops.expert_stack = lambda *a: None
            out, st = M.moe_forward(ops, cfg, pp, n2, h1, True, False)
            assert (st.slabs is not None) == (name == "grouped")
            res[name] = (out, M.moe_backward(ops, cfg, pp, gg, st, n2, dout))
    finally:
        del ops.expert_stack
    ops.check_status()
    # same products in bf16; the loop rounds the weighted rows and the scaled gradients to bf16 where the kernels do not
    for a, b in zip(res["grouped"], res["loop"]):
        assert rel_err(a, b) < 1e-2
    for n in p:
        if gl[n].float().norm() == 0:
            assert g[n].float().norm() == 0, n
        else:
            assert rel_err(g[n], gl[n]) < 1.5e-2, n
    again = M.moe_forward(ops, cfg, p, n2, h1, True, False)
    assert torch.equal(again[0], res["grouped"][0])
    first = {n: w.clone() for n, w in g.items()}
    dn2 = M.moe_backward(ops, cfg, p, g, again[1], n2, dout)
    assert torch.equal(dn2, res["grouped"][1]) and all(torch.equal(first[n], g[n]) for n in g)
    # gradients that are not stacked like the weights come out the same
    gs = {n: torch.full_like(w, float("nan")) for n, w in p.items()}
    gs["wgu0"] = torch.cat([gs["wgu0"].reshape(-1), gs["wgu0"].new_zeros(8)])[: gs["wgu0"].numel()].view_as(p["wgu0"])
    M.moe_backward(ops, cfg, p, gs, again[1], n2, dout)
    assert all(torch.equal(first[n], gs[n]) for n in gs)


# work items per tile > 1: few tiles and a long reduction, odd sizes, both kernels, every operand layout, bias / residual / fp32
@pytest.mark.parametrize("M,N,K", [(128, 256, 4096), (1536, 1536, 6000), (136, 264, 1000), (2048, 520, 7777)])
@pytest.mark.parametrize("two_cta", [False, True])
def test_gemm_split_k(ops, M, N, K, two_cta):
    torch.manual_seed(M + K)
    K8 = -(-K // 8) * 8
    a, b = bf(M, K8), bf(N, K8, scale=0.1)
    a, b = a[:, :K], b[:, :K]
    ref = a.float() @ b.float().t()
    res, bias = bf(M, N), bf(N)
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ops.gemm(a, False, b, False, out, M, N, K, residual=res, bias=bias, alpha=0.5, two_cta=two_cta)
    want = 0.5 * ref + bias.float() + res.float()
    assert rel_err(out, want) < 4e-3
    first = out.clone()
    ops.gemm(a, False, b, False, out, M, N, K, residual=res, bias=bias, alpha=0.5, two_cta=two_cta)
    assert torch.equal(first, out)     # one order of summation, whoever arrives last
    o32 = torch.empty(M, N, dtype=torch.float32, device="cuda")
    if M % 8 == 0:
        at, bt = a.t().contiguous(), b.t().contiguous()
        ops.gemm(at, True, bt, True, o32, M, N, K, two_cta=two_cta)
        assert rel_err(o32, ref) < 1e-5    # fp32 sums of exact products of bf16 values
    ops.check_status()


# work tables longer than one round of persistent CTAs; key blocks whose heads one CTA keeps (many units) or several share (few);
# query tiles that pair up by head (even GQA ratio) or by row block (odd), with a last row block that has no partner
@pytest.mark.parametrize("D,hq,hkv,lens", [(64, 4, 2, [130] * 100), (128, 6, 2, [257, 1, 128, 255, 256, 300] * 12), (64, 3, 1, [700, 384, 90]),
                                           (128, 2, 2, [129] * 80)])
def test_attention_work_distribution(ops, D, hq, hkv, lens):
    torch.manual_seed(sum(lens))
    T = sum(lens)
    qkv, dout = bf(T, (hq + 2 * hkv) * D), bf(T, hq * D)
    cu_host, cu = _cu(lens)
    out, lse = ops.attention(qkv, cu, cu_host, max(lens), hq, hkv, D)
    dqkv = ops.attention_bwd(dout, qkv, out, lse, cu, cu_host, max(lens), hq, hkv, D)
    ops.check_status()
    ro, rl = REF.attention(qkv.float(), cu, cu_host, max(lens), hq, hkv, D)
    rd = REF.attention_bwd(dout.float(), qkv.float(), ro, rl, cu, cu_host, max(lens), hq, hkv, D)
    assert rel_err(lse, rl) < 2e-3 and rel_err(out, ro) < 1e-2 and max_err(out, ro) < 0.1
    assert rel_err(dqkv, rd) < 1.5e-2
    again = ops.attention_bwd(dout, qkv, out, lse, cu, cu_host, max(lens), hq, hkv, D)
    kv = hq * D
    assert torch.equal(again[:, kv:], dqkv[:, kv:])     # dK and dV: one order of summation (dQ is accumulated in any order)


# either side of the line between a launch under its predecessor's tail and one behind its end: 20 iterations of a CTA on average
@pytest.mark.parametrize("lens", [[4864], [4992], [1500, 1600], [5200, 4900]])
def test_attention_backward_waits_for_what_it_reads(ops, lens):
    torch.manual_seed(sum(lens))
    D, hq, hkv, T = 128, 8, 8, sum(lens)
    qkv, a, b = bf(T, 3 * hq * D), bf(T, 2048, scale=2048 ** -0.5), bf(hq * D, 2048)
    cu_host, cu = _cu(lens)
    args = (cu, cu_host, max(lens), hq, hkv, D)
    out, lse = ops.attention(qkv, *args)
    assert ops._plan_attention_bwd(cu_host, hq, hkv, D)[1::2] == (1, int(min(lens) > 4864))
    want = ops.linear(a, b)
    torch.cuda.synchronize()
    ref = ops.attention_bwd(want, qkv, out, lse, *args)
    rd = REF.attention_bwd(want.float(), qkv.float(), out.float(), lse, *args)
    assert rel_err(ref, rd) < 1.5e-2
    for _ in range(3):   # the gradient and the forward's results as they leave their kernels
        torch.cuda.synchronize()
        o, l = ops.attention(qkv, *args)
        got = ops.attention_bwd(ops.linear(a, b), qkv, o, l, *args)
        assert torch.equal(got[:, hq * D:], ref[:, hq * D:])     # dK and dV: one order of summation
    ops.check_status()


# more rows than resident blocks, row widths of one to eight vectors per thread
@pytest.mark.parametrize("T,H", [(5000, 512), (3001, 2056), (700, 12296), (1300, 5000)])
def test_norms_many_rows(ops, T, H):
    torch.manual_seed(T)
    x, w, b, dy, add = bf(T, H), bf(H), bf(H), bf(T, H), bf(T, H)
    y, rstd = ops.rmsnorm(x, w, 1e-5)
    ry, rr = REF.rmsnorm(x.float(), w.float(), 1e-5)
    assert rel_err(y, ry) < 5e-3 and rel_err(rstd, rr.reshape(-1)) < 1e-5
    dw, rdw = torch.empty_like(w), torch.empty(H, device="cuda")
    dx = ops.rmsnorm_bwd(dy, x, rstd, w, dw, add_to=add)
    assert rel_err(dx, REF.rmsnorm_bwd(dy.float(), x.float(), rr, w.float(), rdw, add_to=add.float())) < 5e-3 and rel_err(dw, rdw) < 5e-3
    if H <= 8192:
        y, st = ops.layernorm(x, w, b, 1e-5)
        ry, rst = REF.layernorm(x.float(), w.float(), b.float(), 1e-5)
        assert rel_err(y, ry) < 5e-3
        db, rdb = torch.empty_like(b), torch.empty(H, device="cuda")
        dx = ops.layernorm_bwd(dy, x, st, w, dw, db, add_to=None)
        assert rel_err(dx, REF.layernorm_bwd(dy.float(), x.float(), rst, w.float(), rdw, rdb)) < 5e-3
        assert rel_err(dw, rdw) < 5e-3 and rel_err(db, rdb) < 5e-3


def test_gelu_backward_with_activation(ops):
    x, dy = bf(333, 72, scale=3.0), bf(333, 72)
    want_dx, want_act = ops.gelu_bwd(dy, x), ops.gelu(x)
    d = dy.clone()
    dx, act = ops.gelu_bwd_act(d, x)
    assert act is d and torch.equal(dx, want_dx) and torch.equal(act, want_act)


# one chunk (dW straight to bf16, with and without what is already there) against several (fp32 sums)
@pytest.mark.parametrize("V", [4104, 520])
def test_linear_ce_chunks(ops, V):
    torch.manual_seed(V)
    T, H = 300, 256
    x, w = bf(T, H), bf(V, H, scale=0.05)
    tg = torch.randint(0, V, (T,), device="cuda")
    tg[::7] = -100
    keep = ops.ce_chunk
    res = []
    try:
        for chunk in (8192, 128):
            ops.ce_chunk = chunk
            dw = torch.full_like(w, 0.25)
            loss, dx = ops.linear_ce(x, w, tg, 0.01, dw, accumulate_dw=True)
            dw2 = torch.full_like(w, float("nan"))
            ops.linear_ce(x, w, tg, 0.01, dw2)
            res.append((loss, dx, dw, dw2))
    finally:
        ops.ce_chunk = keep
    ref = torch.nn.functional.cross_entropy((x.float() @ w.float().t()).bfloat16().float(), tg, reduction="none", ignore_index=-100)
    assert (res[0][0] - ref).abs().max() < 2e-3     # bf16 logits on both sides, fp32 sums of up to V exponentials
    for a, b in zip(*res):
        assert rel_err(a, b) < 4e-3


# heads that do not fill a warp's group of four; the pass with the rotation against the norm and the rotation as passes of their own
@pytest.mark.parametrize("D,hq,hkv,T", [(128, 4, 1, 257), (64, 4, 2, 33), (256, 2, 1, 100), (128, 16, 8, 1031)])
def test_qk_norm_with_rotation(ops, D, hq, hkv, T):
    torch.manual_seed(T)
    nh = hq + hkv
    qkv, dqkv = bf(T, (hq + 2 * hkv) * D), bf(T, (hq + 2 * hkv) * D)
    wq, wk = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16(), (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16()
    pos = (torch.arange(T, device="cuda") * 7 % 5000).to(torch.int32)
    inv = (1e4 ** (-torch.arange(0, D, 2, device="cuda").float() / D))
    a, b = qkv.clone(), qkv.clone()
    pre, rstd = ops.qk_norm_rope_(a, wq, wk, 1e-6, hq, hkv, D, pos, inv)
    r2 = ops.head_rmsnorm_(b, wq, wk, 1e-6, hq, hkv, D)
    ops.rope_(b, pos, inv, hq, hkv, D)
    assert torch.equal(pre, qkv[:, : nh * D]) and torch.equal(rstd, r2) and torch.equal(a[:, nh * D:], qkv[:, nh * D:])
    # same roundings in between; the compiler may contract the rotation's products differently, one bf16 step
    assert (a.float() - b.float()).abs().max() <= 2 ** -7 * b.float().abs().max() and rel_err(a, b) < 1e-3
    g = [torch.empty_like(wq) for _ in range(4)]
    c, d = dqkv.clone(), dqkv.clone()
    ops.qk_norm_rope_bwd_(c, pre, rstd, wq, wk, g[0], g[1], hq, hkv, D, pos, inv)
    ops.rope_(d, pos, inv, hq, hkv, D, inverse=True)
    ops.head_rmsnorm_bwd_(d, pre, rstd, wq, wk, g[2], g[3], hq, hkv, D)
    assert rel_err(c, d) < 1e-3 and rel_err(g[0], g[2]) < 5e-3 and rel_err(g[1], g[3]) < 5e-3
    assert torch.equal(c[:, nh * D:], dqkv[:, nh * D:])


def test_split_workspaces_are_per_stream_and_bounded(ops):
    """Split GEMMs on several streams at once, more streams than workspaces are kept, and a captured one."""
    torch.manual_seed(3)
    M, N, K = 256, 256, 8192
    a, b = bf(M, K), bf(N, K, scale=0.1)
    ref = a.float() @ b.float().t()
    streams = [torch.cuda.Stream() for _ in range(11)]
    outs = [torch.empty(M, N, dtype=torch.bfloat16, device="cuda") for _ in streams]
    torch.cuda.synchronize()
    for _ in range(3):
        for s, o in zip(streams, outs):
            with torch.cuda.stream(s):
                ops.gemm(a, False, b, False, o, M, N, K)
    torch.cuda.synchronize()
    assert len(ops._gemm_ws) <= 8
    assert all(torch.equal(o, outs[0]) for o in outs) and rel_err(outs[0], ref) < 4e-3
    out = torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")
    g = torch.cuda.CUDAGraph()
    kept = set(ops._gemm_ws)
    with torch.cuda.graph(g):
        ops.gemm(a, False, b, False, out, M, N, K)
    assert set(ops._gemm_ws) == kept
    g.replay()
    torch.cuda.synchronize()
    assert rel_err(out, ref) < 4e-3
    ops.check_status()


def _ints(*shape):
    return torch.randint(-1, 2, shape, device="cuda").to(torch.bfloat16)


# last row tiles of which only one to three of the four 32-row quarters exist, many tiles per worker and reductions so short that the
# next accumulator is ready while the last box of a tile is still being stored; operands of -1, 0, 1: every sum is exact
@pytest.mark.parametrize("rows", [1, 33, 65, 129, 193])
@pytest.mark.parametrize("two_cta", [False, True])
@pytest.mark.parametrize("f32", [False, True])
def test_gemm_ragged_last_tile_is_exact(ops, rows, two_cta, f32):
    M, N = 256 * 37 + rows, 2056 if f32 else 2120
    dt = torch.float32 if f32 else torch.bfloat16
    for K in (64, 200):
        a, b = _ints(M, K), _ints(N, K)
        want = (a.float() @ b.float().t()).to(dt)
        for _ in range(4):
            out = torch.full((M, N), float("nan"), dtype=dt, device="cuda")
            ops.gemm(a, False, b, False, out, M, N, K, two_cta=two_cta)
            assert torch.equal(out, want)
    ops.check_status()


@pytest.mark.parametrize("M,N", [(136, 264), (72, 136), (648, 520)])
def test_grouped_weight_gradient_ragged_rows_is_exact(ops, M, N):
    """Output matrices with partial last row tiles, slabs of a few k-blocks and experts without rows."""
    T, E, k = 900, 48, 2
    topi = torch.randint(0, E // 2, (T, k), device="cuda") * 2
    sl = ops.expert_slabs(topi, E)
    dy, x = _ints(T, M), _ints(T, N)
    dys, xs = ops.gather_rows(dy, sl), ops.gather_rows(x, sl)
    flat = topi.reshape(-1)
    for _ in range(4):
        dw = torch.full((E, M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.grouped_wgrad(dys, xs, (dw[0], M * N), sl)
        for e in range(E):
            tok = (flat == e).nonzero().reshape(-1) // k
            assert torch.equal(dw[e], (dy[tok].float().t() @ x[tok].float()).bfloat16()), e
    ops.check_status()


# every operand layout, both kernels, whole tiles and split reductions, a last column tile that is not full
@pytest.mark.parametrize("M,N,K", [(300, 776, 320), (136, 264, 4096), (1031, 2120, 128)])
@pytest.mark.parametrize("layout", ["nt", "nn", "tn", "tt"])
@pytest.mark.parametrize("two_cta", [False, True])
def test_gemm_row_statistics(ops, M, N, K, layout, two_cta):
    """Maximum and sum of exponentials per row and 256 columns, against the same of the output as it was stored."""
    if layout[0] == "t":
        M = -(-M // 8) * 8
    torch.manual_seed(M + N)
    a, b = bf(M, K), bf(N, K, scale=4 * K ** -0.5)
    at, bt = (a.t().contiguous() if layout[0] == "t" else a), (b if layout[1] == "t" else b.t().contiguous())
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    tiles = -(-N // 256)
    stats = torch.full((M, tiles, 2), float("nan"), device="cuda")
    ops.gemm(at, layout[0] == "t", bt, layout[1] == "n", out, M, N, K, two_cta=two_cta, stats=stats)
    ops.check_status()
    ref = a.float() @ b.float().t()
    assert rel_err(out, ref) < 6e-3
    x = torch.full((M, tiles * 256), float("-inf"), device="cuda")
    x[:, :N] = out.float()
    x = x.view(M, tiles, 256)
    mx = x.max(-1).values
    assert torch.equal(stats[..., 0], mx)
    # fp32 sums of up to 256 exponentials, each within a few ulp
    assert rel_err(stats[..., 1], (x.double() - mx.double()[..., None]).exp().sum(-1)) < 1e-5
    plain = torch.empty_like(out)
    ops.gemm(at, layout[0] == "t", bt, layout[1] == "n", plain, M, N, K, two_cta=two_cta)
    assert torch.equal(plain, out)


@pytest.mark.parametrize("pairs", [True, False])
@pytest.mark.parametrize("D,hq,hkv,lens", ATTN_CASES + [(64, 3, 1, [257, 1, 128, 384]), (64, 14, 2, [2049, 63]), (64, 4, 2, [130] * 100),
                                                        (128, 6, 2, [257, 1, 128, 255, 256, 300] * 12), (128, 2, 2, [129] * 80)])
def test_attention_forward_both_forms(ops, D, hq, hkv, lens, pairs, monkeypatch):
    """Every batch through pairs of query tiles and through one tile per CTA, whichever the sizes would choose; among them batches of
    several rounds of the persistent CTAs."""
    from mini_trainer_b200.ops import attention_plan
    monkeypatch.setattr(attention_plan, "forward_in_pairs", lambda *a: pairs)
    torch.manual_seed(sum(lens) + pairs)
    T = sum(lens)
    qkv = bf(T, (hq + 2 * hkv) * D)
    qkv[: T // 2] *= 4    # maxima that move by more than the rescale threshold
    cu_host, cu = _cu(lens)
    n0 = ops.launches
    out, lse = ops.attention(qkv, cu, cu_host, max(lens), hq, hkv, D)
    assert ops.launches == n0 + 1
    ro, rl = REF.attention(qkv.float(), cu, cu_host, max(lens), hq, hkv, D)
    ops.check_status()
    assert rel_err(lse, rl) < 2e-3 and (lse - rl).abs().max() < 3e-2
    assert rel_err(out, ro) < 1e-2 and max_err(out, ro) < 0.1
    out2, lse2 = ops.attention(qkv, cu, cu_host, max(lens), hq, hkv, D)
    assert torch.equal(out, out2) and torch.equal(lse, lse2)


# both sides of every line the forward of the norms is drawn by: few and many row sets per block, one block per row, the widths at
# which a row takes one to eight warps, partial last row sets
@pytest.mark.parametrize("T,H", [(1, 8), (3, 256), (2368 * 2 + 1, 512), (20011, 512), (740, 896), (15000, 896), (1481, 12288), (450, 12288), (3, 16384),
                                 (800, 16384), (2930, 2048), (2929, 2048), (5857, 1024), (1023, 1024), (1024, 1024), (9400, 2560), (9375, 2560), (6001, 4096), (5000, 5120), (2930, 8192),
                                 (100, 8192)])
def test_norm_forward_forms(ops, T, H):
    torch.manual_seed(T + H)
    x, w, b = bf(T, H), bf(H), bf(H)
    x += 0.5
    y, rstd = ops.rmsnorm(x, w, 1e-5)
    xf = x.double()
    r = (xf.pow(2).mean(-1, keepdim=True) + 1e-5).rsqrt()
    assert rel_err(rstd, r.reshape(-1)) < 1e-6                    # fp32 sums of up to 16384 squares
    assert max_err(y, (xf * r).bfloat16().double() * w.double()) < 2e-2   # one bf16 step of the normalised value, one of the product
    if H <= 8192:
        y, (mean, rstd) = ops.layernorm(x, w, b, 1e-5)
        mu = xf.mean(-1, keepdim=True)
        r = ((xf - mu).pow(2).mean(-1, keepdim=True) + 1e-5).rsqrt()
        assert (mean - mu.reshape(-1)).abs().max() < 1e-6 and rel_err(rstd, r.reshape(-1)) < 1e-6
        assert max_err(y, (xf - mu) * r * w.double() + b.double()) < 1e-2
    ops.check_status()


@pytest.mark.parametrize("T,N", [(1, 512), (8, 896), (37, 66), (4000, 1024), (4000, 1032), (8191, 264), (8192, 264), (9001, 5120), (9001, 5128), (700, 6)])
def test_column_sums_forms(ops, T, N):
    """Both load widths, both unrollings, one to 32 partial rows."""
    torch.manual_seed(T + N)
    x = bf(T, N)
    out, scratch = torch.empty(N, dtype=torch.bfloat16, device="cuda"), torch.empty(32 * N, device="cuda")
    ops._call("mtb200_colsum", x.data_ptr(), x.stride(0), out.data_ptr(), scratch.data_ptr(), T, N, ops._st())
    ref = x.double().sum(0)
    # one rounding to bf16, and fp32 sums whose terms have the size of the column's norm
    assert ((out.double() - ref).abs() <= ref.abs() * 2 ** -8 + x.double().pow(2).sum(0).sqrt() * 1e-5).all()


def test_split_launches_behind_one_that_gave_up(ops):
    """Arrivals that a launch which gave up has left in the counters do not count in the launches after it."""
    torch.manual_seed(5)
    M, N, K = 136, 264, 4096
    a, b = bf(M, K), bf(N, K, scale=0.1)
    lens, hq, hkv, D = [300, 200], 8, 2, 64
    T = sum(lens)
    qkv, dout = bf(T, (hq + 2 * hkv) * D), bf(T, hq * D)
    cu_host, cu = _cu(lens)
    out, lse = ops.attention(qkv, cu, cu_host, max(lens), hq, hkv, D)

    def both():
        o = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.gemm(a, False, b, False, o, M, N, K)
        return o, ops.attention_bwd(dout, qkv, out, lse, cu, cu_host, max(lens), hq, hkv, D)[:, hq * D:]
    first = both()
    counters = ops._split_workspace(ops._st())
    assert not counters.any()
    epoch = next(ops._epoch)
    for stale in (1, 3, 7):
        counters.fill_((epoch << 16) + stale)
        for x, y in zip(both(), first):
            assert torch.equal(x, y)
    counters.zero_()
    ops.check_status()


def test_split_launches_hold_no_scratch(ops):
    """What a split product takes beyond its output goes back to the allocator; one that does not split takes nothing."""
    a, b = bf(256, 8192), bf(256, 8192, scale=0.1)
    out = torch.empty(256, 256, dtype=torch.bfloat16, device="cuda")
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        ops.gemm(a, False, b, False, out, 256, 256, 8192)
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        ops.gemm(a, False, b, False, out, 256, 256, 8192)
        assert torch.cuda.memory_allocated() == before and 0 < torch.cuda.max_memory_allocated() - before <= 8 << 20
        torch.cuda.reset_peak_memory_stats()
        ops.gemm(a, False, b, False, out, 256, 256, 256)
        assert torch.cuda.max_memory_allocated() == before
    assert all(w.numel() * w.element_size() <= 32768 for w in ops._gemm_ws.values())
    torch.cuda.synchronize()
    ops.check_status()


# the parts of a routed layer that a Mixtral leaves out: a shared expert behind a sigmoid gate, a branch multiplier, weights that are not
# renormalised over the chosen experts; alone and together, with idle experts and sizes off the tile edges
@pytest.mark.parametrize("shared,rm,renorm", [(72, 1.0, True), (0, 0.22, True), (0, 1.0, False), (136, 0.22, False)])
@pytest.mark.parametrize("T,H,F,E,k,popular", [(300, 264, 136, 8, 2, 5), (65, 128, 72, 40, 4, 40)])
def test_grouped_experts_shared_scaled_unnormalised(ops, T, H, F, E, k, popular, shared, rm, renorm):
    from dataclasses import replace
    from mini_trainer_b200.models import layout as L, moe as M
    cfg, p0, _, n2, h1, dout = _moe_layer(T, H, F, E, k, popular, seed=3)
    cfg = replace(cfg, residual_multiplier=rm, norm_topk_prob=renorm, shared_expert_intermediate_size=shared or None,
                  model_type="qwen2_moe" if shared else "mixtral")
    entries = [(n, tuple(w.shape)) for n, w in p0.items()]
    if shared:
        entries += [("wgus", (2 * shared, H)), ("wds", (H, shared)), ("wsg", (1, H))]
    lay = L.GroupLayout("x", entries, 1)
    p = lay.views(bf(lay.padded_numel, scale=0.05))
    for n, w in p0.items():
        p[n].copy_(w)
    res, grads = {}, {}
    try:
        for name in ("grouped", "loop"):
            if name == "loop":
                ops.expert_stack = lambda *a: None
            pp = p if name == "grouped" else {n: w.clone() for n, w in p.items()}
            grads[name] = lay.views(torch.full((lay.padded_numel,), float("nan"), dtype=torch.bfloat16, device="cuda"))
            out, st = M.moe_forward(ops, cfg, pp, n2, h1, True, False)
            assert (st.slabs is not None) == (name == "grouped")
            res[name] = (out, M.moe_backward(ops, cfg, pp, grads[name], st, n2, dout))
    finally:
        del ops.expert_stack
    ops.check_status()
    # and both against the layer in fp32 on the experts that were chosen
    ref_ops = TorchOps()
    pf = {n: w.float() for n, w in p.items()}
    gf = {n: torch.full_like(w, float("nan")) for n, w in pf.items()}
    real = M.route
    try:
        M.route = lambda c, w, x, topi=None: real(c, w, x, topi=st.topi)
        fo, fst = M.moe_forward(ref_ops, cfg, pf, n2.float(), h1.float(), True, False)
        fd = M.moe_backward(ref_ops, cfg, pf, gf, fst, n2.float(), dout.float())
    finally:
        M.route = real
    for a, b, f in zip(res["grouped"], res["loop"], (fo, fd)):
        assert rel_err(a, b) < 1e-2       # bf16 on both sides; the loop rounds weighted rows and scaled gradients in between
        assert rel_err(a, f) < 1.5e-2 and rel_err(a, f) < 1.1 * rel_err(b, f) + 1e-4
    for n in p:
        a, b, f = grads["grouped"][n], grads["loop"][n], gf[n]
        if f.norm() == 0:
            assert a.float().norm() == 0, n
        else:
            assert rel_err(a, b) < 2e-2 and rel_err(a, f) < 1.3 * rel_err(b, f) + 1e-3, n


# every number of work items per tile that the choice may take, also where it would not: reductions of 16 to 122 k-blocks divided evenly
# and unevenly, both kernels
@pytest.mark.parametrize("splits", [2, 3, 7, 16])
@pytest.mark.parametrize("two_cta", [False, True])
@pytest.mark.parametrize("M,N,K", [(136, 264, 1024), (300, 520, 7776)])
def test_gemm_every_split(ops, M, N, K, two_cta, splits, monkeypatch):
    from mini_trainer_b200.ops import gemm_plan
    monkeypatch.setattr(gemm_plan, "narrow", lambda *a: None)   # which products of these sizes take by themselves
    monkeypatch.setattr(gemm_plan, "wide", lambda *a: 0)
    monkeypatch.setattr(gemm_plan, "choose", lambda *a: (two_cta, splits))
    monkeypatch.setattr(ops, "_gemm_plans", {})
    ran = []
    monkeypatch.setattr(ops, "_call", lambda name, *a, call=ops._call, **kw: ran.append((name, a[16])) or call(name, *a, **kw))
    a, b, res = _ints(M, K), _ints(N, K), _ints(M, N)
    want = a.float() @ b.float().t()       # integers below 2^24: exact in fp32 in any order
    for dt in (torch.float32, torch.bfloat16):
        out = torch.full((M, N), float("nan"), dtype=dt, device="cuda")
        ops.gemm(a, False, b, False, out, M, N, K, residual=res.to(dt))
        assert torch.equal(out, (want + res.float()).to(dt))
    assert ran == [("mtb200_gemm2_bf16" if two_cta else "mtb200_gemm_bf16", splits)] * 2
    ops.check_status()


@pytest.mark.parametrize("D,hq,hkv,lens", [(128, 7, 1, [300, 129, 1]), (64, 12, 2, [640, 90])])
def test_attention_backward_every_division(ops, D, hq, hkv, lens, monkeypatch):
    """A key block's query heads on one to as many CTAs as there are heads, evenly divided or not."""
    from mini_trainer_b200.ops import attention_plan
    torch.manual_seed(9)
    T = sum(lens)
    qkv, dout = bf(T, (hq + 2 * hkv) * D), bf(T, hq * D)
    cu_host, cu = _cu(lens)
    out, lse = ops.attention(qkv, cu, cu_host, max(lens), hq, hkv, D)
    ro, rl = REF.attention(qkv.float(), cu, cu_host, max(lens), hq, hkv, D)
    rd = REF.attention_bwd(dout.float(), qkv.float(), ro, rl, cu, cu_host, max(lens), hq, hkv, D)
    first = None
    for s in range(1, hq // hkv + 1):
        monkeypatch.setattr(attention_plan, "backward_splits", lambda *a: s)
        cu_host = list(cu_host)            # another minibatch: nothing planned for it
        d = ops.attention_bwd(dout, qkv, out, lse, cu, cu_host, max(lens), hq, hkv, D)
        assert rel_err(d, rd) < 1.5e-2
        first = d if first is None else first
        # the sums of the CTAs' parts are fp32: what differs from the undivided sum is its rounding to bf16
        assert rel_err(d[:, hq * D:], first[:, hq * D:]) < 3e-3
    ops.check_status()


# rows held in registers (up to 32768 columns, 1024 to a warp), longer ones and ones with statistics, by blocks of 1024 threads and of 512; fewer rows than
# blocks, and several to a block
@pytest.mark.parametrize("R,V,stats", [(1, 8, False), (700, 1024, False), (300, 1032, False), (1300, 5000, False), (400, 16392, False), (1, 32768, False),
                                       (310, 32768, False), (5, 32776, False), (150, 65544, False), (888, 32776, False), (887, 5000, True), (888, 5000, True),
                                       (888, 57344, True), (3, 296, True)])
@pytest.mark.parametrize("in_place", [True, False])
def test_cross_entropy_rows(ops, R, V, stats, in_place):
    torch.manual_seed(R + V)
    ld = V + 16
    lg = bf(R, ld, scale=4)
    if R > 1:
        lg[0, V // 2:V] = float("-inf")
    lg[-1, :V // 2] = torch.finfo(torch.bfloat16).min
    tg = torch.randint(0, V, (R,), device="cuda")
    tg[0], tg[-1] = 0, V - 1   # not where a row is masked
    tg[1::7] = -100
    x = lg[:, :V].double()
    lse = torch.logsumexp(x, 1)
    want = lse - x.gather(1, tg.clamp_min(0)[:, None])[:, 0]
    grad = (x - lse[:, None]).exp()
    grad.scatter_add_(1, tg.clamp_min(0)[:, None], torch.full((R, 1), -1.0, device="cuda", dtype=torch.double))
    want[tg == -100], grad[tg == -100] = 0, 0
    kept = lg[:, V:].clone()
    st = None
    if stats:
        tiles = torch.nn.functional.pad(x, (0, -V % 256), value=float("-inf")).view(R, -1, 256)
        top = tiles.amax(-1)
        st = torch.stack([top, (tiles - top.clamp_min(-1e38)[..., None]).exp().sum(-1)], -1).float().contiguous()
    out, loss = lg if in_place else torch.full_like(lg, 7.0), torch.full((R,), 7.0, device="cuda")
    rest = kept if in_place else torch.full_like(kept, 7.0)
    ops._call("mtb200_ce_fwd_bwd", lg.data_ptr(), ld, 1, st.data_ptr() if stats else 0, tg.data_ptr(), loss.data_ptr(), out.data_ptr(), ld, R, V, 0.5, -100, ops._st())
    # fp32 sums of V positive terms, each thread's and warp's in turn, and the rounding of a logarithm and a logit of up to 32
    assert (loss - want).abs().max() < 1e-5
    assert ((out[:, :V].double() - 0.5 * grad).abs() <= 0.5 * (2 ** -8 * grad.abs() + 2e-6)).all()   # one rounding to bf16
    assert torch.equal(out[:, V:], rest)
    ops.check_status()


# rows held in registers, rows that are read twice, rows with statistics, fp32 logits
CE_FORMS = [(264, "rows"), (32776, "rows"), (264, "statistics"), (520, "fp32")]


def _ce_forms(ops, lg, ld, V, form, tg):
    """``(loss, gradient)`` of ``lg[:, :V]`` (a scale of 1, -100 ignored) from the form of the kernel that is named."""
    R = lg.shape[0]
    st = 0
    if form == "statistics":
        tiles = torch.nn.functional.pad(lg[:, :V].double(), (0, -V % 256), value=float("-inf")).view(R, -1, 256)
        top = tiles.amax(-1)
        st = torch.stack([top, (tiles - top.clamp_min(-1e38)[..., None]).exp().sum(-1)], -1).float().contiguous()
    src = lg.float() if form == "fp32" else lg
    out, loss = torch.full_like(lg, 7.0), torch.full((R,), 7.0, device="cuda")
    ops._call("mtb200_ce_fwd_bwd", src.data_ptr(), ld, int(form != "fp32"), st if isinstance(st, int) else st.data_ptr(), tg.data_ptr(), loss.data_ptr(),
              out.data_ptr(), ld, R, V, 1.0, -100, ops._st())
    return loss, out[:, :V]


@pytest.mark.parametrize("V,form", CE_FORMS)
def test_cross_entropy_of_a_target_that_is_no_column(ops, V, form):
    """Nothing outside the row is read for it: the loss is NaN, the gradient that of no target, and other rows are what they are without it."""
    torch.manual_seed(V)
    lg = bf(6, V + 16, scale=4)
    tg = torch.tensor([3, V, V - 1, -1, 1 << 40, 0], device="cuda")
    loss, grad = _ce_forms(ops, lg, V + 16, V, form, tg)
    x = lg[:, :V].double()
    want = torch.softmax(x, 1)
    for r in (0, 2, 5):
        want[r, tg[r]] -= 1
    none = torch.tensor([False, True, False, True, True, False], device="cuda")
    assert loss[none].isnan().all() and (loss - torch.nn.functional.cross_entropy(x, tg.clamp(0, V - 1), reduction="none"))[~none].abs().max() < 1e-5
    assert ((grad.double() - want).abs() <= 2 ** -8 * want.abs() + 2e-6).all()   # one rounding to bf16
    ops.check_status()


@pytest.mark.parametrize("V,form", CE_FORMS + [(5000, "rows")])
def test_cross_entropy_of_low_logits_beside_masked_ones(ops, V, form):
    """Every 32nd vector of eight columns is masked, which are all that some threads have, and the others are far below zero."""
    torch.manual_seed(V)
    lg = bf(5, V + 16, scale=2) - 300
    lg[:, (torch.arange(V + 16, device="cuda") // 8) % 32 == 0] = float("-inf")
    tg = torch.tensor([8, 9, -100, 200, 255], device="cuda")
    loss, grad = _ce_forms(ops, lg, V + 16, V, form, tg)
    x = lg[:, :V].double()
    want = torch.softmax(x, 1)
    want[torch.arange(5), tg.clamp_min(0)] -= 1
    want[2] = 0
    # the maximum and its sum's logarithm are added at 2^-15 a step
    assert (loss - torch.nn.functional.cross_entropy(x, tg, reduction="none", ignore_index=-100)).abs().max() < 2 ** -15
    assert ((grad.double() - want).abs() <= 2 ** -8 * want.abs() + 2e-6).all()   # one rounding to bf16
    ops.check_status()


@pytest.mark.parametrize("form", ["one", "pair", "wide"])
def test_softmax_statistics_of_overflowing_logits(ops, form, monkeypatch):
    """Columns of -infinity count for nothing, also where they are the first of a tile or all of it."""
    from mini_trainer_b200.ops import gemm_plan
    T, K, V = 300, 128, 1032
    monkeypatch.setattr(gemm_plan, "wide", lambda *a: int(form == "wide"))
    monkeypatch.setattr(gemm_plan, "choose", lambda *a: (form == "pair", 1))
    monkeypatch.setattr(ops, "_gemm_plans", {})
    names = []
    monkeypatch.setattr(ops, "_call", lambda name, *a, call=ops._call, **kw: names.append(name) or call(name, *a, **kw))
    torch.manual_seed(6)
    x = (torch.rand(T, K, device="cuda") + 0.5).bfloat16() * 2.0 ** 100
    w = (bf(V, K, scale=K ** -0.5).float() * 2.0 ** -100).bfloat16()
    for a, b in ((0, 8), (40, 48), (256, 512), (768, 808), (1024, 1032)):
        w[a:b] = -(2.0 ** 100)   # products of -2^200 overflow
    out, st = torch.empty(T, V, dtype=torch.bfloat16, device="cuda"), torch.full((T, -(-V // 256), 2), float("nan"), device="cuda")
    ops.gemm(x, False, w, False, out, T, V, K, stats=st)
    assert names == [{"one": "mtb200_gemm_bf16", "pair": "mtb200_gemm2_bf16", "wide": "mtb200_gemm2_wide_bf16"}[form]]
    assert (out[:, :8] == float("-inf")).all() and out[:, 8:40].isfinite().all()
    tiles = torch.nn.functional.pad(out.double(), (0, -V % 256), value=float("-inf")).view(T, -1, 256)
    top = tiles.amax(-1)
    assert torch.equal(st[..., 0].double(), top) and (top[:, 1] == float("-inf")).all() and (top[:, 4] == float("-inf")).all()
    want = (tiles - top.clamp_min(-1e38)[..., None]).exp().sum(-1)
    # 256 fp32 terms of at most one, added one by one
    assert ((st[..., 1].double() - want).abs() <= 256 * 2 ** -24 * want).all()
    ops.check_status()


# logits whose product leaves the statistics and logits whose rows are read for them, in one chunk and in several
@pytest.mark.parametrize("T,H,V", [(130, 1536, 17008), (130, 1528, 17008), (130, 1536, 16384), (70, 64, 520)])
def test_linear_ce_with_and_without_statistics(ops, T, H, V, monkeypatch):
    torch.manual_seed(V + H)
    x, w = bf(T, H), bf(V, H, scale=3 * H ** -0.5)
    tg = torch.randint(0, V, (T,), device="cuda")
    tg[::9] = -100
    seen = []
    gemm = ops.gemm
    monkeypatch.setattr(ops, "gemm", lambda *a, **k: (seen.append(k.get("stats") is not None), gemm(*a, **k))[1])
    lg = (x.float() @ w.float().t()).bfloat16().double()
    ref = torch.nn.functional.cross_entropy(lg, tg, reduction="none", ignore_index=-100)
    p = torch.softmax(lg, -1)
    p[torch.arange(T, device="cuda"), tg.clamp_min(0)] -= 1
    p[tg == -100] = 0
    for chunk in (8192, 64):
        monkeypatch.setattr(ops, "ce_chunk", chunk)
        dw = torch.empty_like(w)
        loss, dx = ops.linear_ce(x, w, tg, 0.5, dw)
        assert (loss - ref).abs().max() < 2e-3        # a bf16 step of a logit near the row's maximum is what may differ
        assert rel_err(dx, 0.5 * p @ w.double()) < 1e-2 and rel_err(dw, 0.5 * p.t() @ x.double()) < 1e-2
    assert any(seen) == (V > 16384 and H >= 1536)
    ops.check_status()


# both sides of the line between one head per warp and four: 2 blocks per SM of 8 warps of four heads
@pytest.mark.parametrize("D,hq,hkv", [(128, 16, 8), (64, 14, 2), (256, 3, 2)])
def test_head_norm_heads_per_warp(ops, D, hq, hkv):
    nh = hq + hkv
    edge = -(-2 * ops.sms * 8 // -(-nh // 4))
    torch.manual_seed(D)
    wq, wk = bf(D), bf(D)
    T = edge
    qkv = bf(T, (hq + 2 * hkv) * D)
    pos = torch.arange(T, device="cuda", dtype=torch.int32)
    inv = 1e4 ** (-torch.arange(0, D, 2, device="cuda").float() / D)
    for rope in (False, True):
        a, b = qkv.clone(), qkv.clone()
        pre, ra = ops.qk_norm_rope_(a, wq, wk, 1e-6, hq, hkv, D, pos if rope else None, inv if rope else None)
        part, rb = ops.qk_norm_rope_(b[: T - 1], wq, wk, 1e-6, hq, hkv, D, pos if rope else None, inv if rope else None)
        assert torch.equal(a[: T - 1], b[: T - 1]) and torch.equal(ra[: (T - 1) * nh], rb)     # the same work, dealt differently
        assert torch.equal(pre[: T - 1], part) and torch.equal(pre, qkv[:, : nh * D]) and torch.equal(a[:, nh * D:], qkv[:, nh * D:])
    x = qkv[:, : nh * D].float().view(T, nh, D)
    assert rel_err(ra, (x.pow(2).mean(-1) + 1e-6).rsqrt().reshape(-1)) < 1e-6
    ops.check_status()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("lens", [[1], [100, 29], [1900, 1100]])
def test_kernels_that_start_under_their_predecessors_tail_wait_for_its_results(ops, lens, captured, monkeypatch):
    """A chain of kernels over few buffers, each overwriting what an earlier one still read: bit for bit what it is with the device idle
    between any two. (A graph's products never split their reduction, so neither do those it is compared with.)"""
    T, hq, hkv, D = sum(lens), 8, 4, 128
    torch.manual_seed(T)
    H, F = 512, 1024
    w1, w2, wn = bf(2 * F, H, scale=0.05), bf(H, F, scale=0.05), bf(H)
    x0, pos = bf(T, H), torch.arange(T, dtype=torch.int32, device="cuda")
    cu_host, cu = _cu(lens)
    inv = 10000.0 ** (-torch.arange(0, 64, device="cuda").float() / 64)
    dw = [torch.empty(2 * F, H, dtype=torch.bfloat16, device="cuda"), torch.empty(H, dtype=torch.bfloat16, device="cuda")]

    def chain(between):
        x, out = x0.clone(), []
        for _ in range(4):
            n, rstd = ops.rmsnorm(x, wn, 1e-5); between()
            gu = ops.linear(n, w1); between()
            act = ops.swiglu(gu); between()
            x = ops.linear(act, w2, residual=x, out=x); between()
            gu, act = ops.linear_act(n, w1); between()
            x = ops.linear(act, w2, residual=x, out=x); between()
            att, lse = ops.attention(gu, cu, cu_host, max(lens), hq, hkv, D); between()
            x = ops.linear(att, w2, residual=x, out=x); between()
            dqkv = ops.attention_bwd(act, gu, att, lse, cu, cu_host, max(lens), hq, hkv, D); between()
            ops.rope_(x, pos, inv, 2, 2, 128); between()
            ops.linear_wgrad(gu, n, dw[0]); between()
            dx = ops.rmsnorm_bwd(n, x, rstd, wn, dw[1], add_to=x); between()
            x = dx
            out += [x.clone(), dw[0].clone(), dw[1].clone(), dqkv[:, hq * D:].clone()]   # (dQ tiles are added in the order they arrive)
            between()
        return out

    if captured:
        monkeypatch.setattr(ops, "_split_workspace", lambda st: None)
    want = chain(torch.cuda.synchronize)
    monkeypatch.undo()
    if captured:
        graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.stream(side):
            chain(lambda: None)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            got = chain(lambda: None)
        for _ in range(3):
            graph.replay()
    else:
        got = chain(lambda: None)
    torch.cuda.synchronize()
    for k, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), k
        assert b.isfinite().all()
    ops.check_status()


# widths at and around a tile's 128 gated or 256 plain columns and a box's 32; heights around a quarter, a CTA and a pair
@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("fn", ["silu", "gelu_tanh"])
@pytest.mark.parametrize("T,H,F", [(1, 64, 8), (31, 72, 40), (128, 64, 128), (129, 128, 136), (257, 200, 264), (300, 264, 1032), (5000, 512, 1544),
                                   (2048, 1024, 4096)])
def test_products_with_an_activation(ops, T, H, F, fn, gated):
    torch.manual_seed(T + F)
    f = {"silu": torch.nn.functional.silu, "gelu_tanh": lambda x: torch.nn.functional.gelu(x, approximate="tanh")}[fn]
    W = 2 * F if gated else F
    x, w = bf(T, H), bf(W, H, scale=2.0 / H ** 0.5)
    bias = None if gated else bf(F)

    def act_of(p):
        return f(p[:, :F]) * p[:, F:] if gated else f(p)

    for pair_max in (0.0, 1e12):   # on one CTA, and by size
        ops.pair_max_flops, before = pair_max, ops.pair_max_flops
        ops._gemm_plans.clear()
        pre, act = ops.linear_act(x, w, fn, gated, bias)
        ops.pair_max_flops = before
        ops._gemm_plans.clear()
        want = x.float() @ w.float().t() + (0 if bias is None else bias.float())
        assert rel_err(pre, want) < 6e-3 and max_err(pre, want) < 5e-2
        # of the pre-activations as they were stored: one rounding of an fp32 value
        assert rel_err(act, act_of(pre.float())) < 4e-3 and max_err(act, act_of(pre.float()), rtol=1e-2) < 1e-2
    ops.check_status()


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("sizes,max_norm", [([128], 1.0), ([1 << 16, 4, 1028, 999936], 0.05), ([256 * k + 4 for k in range(1, 101)], 1e9), ([640] * 48, 0.0)])
def test_optimizer_over_groups_is_the_optimizer_of_each(ops, sizes, max_norm, fp32):
    """One group, sizes below and above a block, more groups than one launch holds, exactly as many; clipped, not clipped and without a limit."""
    torch.manual_seed(len(sizes))
    sd = torch.float32 if fp32 else torch.bfloat16
    f = lambda n: torch.randn(n, device="cuda")   # noqa: E731
    groups = [(f(n), f(n).to(sd), f(n).square().to(sd), f(n), torch.zeros(n, dtype=torch.bfloat16, device="cuda")) for n in sizes]
    alone = [tuple(t.clone() for t in g) for g in groups]
    table = ops.group_table(groups)
    sq = torch.zeros(1, device="cuda")
    ops.add_sumsq_groups(table, sq)
    want = sum(g[3].double().square().sum() for g in groups)
    assert abs(sq.item() - want.item()) < 1e-5 * want.item()
    norm = ops.adamw_groups(table, fp32, sq, max_norm, 1e-3, 0.9, 0.95, 1e-8, 0.01, 3)
    assert torch.equal(norm, sq.sqrt().squeeze(0))
    # (a number over a tensor is a product with the reciprocal in torch, up to one rounding off the quotient)
    coef = torch.div(torch.full((), max_norm, device="cuda"), norm + 1e-6).clamp(max=1.0) if max_norm else torch.ones((), device="cuda")
    for a, b in zip(alone, groups):
        ops.adamw_step(*a, 1e-3, 0.9, 0.95, 1e-8, 0.01, 3, coef)
        assert all(torch.equal(x, y) for x, y in zip(a, b))


def test_optimizer_over_groups_with_a_norm_that_is_not_a_number(ops):
    n = 512
    g = tuple(torch.ones(n, device="cuda") for _ in range(4)) + (torch.zeros(n, dtype=torch.bfloat16, device="cuda"),)
    norm = ops.adamw_groups(ops.group_table([g]), True, torch.full((1,), float("nan"), device="cuda"), 1.0, 1e-3, 0.9, 0.95, 1e-8, 0.0, 1)
    assert norm.isnan() and g[0].isnan().all()   # as the clip coefficient of that norm makes it


@pytest.mark.parametrize("T,V,H", [(1, 8, 8), (255, 3, 64), (257, 40, 136), (300, 1, 2056), (4096, 32000, 256), (2049, 500, 4096), (8192, 900, 128), (8193, 64, 128)])
def test_embedding_gradient_without_a_sort_is_that_with_one(ops, T, V, H, monkeypatch):
    """Few ids and many, one for all tokens, rows wider than a block, the most tokens that are searched and one more: bit for bit."""
    from mini_trainer_b200.ops import native
    torch.manual_seed(T)
    ids, dx = torch.randint(0, V, (T,), device="cuda"), bf(T, H)
    got, want = bf(V, H), None
    want = got.clone()
    ops.embedding_bwd(got, ids, dx)
    monkeypatch.setattr(native, "_EMB_SCAN", 0)
    ops.embedding_bwd(want, ids, dx)
    assert torch.equal(got, want)
    ops.check_status()


def test_embedding_gradient_reports_an_id_outside_the_table(ops):
    ids = torch.tensor([2, 9, 2, -1], device="cuda")
    dw, dx = torch.zeros(4, 64, dtype=torch.bfloat16, device="cuda"), bf(4, 64)
    ops.embedding_bwd(dw, ids, dx)
    assert rel_err(dw[2], dx[0].float() + dx[2].float()) < 1e-2 and dw[[0, 1, 3]].abs().sum() == 0
    with pytest.raises(RuntimeError, match="token id"):
        ops.check_status()


@pytest.mark.parametrize("T,R,H", [(1, 1, 8), (130, 1, 1032), (777, 776, 512), (64, 0, 64)])
def test_rows_scattered_into_zeros(ops, T, R, H):
    torch.manual_seed(T)
    rows = torch.randperm(T, device="cuda")[:R]
    src, vec = bf(R, H), torch.randn(R, device="cuda")
    out, v = ops.scatter_rows(rows, src, vec, T)
    want, wv = torch.zeros(T, H, dtype=torch.bfloat16, device="cuda"), torch.zeros(T, device="cuda")
    want[rows], wv[rows] = src, vec
    assert torch.equal(out, want) and torch.equal(v, wv)
    ops.check_status()


# the largest output that the kernel zeroes (8 M pieces of 16 bytes) and the first that memsets do
@pytest.mark.parametrize("T", [16384, 16385])
def test_rows_scattered_into_many_zeros(ops, T):
    rows, src, vec = torch.tensor([T - 1, 3], device="cuda"), bf(2, 4096), torch.randn(2, device="cuda")
    out, v = ops.scatter_rows(rows, src, vec, T)
    assert torch.equal(out[rows], src) and torch.equal(v[rows], vec)
    out[rows], v[rows] = 0, 0
    assert not out.any() and not v.any()
    ops.check_status()


FAMILIES = {"llama": {}, "qwen2": dict(attention_bias=True), "qwen3": dict(qk_norm=True),
            "starcoder2": dict(norm_type="layernorm", mlp_gated=False, attention_bias=True, mlp_bias=True, hidden_act="gelu_pytorch_tanh"),
            "gemma-like": dict(model_type="llama", hidden_act="gelu_pytorch_tanh"), "granite": dict(residual_multiplier=0.22, attention_multiplier=0.02)}


@pytest.mark.parametrize("family", list(FAMILIES))
@pytest.mark.parametrize("T,keep", [(40, "compact"), (700, "compact"), (700, True), (1500, False)])
def test_block_in_one_call_is_the_block_launch_by_launch(ops, family, T, keep, monkeypatch):
    """Every form that the native call takes, with kept, partly kept and recomputed activations, against the Python form on the same kernels."""
    from mini_trainer_b200.data.sampler import mb_collate_fn
    from mini_trainer_b200.models import decoder as D, layout as L
    from mini_trainer_b200.models.config import ModelConfig
    kw = dict(model_type=family, vocab_size=64, hidden_size=256, intermediate_size=392, num_hidden_layers=1, num_attention_heads=6, num_key_value_heads=2,
              head_dim=128 if family == "qwen3" else 64)
    cfg = ModelConfig(**{**kw, **FAMILIES[family]})
    torch.manual_seed(T)
    lay = L.GroupLayout("block0", L.block_entries(cfg), 1)
    p = lay.views((torch.randn(lay.padded_numel, device="cuda") * 0.05).bfloat16())
    ids = [torch.randint(0, 64, (n,)) for n in (T // 3, T - T // 3)]
    batch = D.make_packed_batch(mb_collate_fn([{"input_ids": i, "labels": i.clone(), "len": len(i), "num_loss_counted_tokens": len(i)} for i in ids], T), "cuda")
    inv, x, dout = cfg.rope_inv_freq().cuda(), bf(T, 256), bf(T, 256, scale=0.1)
    cls = type(ops)

    def one(native_call):
        done = []
        for name in ("block_forward", "block_backward"):
            real = getattr(cls, name)
            monkeypatch.setattr(cls, name, (lambda self, *a, real=real: done.append(real(self, *a)) or done[-1]) if native_call else lambda self, *a: None)
        g = lay.views(torch.full((lay.padded_numel,), float("nan"), dtype=torch.bfloat16, device="cuda"))
        out, acts, attn = D.block_forward(ops, cfg, p, x, batch, inv, keep=keep, want_attn=not keep)
        if not keep:
            out2, acts, _ = D.block_forward(ops, cfg, p, x, batch, inv, keep=True, saved_attn=attn, need_out=False)
            assert out2 is None
        dx = D.block_backward(ops, cfg, p, g, acts, dout, batch, inv)
        monkeypatch.undo()
        assert not native_call or (len(done) == (2 if keep else 3) and all(d is not None for d in done))
        return out, dx, g

    n0 = ops.launches
    out, dx, g = one(True)
    n1 = ops.launches
    out_ref, dx_ref, g_ref = one(False)
    assert n1 - n0 == ops.launches - n1
    assert torch.equal(out, out_ref)
    # behind the attention backward, whose sum of dQ tiles has no fixed order, up to that
    for a, b in [(dx, dx_ref)] + [(g[n], g_ref[n]) for n in g]:
        assert rel_err(a, b) < 5e-3, family
    assert all(torch.equal(g[n], g_ref[n]) for n in ("wd", "wgu", "wo"))
    ops.check_status()


@pytest.mark.parametrize("form,splits", [("mtb200_gemm2_wide_bf16", 1), ("mtb200_gemm2_wide_bf16", 2), ("mtb200_gemm_n64_bf16", 1), ("mtb200_gemm_n128_bf16", 2)])
@pytest.mark.parametrize("family,keep", [("llama", "compact"), ("starcoder2", True), ("qwen3", False)])
def test_block_in_one_call_on_every_kernel(ops, family, keep, form, splits, monkeypatch):
    """The same with all products on one of the kernels that long and short ones take."""
    from mini_trainer_b200.ops import gemm_plan
    tile = {"mtb200_gemm_n64_bf16": 64, "mtb200_gemm_n128_bf16": 128}.get(form)
    with pytest.MonkeyPatch.context() as plans:
        plans.setattr(gemm_plan, "narrow", lambda *a: (tile, splits) if tile else None)
        plans.setattr(gemm_plan, "wide", lambda *a: 0 if tile else splits)
        plans.setattr(ops, "_gemm_plans", {})
        plans.setattr(ops, "_block_specs", {})
        test_block_in_one_call_is_the_block_launch_by_launch(ops, family, 700, keep, monkeypatch)
        (spec, *_), = ops._block_specs.values()
        assert set(spec.form) == {gemm_plan.FORMS[form]} and set(spec.splits) == {splits} and (spec.act_form == 2) == (tile is None)


def test_block_in_one_call_leaves_to_the_python_form_what_it_does_not_cover(ops):
    from mini_trainer_b200.models import decoder as D, layout as L
    from mini_trainer_b200.models.config import ModelConfig
    batch = D.PackedBatch(*(torch.zeros(8, dtype=torch.int64, device="cuda"),) * 2, torch.arange(8, dtype=torch.int32, device="cuda"), None, [0, 8], 8)
    x = bf(8, 64)
    for change, strided in ((dict(post_norm=True), False), (dict(norm_weight_offset=1.0), False), (dict(mlp_bias=True), False),
                            (dict(residual_multiplier=0.5, attention_bias=True, attention_out_bias=True), True), (dict(head_dim=32), False)):
        known = {k: v for k, v in change.items() if k in ModelConfig.__dataclass_fields__}
        cfg = ModelConfig(**{**dict(vocab_size=64, hidden_size=64, intermediate_size=64, num_hidden_layers=1, num_attention_heads=1, num_key_value_heads=1,
                                    head_dim=64), **known})
        p = L.GroupLayout("block0", L.block_entries(cfg), 1)
        p = p.views(torch.zeros(p.padded_numel, dtype=torch.bfloat16, device="cuda"))
        if strided:
            p["wo"] = bf(64, 128)[:, :64]
        assert ops.block_forward(D.BlockActs, cfg, p, x, batch, None, False, None, False, True) is None


@pytest.mark.parametrize("D,hq,hkv", [(64, 1, 1), (64, 6, 2), (128, 3, 3), (128, 8, 2)])
@pytest.mark.parametrize("lens", [[1], [17, 3], [129], [700, 45, 260]])
def test_attention_backward_zeroes_its_accumulator(ops, lens, D, hq, hkv):
    """Rows that fill no block of the pass that zeroes; the scratch comes from memory that held no numbers."""
    torch.manual_seed(sum(lens))
    T, cu = sum(lens), [0]
    for n in lens:
        cu.append(cu[-1] + n)
    qkv, dout = bf(T, (hq + 2 * hkv) * D), bf(T, hq * D)
    args = (torch.tensor(cu, dtype=torch.int32, device="cuda"), cu, max(lens), hq, hkv, D)
    out, lse = ops.attention(qkv, *args)
    for n in (T * hq * D, T * hq):   # what the call takes its fp32 scratch from
        poison = [torch.full((n,), float("nan"), device="cuda") for _ in range(4)]
        del poison
    got = ops.attention_bwd(dout, qkv, out, lse, *args)
    q32 = qkv.float().requires_grad_()
    q, k, v = q32.split([hq * D, hkv * D, hkv * D], -1)
    ref = []
    for a, b in zip(cu[:-1], cu[1:]):
        heads = [t[a:b].view(b - a, -1, D).transpose(0, 1) for t in (q, k, v)]
        heads[1:] = [t.repeat_interleave(hq // hkv, 0) for t in heads[1:]]
        ref.append(torch.nn.functional.scaled_dot_product_attention(*heads, is_causal=True).transpose(0, 1).reshape(b - a, hq * D))
    torch.cat(ref).backward(dout.float())
    assert rel_err(got, q32.grad) < 1.5e-2
    ops.check_status()


# rows of the experts: none, one, around half and all of a slab's 128 rows, two to five tiles
EXPERT_ROWS = [0, 1, 63, 64, 65, 127, 128, 129, 0, 192, 255, 256, 257, 320, 500, 513, 0]


def _slabs(ops, counts):
    from mini_trainer_b200.ops.native import ExpertSlabs
    E = len(counts)
    starts = [0]
    for c in counts:
        starts.append(starts[-1] + -(-c // 128) * 128)
    cap = -(-(sum(counts) + 127 * E) // 128) * 128
    t = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731
    return ExpertSlabs(t(starts), t(counts), None, None, cap, 1), starts


def _rows(counts, starts, cap, width):
    x = torch.full((cap, width), float("nan"), dtype=torch.bfloat16, device="cuda")   # past the slabs: must not matter
    x[: starts[-1]] = 0
    for c, s in zip(counts, starts):
        x[s:s + c] = bf(c, width)
    return x


@pytest.mark.parametrize("H,F", [(72, 8), (64, 136), (200, 264), (520, 128)])
def test_grouped_products(ops, H, F):
    torch.manual_seed(H + F)
    counts, E = EXPERT_ROWS, len(EXPERT_ROWS)
    sl, starts = _slabs(ops, counts)
    wgu, wd = bf(E, 2 * F, H, scale=0.1), bf(E, H, F, scale=0.1)
    x, y, d = _rows(counts, starts, sl.cap, H), _rows(counts, starts, sl.cap, F), _rows(counts, starts, sl.cap, 2 * F)
    gu = ops.grouped_linear(x, (wgu[0], 2 * F * H), sl)
    for fn in ("silu", "gelu_tanh"):
        pre, act = ops.grouped_linear_act(x, (wgu[0], 2 * F * H), sl, fn)
        for c, s in zip(counts, starts):
            assert torch.equal(pre[s:s + c], gu[s:s + c])
            f = torch.nn.functional.silu(pre[s:s + c, :F].float()) if fn == "silu" else torch.nn.functional.gelu(pre[s:s + c, :F].float(), approximate="tanh")
            if c:
                assert rel_err(act[s:s + c], f * pre[s:s + c, F:].float()) < 4e-3
            assert (act[s + c: s + -(-c // 128) * 128] == 0).all()   # the slab's padding: what a reduction over it reads behind its rows
    dx = ops.grouped_dgrad(d, (wgu[0], 2 * F * H), sl)
    for e, (c, s) in enumerate(zip(counts, starts)):
        if c:
            assert rel_err(gu[s:s + c], x[s:s + c].float() @ wgu[e].float().t()) < 6e-3
            assert max_err(gu[s:s + c], x[s:s + c].float() @ wgu[e].float().t()) < 5e-2
            assert rel_err(dx[s:s + c], d[s:s + c].float() @ wgu[e].float()) < 6e-3
            assert max_err(dx[s:s + c], d[s:s + c].float() @ wgu[e].float()) < 5e-2
    g = torch.full((E, H, F), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.grouped_wgrad(x, y, (g[0], H * F), sl)
    for e, (c, s) in enumerate(zip(counts, starts)):
        want = x[s:s + c].float().t() @ y[s:s + c].float()
        assert (g[e] == 0).all() if c == 0 else rel_err(g[e], want) < 6e-3 and max_err(g[e], want) < 5e-2
    ops.check_status()


@pytest.mark.parametrize("T,E,k,renorm", [(1, 1, 1, True), (300, 8, 2, True), (77, 33, 5, False), (2051, 64, 8, True), (40, 256, 32, True)])
def test_router_in_one_launch(ops, T, E, k, renorm):
    """Against the tensor operations; equal logits (bf16 has few values) go to the lower index."""
    from mini_trainer_b200.ops.native import route_topk
    torch.manual_seed(T)
    logits = torch.randint(-6, 7, (T, E), device="cuda").bfloat16() if T == 77 else bf(T, E, scale=3.0)
    probs, topi, w = route_topk(logits, k, renorm)
    want = torch.softmax(logits.float(), -1)
    assert torch.allclose(probs, want, rtol=1e-5, atol=1e-7)
    by_rank = torch.sort(probs, dim=-1, descending=True, stable=True).indices[:, :k]
    assert torch.equal(topi, by_rank)
    chosen = probs.gather(1, topi)
    assert torch.allclose(w, chosen / chosen.sum(-1, keepdim=True) if renorm else chosen, rtol=1e-5)


def test_router_leaves_other_types_to_the_tensor_operations(ops):
    from mini_trainer_b200.ops.native import route_topk
    assert route_topk(torch.zeros(4, 8, device="cuda"), 2, True) is None
    assert route_topk(bf(4, 257), 2, True) is None and route_topk(bf(4, 64), 33, True) is None and route_topk(bf(8, 8).t(), 2, True) is None


@pytest.mark.parametrize("n,E,k", [(1, 1, 1), (31, 3, 1), (4096, 64, 8), (4104, 7, 3), (16408, 256, 8)])
def test_pairs_are_numbered_in_order_by_expert(ops, n, E, k):
    torch.manual_seed(n)
    topi = (torch.rand(n // k, k, device="cuda") ** 3 * E).long()   # uneven, some experts without pairs
    sl = ops.expert_slabs(topi, E)
    flat = topi.reshape(-1).cpu()
    starts, counts, pair_of, row_of = (t.cpu() for t in (sl.starts, sl.counts, sl.pair_of, sl.row_of))
    at, want = 0, torch.full((sl.cap,), -1, dtype=torch.int32)
    for e in range(E):
        mine = (flat == e).nonzero().flatten().int()
        assert starts[e] == at and counts[e] == len(mine)
        want[at:at + len(mine)] = mine
        at += -(-len(mine) // 128) * 128
    assert starts[E] == at and torch.equal(pair_of, want)
    assert torch.equal(pair_of[row_of.long()], torch.arange(flat.numel(), dtype=torch.int32))
    ops.check_status()


@pytest.mark.parametrize("T,E,k,W", [(5, 2, 1, 8), (130, 4, 3, 2048), (61, 8, 5, 2056), (40, 3, 2, 4104), (33, 2, 2, 8200)])
def test_expert_rows_gathered_weighted_and_combined(ops, T, E, k, W):
    """Widths of a vector, and below and above those at which a row gets more lanes or a second round of them."""
    torch.manual_seed(W)
    topi = torch.stack([torch.randperm(max(E, k), device="cuda")[:k] % E for _ in range(T)])
    sl = ops.expert_slabs(topi, E)
    src, w = bf(T, W), torch.rand(T, k, device="cuda")
    rows = ops.gather_rows(src, sl, 0.5)
    pair = sl.pair_of.long()
    real = pair >= 0
    end = int(sl.starts[-1])
    assert torch.equal(rows[real], (src.float() * 0.5).bfloat16()[pair[real] // k]) and (rows[:end][~real[:end]] == 0).all()
    base, add = bf(T, W), torch.randn(T, W, device="cuda")
    out = ops.combine_rows(rows, sl, base, w=w, add=add, scale=0.7)
    want = base.float() + 0.7 * ((w[..., None] * rows[sl.row_of.long()].view(T, k, W).float()).sum(1) + add)
    assert rel_err(out, want) < 4e-3
    gu, du = bf(sl.cap, 2 * W), bf(sl.cap, W)
    for fn in ("silu", "gelu_tanh"):
        f = torch.nn.functional.silu if fn == "silu" else lambda x: torch.nn.functional.gelu(x, approximate="tanh")
        g32 = gu.float().requires_grad_()
        y = f(g32[:, :W]) * g32[:, W:]
        wr = torch.zeros(sl.cap, device="cuda")
        wr[real] = w.reshape(-1)[pair[real]]
        (y * wr[:, None]).backward(du.float())
        dgu, wact, dw = ops.expert_glu_bwd(du.clone(), gu, w, sl, fn)
        assert rel_err(dgu[:end], g32.grad[:end]) < 6e-3 and rel_err(wact[:end], (y * wr[:, None])[:end]) < 6e-3
        dots = (du.float() * y).sum(-1)
        assert torch.allclose(dw.reshape(-1)[pair[real]], dots[real].detach(), rtol=1e-3, atol=1e-3 * W ** 0.5)
    ops.check_status()


def test_product_with_an_activation_takes_what_the_two_launches_take(ops):
    """Weights that are rows of a wider matrix, and a reduction that is no multiple of eight inside padded rows."""
    torch.manual_seed(0)
    x, w = bf(50, 64), bf(2 * 40, 96, scale=0.2)
    for xs, ws in ((x, w[:, :64]), (x[:, :60], w[:, :60])):
        pre, act = ops.linear_act(xs, ws)
        assert rel_err(pre, xs.float() @ ws.float().t()) < 6e-3
        assert torch.equal(act, ops.swiglu(pre))
    with pytest.raises(AssertionError):
        ops.linear_act(x.float(), w[:, :64].contiguous())


@pytest.mark.parametrize("fn", ["silu", "gelu_tanh"])
@pytest.mark.parametrize("gated", [True, False])
def test_product_with_an_activation_and_weights_that_are_rows_of_a_wider_matrix(ops, gated, fn):
    torch.manual_seed(1)
    f = {"silu": torch.nn.functional.silu, "gelu_tanh": lambda x: torch.nn.functional.gelu(x, approximate="tanh")}[fn]
    x, w = bf(50, 64), bf(80, 96, scale=0.2)
    for xs, ws in ((x, w[:, :64]), (x[:, :60], w[:, :60])):
        pre, act = ops.linear_act(xs, ws, fn, gated)
        assert rel_err(pre, xs.float() @ ws.float().t()) < 6e-3
        p = pre.float()
        assert rel_err(act, f(p[:, :40]) * p[:, 40:] if gated else f(p)) < 4e-3   # one rounding of an fp32 value
    ops.check_status()


def test_activations_that_no_kernel_has_are_refused(ops):
    x, w = bf(8, 64), bf(32, 64)
    sl, _ = _slabs(ops, [3, 5])
    for call in (lambda: ops.linear_act(x, w, "relu"), lambda: ops.linear_act(x, w, "relu", False), lambda: ops.linear_act(x, w.t().contiguous().t(), "relu", False),
                 lambda: ops.grouped_linear_act(bf(sl.cap, 64), (bf(16, 64), 16 * 64), sl, "relu")):
        with pytest.raises(KeyError):
            call()


def test_block_without_memory_for_its_temporaries_goes_launch_by_launch(ops, monkeypatch):
    from mini_trainer_b200.data.sampler import mb_collate_fn
    from mini_trainer_b200.models import decoder as D, layout as L
    from mini_trainer_b200.models.config import ModelConfig
    from mini_trainer_b200.ops import block_exec
    cfg = ModelConfig(model_type="llama", vocab_size=64, hidden_size=128, intermediate_size=256, num_hidden_layers=1, num_attention_heads=2, num_key_value_heads=1,
                      head_dim=64)
    torch.manual_seed(0)
    lay = L.GroupLayout("block0", L.block_entries(cfg), 1)
    p = lay.views((torch.randn(lay.padded_numel, device="cuda") * 0.05).bfloat16())
    g = lay.views(torch.zeros(lay.padded_numel, dtype=torch.bfloat16, device="cuda"))
    ids = torch.randint(0, 64, (90,))
    batch = D.make_packed_batch(mb_collate_fn([{"input_ids": ids, "labels": ids.clone(), "len": 90, "num_loss_counted_tokens": 90}], 90), "cuda")
    x, dout, inv = bf(90, 128), bf(90, 128, scale=0.1), cfg.rope_inv_freq().cuda()
    want, acts, _ = D.block_forward(ops, cfg, p, x, batch, inv, keep="compact")

    class Torch:   # no memory for the workspace, which is the only tensor of bytes
        def __getattr__(self, name):
            return getattr(torch, name)

        def empty(self, *a, dtype=None, **kw):
            if dtype == torch.uint8:
                raise torch.OutOfMemoryError("no memory")
            return torch.empty(*a, dtype=dtype, **kw)
    monkeypatch.setattr(block_exec, "torch", Torch())
    out, acts, _ = D.block_forward(ops, cfg, p, x, batch, inv, keep="compact")
    assert torch.equal(out, want)
    dx = D.block_backward(ops, cfg, p, g, acts, dout, batch, inv)
    assert dx.isfinite().all() and all(t.isfinite().all() for t in g.values())
    ops.check_status()


def test_router_gradient_of_another_type(ops):
    """A gradient tensor that is not of the activations' type gets the converted values; one of another shape is refused."""
    from mini_trainer_b200.models import moe as M
    cfg, p, g, n2, h1, dout = _moe_layer(70, 64, 40, 4, 2, 4)
    got = []
    for dtype in (torch.bfloat16, torch.float32):
        g["router"] = torch.full_like(p["router"], float("nan"), dtype=dtype)
        out, st = M.moe_forward(ops, cfg, p, n2, h1, True, False)
        assert st.slabs is not None
        M.moe_backward(ops, cfg, p, g, st, n2, dout)
        got.append(g["router"])
    assert got[1].dtype == torch.float32 and torch.equal(got[0].float(), got[1])
    for wrong in (torch.empty(5, 64, dtype=torch.bfloat16, device="cuda"), torch.empty(4, 32, dtype=torch.bfloat16, device="cuda")):
        g["router"] = wrong
        with pytest.raises(RuntimeError):
            M.moe_backward(ops, cfg, p, g, st, n2, dout)
    ops.check_status()


@pytest.mark.parametrize("T", [40, 8193])
def test_embedding_gradient_of_strided_ids(ops, T):
    torch.manual_seed(T)
    ids, dx = torch.randint(0, 50, (T, 2), device="cuda"), bf(T, 64)
    got, want = torch.zeros(50, 64, dtype=torch.bfloat16, device="cuda"), torch.zeros(50, 64, dtype=torch.bfloat16, device="cuda")
    ops.embedding_bwd(got, ids[:, 0], dx)
    ops.embedding_bwd(want, ids[:, 0].contiguous(), dx)
    assert torch.equal(got, want)
    ops.check_status()


@pytest.mark.parametrize("fp32", [True, False])
def test_optimizer_over_groups_without_elements(ops, fp32):
    """The norm is written whatever the groups of the first launch hold."""
    sd = torch.float32 if fp32 else torch.bfloat16
    kinds = (torch.float32, sd, sd, torch.float32, torch.bfloat16)
    empty, full = (tuple(torch.ones(n, dtype=d, device="cuda") for d in kinds) for n in (0, 8))
    for groups in ([empty] * 48 + [full], [empty], [empty] * 49, []):
        poison = [torch.full((), float("nan"), device="cuda") for _ in range(8)]
        del poison
        sq = torch.full((1,), 9.0, device="cuda")
        table = ops.group_table(groups)
        ops.add_sumsq_groups(table, sq)
        assert torch.equal(ops.adamw_groups(table, fp32, sq, 1.0, 1e-3, 0.9, 0.95, 1e-8, 0.0, 1), sq.sqrt().squeeze(0))


def test_router_kernel_belongs_to_the_native_backend(ops, monkeypatch):
    """It is launched, and counted, for a layer on that backend only; the plain call stays a chain of differentiable tensor operations."""
    from mini_trainer_b200.models import moe as M
    from mini_trainer_b200.ops import native
    cfg, p, _, n2, h1, _ = _moe_layer(70, 64, 40, 4, 2, 4)
    calls, real = [], ops.lib.mtb200_moe_route

    class Lib:
        def __getattr__(self, name):
            return getattr(ops.lib, name) if name != "mtb200_moe_route" else lambda *a: calls.append("not counted") or real(*a)
    monkeypatch.setattr(native, "_LIB", Lib())
    monkeypatch.setitem(ops._fn, "mtb200_moe_route", lambda *a: calls.append("counted") or real(*a))
    w = p["router"].clone().requires_grad_()
    wt = M.route(cfg, w, n2)[2]
    assert not calls and wt.requires_grad
    wt.sum().backward()
    assert w.grad is not None
    M.moe_forward(TorchOps(), cfg, p, n2, h1, True, False)
    assert not calls
    before = ops.launches
    M.moe_forward(ops, cfg, p, n2, h1, False, False)   # router, slabs, gather, gate/up
    assert calls == ["counted"] and ops.launches == before + 4


# partial last row and column tiles, one or two halves of a wide tile, a last round given out as halves (37 * 256 rows), reductions of one to a few
# k-blocks, split ones; operands of -1, 0, 1: every sum is exact
@pytest.mark.parametrize("M,N", [(33, 264), (300, 520), (256 * 37, 2120), (256 * 37 + 65, 2568)])
@pytest.mark.parametrize("K,splits", [(64, 1), (72, 1), (200, 1), (1032, 2), (1032, 4)])
def test_gemm_wide_tiles_are_exact(ops, M, N, K, splits, monkeypatch):
    from mini_trainer_b200.ops import gemm_plan
    monkeypatch.setattr(gemm_plan, "narrow", lambda *a: None)
    monkeypatch.setattr(gemm_plan, "wide", lambda M, N, K, *a: splits if 2 * -(-M // 256) * -(-N // 256) * splits <= 1024 else 1)
    monkeypatch.setattr(ops, "_gemm_plans", {})
    names = []
    monkeypatch.setattr(ops, "_call", lambda name, *a, call=ops._call, **kw: names.append(name) or call(name, *a, **kw))
    rows = -(-M // 8) * 8
    a, b = _ints(rows, K), _ints(N, K)
    at, bt = a.t().contiguous(), b.t().contiguous()
    want, res, bias = a.float() @ b.float().t(), _ints(rows, N), _ints(N)
    for a_mn, b_mn in ((False, False), (False, True), (True, False), (True, True)):
        m = rows if a_mn else M
        for dt in (torch.bfloat16, torch.float32):
            for extra in (False, True):
                out = torch.full((m, N), float("nan"), dtype=dt, device="cuda")
                kw = dict(residual=res[:m].to(dt), bias=bias) if extra else {}
                ops.gemm(at if a_mn else a, a_mn, bt if b_mn else b, b_mn, out, m, N, K, **kw)
                ref = want[:m] + (res[:m].float() + bias.float() if extra else 0.0)
                assert torch.equal(out, ref.to(dt)), (a_mn, b_mn, dt, extra)
    assert set(names) == {"mtb200_gemm2_wide_bf16"}
    ops.check_status()


@pytest.mark.parametrize("form", [-1, 3, 4])
def test_activation_behind_a_product_refuses_forms_without_that_epilogue(ops, form):
    """Narrow tiles are numbers 3 and 4 of a plan's kernels."""
    x, w, pre, act = bf(128, 64), bf(128, 64), bf(128, 128), bf(128, 64)
    kept = pre.clone()
    with pytest.raises(RuntimeError, match="code -10"):
        ops._call("mtb200_gemm_act", x.data_ptr(), 64, w.data_ptr(), pre.data_ptr(), act.data_ptr(), None, 1, 0, 128, 64, 64, form, ops.status.data_ptr(), ops._st())
    assert torch.equal(pre, kept)


@pytest.mark.parametrize("T,F,K", [(33, 136, 264), (1000, 1000, 512), (256 * 37, 1096, 72)])
@pytest.mark.parametrize("fn", ["silu", "gelu_tanh"])
def test_wide_tiles_epilogues_match_the_other_kernels(ops, T, F, K, fn, monkeypatch):
    """Activation and softmax statistics behind wide tiles: the same bits as behind 256 x 256 tiles."""
    from mini_trainer_b200.ops import gemm_plan
    if ops.cta_pairs() == 0:
        pytest.skip("no clusters of two CTAs on this device")
    torch.manual_seed(T + F)
    x, w, bias = bf(T, K), bf(2 * F, K, scale=K ** -0.5), bf(2 * F)
    got, ran = [], []
    monkeypatch.setattr(ops, "_call", lambda name, *a, call=ops._call, **kw: ran.append((name, a[11] if name == "mtb200_gemm_act" else None)) or call(name, *a, **kw))
    monkeypatch.setattr(gemm_plan, "narrow", lambda *a: None)
    for splits in (1, 0):
        monkeypatch.setattr(gemm_plan, "wide", lambda *a: splits)
        monkeypatch.setattr(gemm_plan, "choose", lambda *a: (True, 1))
        monkeypatch.setattr(ops, "_gemm_plans", {})
        out, stats = torch.empty(T, 2 * F, dtype=torch.bfloat16, device="cuda"), torch.full((T, -(-2 * F // 256), 2), float("nan"), device="cuda")
        ops.gemm(x, False, w, False, out, T, 2 * F, K, alpha=0.5, stats=stats)
        got.append([*ops.linear_act(x, w, fn), out, stats] + ([*ops.linear_act(x, w, fn, gated=False, bias=bias)] if fn == "gelu_tanh" else []))
    for name, form in (("mtb200_gemm2_wide_bf16", 2), ("mtb200_gemm2_bf16", 1)):
        n = 3 if fn == "gelu_tanh" else 2
        assert ran[:n] == [(name, None)] + [("mtb200_gemm_act", form)] * (n - 1)
        del ran[:n]
    for g, h in zip(*got):
        assert torch.equal(g, h)
    ops.check_status()


# slabs of which the last tile holds 128 rows or 256, experts without rows, partial tiles of every output, a reduction of one k-block
@pytest.mark.parametrize("T,E,k,popular", [(1, 4, 2, 4), (900, 48, 2, 24), (1500, 5, 2, 4), (260, 3, 1, 2)])
@pytest.mark.parametrize("H,F", [(64, 72), (648, 520), (1040, 264)])
def test_grouped_products_in_wide_tiles_match(ops, T, E, k, popular, H, F, monkeypatch):
    from mini_trainer_b200.ops import gemm_plan
    if ops.cta_pairs() == 0:
        pytest.skip("no clusters of two CTAs on this device")
    ran = []
    monkeypatch.setattr(ops, "_call", lambda name, *a, call=ops._call, **kw: (name == "mtb200_gemm_grouped" and ran.append(a[8]), call(name, *a, **kw))[1])
    torch.manual_seed(T + H)
    topi = torch.stack([torch.randperm(popular, device="cuda")[:k] for _ in range(T)]) * (E // popular)
    sl = ops.expert_slabs(topi, E)
    x, d = ops.gather_rows(bf(T, H), sl), ops.gather_rows(bf(T, 2 * F), sl)
    w = bf(E, 2 * F, H, scale=H ** -0.5)
    got = []
    for wide in (False, True):
        monkeypatch.setattr(gemm_plan, "grouped_wide", lambda *a: wide)
        monkeypatch.setattr(ops, "_gemm_plans", {})
        dw = torch.full((E, 2 * F, H), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.grouped_wgrad(d, x, (dw[0], 2 * F * H), sl)
        stack = (w[0], 2 * F * H)
        rows = int(sl.starts[-1])
        got.append([dw, *(t[:rows] for t in (ops.grouped_linear(x, stack, sl), *ops.grouped_linear_act(x, stack, sl), *ops.grouped_linear_act(x, stack, sl, "gelu_tanh"),
                                             ops.grouped_dgrad(d, stack, sl)))])
    assert ran == [2, 0, 3, 3, 1, 6, 4, 7, 7, 5]
    for a, b in zip(*got):
        assert not a.isnan().any() and torch.equal(a, b)
    ops.check_status()


# partial last row and column tiles, one tile, a ring that is not filled once and one that is filled several times, split reductions; every sum is exact
@pytest.mark.parametrize("tile", [64, 128])
@pytest.mark.parametrize("M,N", [(1, 8), (33, 72), (300, 136), (129, 1000), (1160, 520)])
@pytest.mark.parametrize("K,splits", [(64, 1), (200, 1), (1600, 1), (1032, 2), (3000, 7)])
def test_gemm_narrow_tiles_are_exact(ops, tile, M, N, K, splits, monkeypatch):
    from mini_trainer_b200.ops import gemm_plan
    monkeypatch.setattr(gemm_plan, "narrow", lambda *a: (tile, splits))
    monkeypatch.setattr(ops, "_gemm_plans", {})
    names = []
    monkeypatch.setattr(ops, "_call", lambda name, *a, call=ops._call, **kw: names.append(name) or call(name, *a, **kw))
    rows = -(-M // 8) * 8
    a, b = _ints(rows, K), _ints(N, K)
    at, bt = a.t().contiguous(), b.t().contiguous()
    want, res, bias = a.float() @ b.float().t(), _ints(rows, N), _ints(N)
    for a_mn, b_mn in ((False, False), (False, True), (True, False), (True, True)):
        m = rows if a_mn else M
        for dt in (torch.bfloat16, torch.float32):
            for extra in (False, True):
                out = torch.full((m, N), float("nan"), dtype=dt, device="cuda")
                kw = dict(residual=res[:m].to(dt), bias=bias) if extra else {}
                ops.gemm(at if a_mn else a, a_mn, bt if b_mn else b, b_mn, out, m, N, K, **kw)
                assert torch.equal(out, (want[:m] + (res[:m].float() + bias.float() if extra else 0.0)).to(dt)), (a_mn, b_mn, dt, extra)
    assert set(names) == {f"mtb200_gemm_n{tile}_bf16"}
    ops.check_status()
