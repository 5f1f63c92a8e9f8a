"""Numerics of every hand-written CUDA kernel against a plain PyTorch fp32 reference of the same op.

Tolerances: outputs stored in bf16 are compared with rtol ~ 2 bf16 ulps of the reference magnitude;
fp32 outputs (log-probs, entropy, optimizer state) with the tolerances the reference uses for its
fused kernels (tests/utils/test_linear_cross_entropy.py: logprob atol 1e-3 / rtol 2e-4, entropy atol 5e-3).
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf16_close(got, ref, scale=None, ulps=4.0):
    got, ref = got.float(), ref.float().to(got.device)
    scale = ref.abs().max().item() if scale is None else scale
    err = (got - ref).abs().max().item()
    assert err <= ulps * 2 ** -8 * scale + 1e-6, f"max err {err} vs scale {scale}"


@pytest.fixture(autouse=True)
def _status_clean():
    from verl_b200.ops import _lib

    _lib.load()
    yield
    code, blk, detail = _lib.read_status()
    assert code == 0, f"kernel status word reports error {code} (block {blk}, detail {detail})"


@pytest.mark.parametrize("mode", ["tn", "nn", "wg", "an"])
@pytest.mark.parametrize("shape", [(128, 256, 64), (200, 264, 136), (1024, 3584, 3584), (777, 128, 1000),
                                   (8, 1024, 512), (384, 72, 256)])
def test_gemm_layouts(mode, shape):
    from verl_b200.ops import gemm

    torch.manual_seed(0)
    M, N, K = shape
    a_mn, b_mn = {"tn": (False, False), "nn": (False, True), "wg": (True, True), "an": (True, False)}[mode]
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("MN-major operand needs a row stride that is a multiple of 8")
    A = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    B = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    ref = A.float() @ B.float().t()
    out = gemm(A.t().contiguous() if a_mn else A, B.t().contiguous() if b_mn else B, a_mn=a_mn, b_mn=b_mn)
    _bf16_close(out, ref)


@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 24, 25, 32, 33])
@pytest.mark.parametrize("N,K", [(1, 8), (15, 72), (33, 520), (1153, 896), (4745, 2056), (130, 4872), (264, 8200), (37889, 64)])
def test_gemm_few_rows(M, N, K):
    """Few rows of A: every group of rows and of columns with its remainders, strided operands and results, both result types."""
    from verl_b200.ops import gemm

    torch.manual_seed(M * 7 + N)
    A = torch.randn(M, K + 16, device="cuda").bfloat16()[:, 8 : K + 8]
    B = torch.randn(N, K + 8, device="cuda").bfloat16()[:, :K]
    bias = torch.randn(N, device="cuda").bfloat16()
    ref = A.double() @ B.double().t()
    # an fp32 sum of K products: at most K roundings of 2^-24 of the sum of their magnitudes
    bound = (A.double().abs() @ B.double().abs().t()) * K * 2.0 ** -24
    out = torch.full((M, N + 5), 7.0, device="cuda")
    gemm(A, B, out=out[:, :N])
    assert ((out[:, :N] - ref).abs() <= bound).all() and (out[:, N:] == 7.0).all()
    got, want = gemm(A, B, bias=bias).double(), ref + bias.double()
    assert ((got - want).abs() <= bound + 2.0 ** -8 * want.abs() + 2.0 ** -23).all()


@pytest.mark.parametrize("M", [1, 8, 16, 32])
def test_gemm_few_rows_of_operands_just_written(M):
    """Both operands of a few-row product come from the kernels right before it, into the same buffers again and again: the bits are
    those of the ordinary stream order, where no kernel starts before the one before it has ended."""
    from verl_b200 import ops
    from verl_b200.ops import _lib

    gen = torch.Generator(device="cuda").manual_seed(M)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()  # noqa: E731
    K, N = 1024, 264
    xs, ys, wa, wb = rnd(12, M, 512), rnd(12, N, 512), rnd(K, 512), rnd(K, 512)

    def passes():
        a, b = (torch.zeros(r, K, device="cuda", dtype=torch.bfloat16) for r in (M, N))
        outs = []
        for x, y in zip(xs, ys):
            ops.gemm(y, wb, out=b)  # the matrix, by the tile kernel
            ops.gemm(x, wa, out=a)  # the rows, by the few-row kernel itself
            outs.append(ops.gemm(a, b, out_dtype=torch.float32))
            ops.gemm(y[:M], wb, out=b[:M])  # part of the matrix by the kernel right before
            outs.append(ops.gemm(a, b, out_dtype=torch.float32))
        return torch.stack(outs)

    try:
        _lib.set_pdl(False)
        want = passes()
    finally:
        _lib.set_pdl(True)
    for _ in range(3):
        assert torch.equal(passes(), want)


@pytest.mark.parametrize("T,N", [(1, 2), (7, 34), (8, 512), (511, 514), (512, 1026), (3000, 4608), (5, 33)])
def test_colsum(T, N):
    from verl_b200.ops.gemm import colsum

    torch.manual_seed(T)
    x = torch.randn(T, N + 2, device="cuda").bfloat16()[:, :N]
    ref = x.double().sum(0)
    bound = x.double().abs().sum(0) * T * 2.0 ** -24 + 2.0 ** -8 * ref.abs()  # an fp32 sum of T terms, one rounding to bf16
    assert ((colsum(x).double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 600, 2305])
@pytest.mark.parametrize("I,K", [(8, 8), (24, 72), (4864, 896), (2632, 584), (18944, 264)])
def test_linear_swiglu(M, I, K):
    """Few rows, CTA pairs (ragged rows, columns and K) and sizes of neither: the bits of a product and an activation of its own."""
    from verl_b200 import ops

    torch.manual_seed(M + I)
    x = torch.randn(M, K + 8, device="cuda").bfloat16()[:, :K]
    w = (torch.randn(2 * I, K, device="cuda") * 2 * K ** -0.5).bfloat16()
    with torch.no_grad():
        got = ops.linear_swiglu(x, w)
        assert torch.equal(got, ops.swiglu(ops.gemm(x, w)))
        gate, up = (x.double() @ w.double().t()).chunk(2, -1)
        ref = torch.nn.functional.silu(gate) * up
        # gate and up rounded (2^-8 each, silu's slope is below 1.1) after fp32 sums of K products, the result rounded
        silu, sums = torch.nn.functional.silu(gate).abs(), (x.double().abs() @ w.double().abs().t()) * K * 2.0 ** -24
        e_gate, e_up = (2.0 ** -8 * t.abs() + e for t, e in zip((gate, up), sums.chunk(2, -1)))
        bound = 1.05 * (1.1 * e_gate * up.abs() + silu * e_up + 1.1 * e_gate * e_up + 2.0 ** -8 * ref.abs()) + 1e-30
        assert ((got.double() - ref).abs() <= bound).all()
    recorded = ops.linear_swiglu(x, w.clone().requires_grad_(True))
    assert recorded.requires_grad and torch.equal(recorded, got)


def test_gemm_fp32_accumulate_and_bias():
    from verl_b200.ops import gemm

    torch.manual_seed(1)
    M, N, K = 256, 520, 384
    A = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    B = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    C = torch.full((M, N), 3.0, device="cuda")
    gemm(A, B, out=C, accumulate=True)
    torch.testing.assert_close(C, A.float() @ B.float().t() + 3.0, atol=1e-3, rtol=1e-5)
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    _bf16_close(gemm(A, B, bias=bias), A.float() @ B.float().t() + bias.float())


@pytest.mark.parametrize("M,N,K,mode", [(128, 3584, 18944, "tn"), (64, 4608, 3584, "tn"), (7, 520, 2048, "tn"),
                                        (128, 1024, 4096, "nn"), (200, 640, 8192, "tn"), (128, 3584, 3584, "tn"),
                                        (256, 2304, 3584, "tn"), (128, 4608, 3584, "tn"), (100, 1796, 1800, "tn")])
def test_gemm_split_k(M, N, K, mode):
    """Skinny problems split K: over the CTAs of a cluster with the reduction through distributed shared memory
    (uneven row shares when the slice count does not divide 128, ragged N and K), or, with fp32 accumulation into C,
    over fp32 slices in a workspace. Same numbers as the fp32 reference, bit-identical between calls, bias handled by
    the reducing CTA."""
    from verl_b200.ops import gemm, _lib

    torch.manual_seed(3)
    A = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    B = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) * 0.05
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    ref = A.float() @ B.float().t()
    Bm = B.t().contiguous() if mode == "nn" else B
    o1 = gemm(A, Bm, b_mn=(mode == "nn"), bias=bias)
    o2 = gemm(A, Bm, b_mn=(mode == "nn"), bias=bias)
    assert _lib.read_status("cuda")[0] == 0
    _bf16_close(o1, ref + bias.float())
    assert torch.equal(o1, o2)
    C = torch.full((M, N), 2.0, device="cuda")
    gemm(A, Bm, b_mn=(mode == "nn"), out=C, accumulate=True)
    torch.testing.assert_close(C, ref + 2.0, atol=2e-2, rtol=1e-4)


@pytest.mark.parametrize("mode", ["tn", "nn", "wg", "an"])
def test_gemm_cta_pair_path(mode):
    """Large problems run on CTA pairs (256 x 256 tiles, one MMA for two SMs). Odd 128-row block count, ragged N and
    K, every operand layout, bias and fp32 accumulation."""
    from verl_b200.ops import gemm, _lib

    torch.manual_seed(4)
    M, N, K = 4224, 2632, 584
    a_mn, b_mn = {"tn": (False, False), "nn": (False, True), "wg": (True, True), "an": (True, False)}[mode]
    A = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    B = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) * 0.1
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    ref = A.float() @ B.float().t()
    Am = A.t().contiguous() if a_mn else A
    Bm = B.t().contiguous() if b_mn else B
    out = gemm(Am, Bm, a_mn=a_mn, b_mn=b_mn, bias=bias)
    assert _lib.read_status("cuda")[0] == 0
    _bf16_close(out, ref + bias.float())
    assert torch.equal(out, gemm(Am, Bm, a_mn=a_mn, b_mn=b_mn, bias=bias))
    C = torch.full((M, N), -1.0, device="cuda")
    gemm(Am, Bm, a_mn=a_mn, b_mn=b_mn, out=C, accumulate=True)
    torch.testing.assert_close(C, ref - 1.0, atol=2e-2, rtol=1e-4)


def test_gemm_deterministic():
    from verl_b200.ops import gemm

    A = torch.randn(512, 1024, device="cuda", dtype=torch.bfloat16)
    B = torch.randn(768, 1024, device="cuda", dtype=torch.bfloat16)
    assert torch.equal(gemm(A, B), gemm(A, B))


def test_linear_autograd_matches_torch():
    from verl_b200 import ops

    torch.manual_seed(2)
    x = torch.randn(300, 512, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(264, 512, device="cuda") * 0.05).bfloat16().requires_grad_(True)
    b = torch.randn(264, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    dy = torch.randn(300, 264, device="cuda", dtype=torch.bfloat16)
    ops.linear(x, w, b).backward(dy)
    xr, wr, br = (t.detach().float().requires_grad_(True) for t in (x, w, b))
    torch.nn.functional.linear(xr, wr, br).backward(dy.float())
    _bf16_close(x.grad, xr.grad)
    _bf16_close(w.grad, wr.grad)
    _bf16_close(b.grad, br.grad)
    # fused accumulation into an fp32 main_grad
    w2 = w.detach().clone().requires_grad_(True)
    w2.main_grad = torch.ones(w2.shape, device="cuda")
    ops.linear(x.detach(), w2, None).backward(dy)
    assert w2.grad is None
    torch.testing.assert_close(w2.main_grad, wr.grad + 1.0, atol=2e-3, rtol=1e-4)


@pytest.mark.parametrize("T,H,V,temp", [(300, 256, 2048, 1.0), (1937, 3584, 152064, 0.7), (129, 1024, 32000, 1.5)])
def test_fused_lmhead_forward_backward(T, H, V, temp):
    from verl_b200 import ops

    torch.manual_seed(3)
    hid = torch.randn(T, H, device="cuda").bfloat16().requires_grad_(True)
    w = (torch.randn(V, H, device="cuda") * 0.02).bfloat16().requires_grad_(True)
    labels = torch.randint(0, V, (T,), device="cuda")
    lp, ent = ops.lmhead_logprob_entropy(hid, w, labels, temp)
    hr, wr = hid.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    logits = (hr @ wr.t()) / temp
    lse = torch.logsumexp(logits, -1)
    lp_ref = logits.gather(1, labels[:, None])[:, 0] - lse
    ent_ref = lse - (torch.softmax(logits, -1) * logits).sum(-1)
    torch.testing.assert_close(lp, lp_ref, atol=1e-3, rtol=2e-4)
    torch.testing.assert_close(ent, ent_ref, atol=5e-3, rtol=1e-3)
    g_lp = torch.randn(T, device="cuda")
    g_ent = torch.randn(T, device="cuda") * 0.1
    (lp * g_lp + ent * g_ent).sum().backward()
    (lp_ref * g_lp + ent_ref * g_ent).sum().backward()
    _bf16_close(hid.grad, hr.grad, ulps=8)
    _bf16_close(w.grad, wr.grad, ulps=8)


def test_rmsnorm_forward_backward():
    from verl_b200 import ops

    torch.manual_seed(4)
    rows, H = 1000, 3584
    x = torch.randn(rows, H, device="cuda").bfloat16().requires_grad_(True)
    res = torch.randn(rows, H, device="cuda").bfloat16().requires_grad_(True)
    w = (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16().requires_grad_(True)
    y, h = ops.rmsnorm(x, w, 1e-6, res)
    dy, dh = torch.randn_like(y), torch.randn_like(h)
    torch.autograd.backward([y, h], [dy, dh])
    xr, rr, wr = (t.detach().float().requires_grad_(True) for t in (x, res, w))
    hr = (xr + rr) + ((xr + rr).bfloat16().float() - (xr + rr)).detach()  # bf16-rounded value, identity gradient
    yr = hr * torch.rsqrt(hr.pow(2).mean(-1, keepdim=True) + 1e-6) * wr
    torch.autograd.backward([yr, hr], [dy.float(), dh.float()])
    _bf16_close(y, yr)
    _bf16_close(h, hr)
    _bf16_close(x.grad, xr.grad)
    _bf16_close(res.grad, rr.grad)
    _bf16_close(w.grad, wr.grad, ulps=8)


def test_swiglu_and_rope():
    from verl_b200 import ops

    torch.manual_seed(5)
    gu = torch.randn(512, 2 * 1184, device="cuda").bfloat16().requires_grad_(True)
    do = torch.randn(512, 1184, device="cuda").bfloat16()
    out = ops.swiglu(gu)
    out.backward(do)
    gr = gu.detach().float().requires_grad_(True)
    ref = torch.nn.functional.silu(gr[:, :1184]) * gr[:, 1184:]
    ref.backward(do.float())
    _bf16_close(out, ref)
    _bf16_close(gu.grad, gr.grad)

    T, Hq, Hk, D = 333, 28, 4, 128
    qkv = torch.randn(T, (Hq + 2 * Hk) * D, device="cuda").bfloat16()
    pos = torch.randint(0, 4096, (T,), device="cuda")
    cos_t, sin_t = ops.rope_tables(D, 4096, 1e6, "cuda")
    ref = ops.rope_qkv(qkv.cpu().float(), pos.cpu(), cos_t.cpu(), sin_t.cpu(), Hq, Hk, D)
    src = qkv.clone().requires_grad_(True)
    got = ops.rope_qkv(src * 1.0, pos, cos_t, sin_t, Hq, Hk, D)
    _bf16_close(got, ref)
    # backward is the transpose rotation: <rope(x), g> == <x, rope^T(g)>
    g = torch.randn_like(got)
    got.backward(g)
    lhs = (got.float() * g.float()).sum()
    rhs = (qkv.float() * src.grad.float()).sum()
    assert abs(lhs.item() - rhs.item()) <= 2e-2 * abs(lhs.item()) + 1.0


def test_embedding_and_adamw_and_norms():
    from verl_b200 import ops

    torch.manual_seed(6)
    W = torch.randn(5000, 512, device="cuda").bfloat16().requires_grad_(True)
    ids = torch.randint(0, 5000, (777,), device="cuda")
    out = ops.embedding(ids, W)
    assert torch.equal(out, W[ids])
    dy = torch.randn_like(out)
    out.backward(dy)
    ref = torch.zeros(5000, 512, device="cuda").index_add_(0, ids, dy.float())
    _bf16_close(W.grad, ref)

    n = 1_000_003
    p32, g = torch.randn(n, device="cuda"), torch.randn(n, device="cuda")
    m, v = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    p16 = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    pr = torch.nn.Parameter(p32.clone())
    opt = torch.optim.AdamW([pr], lr=1e-3, betas=(0.9, 0.999), eps=1e-8, weight_decay=0.01)
    for step in (1, 2, 3):
        pr.grad = g.clone()
        opt.step()
        ops.adamw_step(p32, g, m, v, p16, lr=1e-3, betas=(0.9, 0.999), eps=1e-8, weight_decay=0.01, step=step)
    torch.testing.assert_close(p32, pr.data, atol=2e-6, rtol=1e-5)
    _bf16_close(p16, pr.data)
    ss = torch.zeros(1, device="cuda")
    ops.sumsq_into(g, ss)
    torch.testing.assert_close(ss[0], g.pow(2).sum(), rtol=1e-4, atol=0)
    scale, skip, norm = torch.zeros(1, device="cuda"), torch.zeros(1, device="cuda", dtype=torch.int32), torch.zeros(1, device="cuda")
    ops.clip_coef(ss, 1.0, 0.5, scale, skip, norm)
    gn = g.norm().item() * 0.5
    assert abs(norm.item() - gn) < 1e-2 and skip.item() == 0 and abs(scale.item() - 0.5 / (gn + 1e-6)) < 1e-6


def test_ppo_loss_fused_matches_torch():
    from verl_b200 import ops
    from verl_b200.trainer.ppo import core_algos

    torch.manual_seed(7)
    B, T = 16, 200
    logp = (torch.randn(B, T, device="cuda") * 0.5 - 2).requires_grad_(True)
    old = logp.detach() + torch.randn(B, T, device="cuda") * 0.3
    ref_lp = logp.detach() + torch.randn(B, T, device="cuda") * 0.2
    adv = torch.randn(B, T, device="cuda")
    mask = (torch.rand(B, T, device="cuda") > 0.3).float()
    ent = torch.rand(B, T, device="cuda").requires_grad_(True)
    loss, sums = ops.ppo_loss_fused(logp, old, adv, mask, entropy=ent, ref_logp=ref_lp, clip_low=0.2, clip_high=0.28,
                                    clip_c=3.0, kl_coef=0.01, kl_type="low_var_kl", entropy_coeff=0.001)
    loss.backward()
    lr, er = logp.detach().clone().requires_grad_(True), ent.detach().clone().requires_grad_(True)
    pg, clipfrac, ppo_kl, clipfrac_lower = core_algos.compute_policy_loss(
        old, lr, adv, mask, cliprange=0.2, cliprange_low=0.2, cliprange_high=0.28, clip_ratio_c=3.0,
        loss_agg_mode="token-mean")
    kld = core_algos.kl_penalty(lr, ref_lp, "low_var_kl")
    kl_loss = core_algos.agg_loss(kld, mask, "token-mean")
    ent_loss = core_algos.agg_loss(er, mask, "token-mean")
    ref_loss = pg - 0.001 * ent_loss + 0.01 * kl_loss
    ref_loss.backward()
    torch.testing.assert_close(loss, ref_loss, atol=1e-5, rtol=1e-4)
    torch.testing.assert_close(logp.grad, lr.grad, atol=1e-7, rtol=1e-3)
    torch.testing.assert_close(ent.grad, er.grad, atol=1e-8, rtol=1e-3)
    n = sums[6]
    torch.testing.assert_close(sums[1] / n, clipfrac, atol=1e-5, rtol=1e-4)
    torch.testing.assert_close(sums[2] / n, ppo_kl, atol=1e-5, rtol=1e-4)
    torch.testing.assert_close(sums[3] / n, clipfrac_lower, atol=1e-5, rtol=1e-4)


def test_gae_and_grpo_match_core_algos():
    from verl_b200 import ops
    from verl_b200.trainer.ppo import core_algos

    torch.manual_seed(8)
    B, T = 37, 129
    r, v = torch.randn(B, T, device="cuda"), torch.randn(B, T, device="cuda")
    mk = (torch.rand(B, T, device="cuda") > 0.2).float()
    adv, ret = ops.gae(r, v, mk, 0.99, 0.95)
    adv_ref, ret_ref = core_algos.compute_gae_advantage_return(r.cpu(), v.cpu(), mk.cpu(), 0.99, 0.95, whiten=False)
    torch.testing.assert_close(adv.cpu(), adv_ref, atol=1e-4, rtol=1e-4)
    torch.testing.assert_close(ret.cpu(), ret_ref, atol=1e-4, rtol=1e-4)

    import numpy as np

    scores_tok = torch.zeros(B, T)
    scores = torch.randn(B)
    lens = mk.cpu().sum(-1).long().clamp(min=1)
    gid = torch.randint(0, 9, (B,))
    gid[0] = 20  # singleton group
    for b in range(B):
        scores_tok[b, 0] = scores[b]
    ref, _ = core_algos.compute_grpo_outcome_advantage(scores_tok, mk.cpu(), np.array(gid.tolist()))
    got = ops.grpo_advantage(scores.cuda(), gid.cuda(), mk, 21)
    torch.testing.assert_close(got.cpu(), ref, atol=1e-4, rtol=1e-4)


def test_sampler_distribution_and_modes():
    from verl_b200 import ops

    torch.manual_seed(9)
    V, n = 1000, 4096
    logits = torch.randn(1, V, device="cuda").repeat(n, 1).contiguous()
    step = torch.zeros(1, device="cuda", dtype=torch.long)
    tok, lp = ops.sample(logits, seed=1234, step=step)
    p = torch.softmax(logits[0], -1)
    freq = torch.bincount(tok, minlength=V).float() / n
    assert (freq - p).abs().sum().item() / 2 < 0.25
    torch.testing.assert_close(lp, torch.log(p)[tok], atol=1e-5, rtol=1e-5)
    tok2, _ = ops.sample(logits, seed=1234, step=step)
    assert torch.equal(tok, tok2)  # same seed and step -> same draw
    step += 1
    tok3, _ = ops.sample(logits, seed=1234, step=step)
    assert not torch.equal(tok, tok3)
    tok, _ = ops.sample(logits, temperature=torch.zeros(n, device="cuda"), seed=1, step=step)
    assert bool((tok == logits[0].argmax()).all())
    tok, lp = ops.sample(logits, top_k=torch.full((n,), 5, device="cuda", dtype=torch.int32), seed=7, step=step)
    top5 = logits[0].topk(5)
    assert set(tok.unique().tolist()) <= set(top5.indices.tolist())
    torch.testing.assert_close(lp, torch.log_softmax(top5.values, -1)[(tok[:, None] == top5.indices[None]).float().argmax(-1)],
                               atol=1e-4, rtol=1e-4)
    tok, _ = ops.sample(logits, top_p=torch.full((n,), 0.5, device="cuda"), seed=7, step=step)
    sp, si = p.sort(descending=True)
    kk = int((sp.cumsum(0) < 0.5).sum().item()) + 1
    assert set(tok.unique().tolist()) <= set(si[:kk].tolist())
    # bf16 logits
    tok, _ = ops.sample(logits.bfloat16(), temperature=torch.zeros(n, device="cuda"), seed=1, step=step)
    assert bool((tok == logits[0].bfloat16().float().argmax()).all())


@pytest.mark.parametrize("V", [7, 1023, 1025, 4099, 32771, 152064])  # one block, the guesses' limit, a ragged last group, clusters
@pytest.mark.parametrize("B", [1, 3, 75, 150])                      # 8, 4, 1 blocks per row and more rows than SMs
@pytest.mark.parametrize("k,p", [(-1, 0.9), (5, 1.0), (12, 0.8), (3, 0.99)])
def test_sampler_support_and_logprob(V, B, k, p):
    """Tokens come from the smaller of the top-k set and the nucleus; log-probs are those of the renormalised support. The strong
    tokens are 0.3 apart (so no set hangs on rounding), the tail together weighs less than a thousandth of the last of them."""
    from verl_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(V + B)
    n = min(V, 40)
    logits = torch.full((B, V), -40.0, device="cuda")
    where = torch.stack([torch.randperm(V, device="cuda", generator=g)[:n] for _ in range(B)])
    logits.scatter_(1, where, -0.3 * torch.arange(n, device="cuda").repeat(B, 1))
    step = torch.zeros(1, dtype=torch.long, device="cuda")
    tok, lp = ops.sample(logits, top_k=torch.full((B,), k, dtype=torch.int32, device="cuda"), top_p=torch.full((B,), p, device="cuda"),
                         seed=3, step=step)
    d = torch.softmax(logits[0].double(), -1).sort(descending=True).values
    size = V
    if 0 < k < V:
        size = k
    if p < 1:
        size = min(size, int((d.cumsum(0) < p).sum()) + 1)
    keep = where[:, :size]
    hit = keep == tok[:, None]
    assert bool(hit.any(1).all())
    ref = torch.log_softmax(-0.3 * torch.arange(size, device="cuda", dtype=torch.float64), -1)[hit.float().argmax(1)]
    assert float((lp - ref).abs().max()) < 2e-5  # fast exp, log and fp32 sums of up to 40 terms


def _sampler_bounds(logits, k, p):
    """Of one row in fp64: log-probs, and which tokens are inside for sure and at most. The threshold is searched in fp32: probabilities
    (fast exp, 2^-21 and the sum's error) within 1e-4 of it, and masses within 1e-5 of ``p``, may fall on either side."""
    lp = torch.log_softmax(logits.double(), -1)
    q = lp.exp()
    d = q.sort(descending=True).values
    cum = d.cumsum(0)

    def threshold(mass):
        thr = d[k - 1] if 0 < k < d.numel() else d[-1] * 0
        return torch.maximum(thr, d[min(int((cum < mass).sum()), d.numel() - 1)]) if p < 1 else thr

    at_most = q >= threshold(p + 1e-5) * (1 - 1e-4) - d[0] * 2.0 ** -29
    return lp, q >= threshold(p - 1e-5) * (1 + 1e-4), at_most


@pytest.mark.parametrize("V,B", [(1024, 3), (1025, 3), (4099, 3), (32771, 3), (152064, 3), (152064, 40), (32771, 150)])  # 1 to 8 blocks per row
@pytest.mark.parametrize("kind,k,p", [("flat", -1, 0.9), ("flat", 900, 1.0), ("flat", 5000, 1.0), ("flat", 3000, 0.5), ("equal", 50, 1.0),
                                      ("equal", -1, 0.3), ("equal", 7, 0.99), ("ties", 1000, 1.0), ("ties", -1, 0.6), ("steps", 2500, 1.0)])
def test_sampler_wide_supports(V, B, kind, k, p):
    """Supports above the short list (1024 tokens): guesses that narrow, counting on the row, the hand-over of what lies between the
    bounds, and more equal probabilities at the threshold than the list holds."""
    from verl_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(V + B)
    logits = torch.randn(B, V, device="cuda", generator=gen)
    if kind == "flat":
        logits *= 0.5
    elif kind == "equal":
        logits[:] = 0.25
    elif kind == "ties":  # 300 stronger ones, then 3000 equal ones (or what there is), the rest far below
        order = torch.rand(B, V, device="cuda", generator=gen).argsort(-1)
        value = torch.full((V,), -20.0, device="cuda")
        value[:3300] = 1.0
        value[:300] = 2.0 + torch.rand(300, device="cuda", generator=gen)
        logits.scatter_(1, order, value.expand(B, V).contiguous())
    else:  # ten levels of equal tokens
        logits = (torch.rand(B, V, device="cuda", generator=gen) * 10).floor() * 0.3
    tok, lp = ops.sample(logits, top_k=torch.full((B,), k, dtype=torch.int32, device="cuda"), top_p=torch.full((B,), p, device="cuda"),
                         seed=9, step=torch.zeros(1, dtype=torch.long, device="cuda"))
    for b in range(0, B, max(1, B // 5)):
        full, least, most = _sampler_bounds(logits[b], k, p)
        t = int(tok[b])
        assert bool(most[t]), (b, t)
        lo, hi = (float(full[t] - torch.logsumexp(full[m], 0)) for m in (most, least if bool(least.any()) else most))
        assert lo - 5e-5 <= float(lp[b]) <= hi + 5e-5, (b, lo, float(lp[b]), hi)  # fast exp and log, fp32 sums of up to V terms


@pytest.mark.parametrize("V", [1000, 5000, 152064])
def test_sampler_rows_without_numbers(V):
    """Rows of NaN, of -inf, with some of either, and with +inf: a token of the vocabulary comes out, a masked one never, and the other
    rows are as they are without them."""
    from verl_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn(7, V, device="cuda", generator=gen) * 3
    clean = x.clone()
    x[0] = float("nan")
    x[1, 17] = float("nan")
    x[2] = float("-inf")
    x[4, 33] = float("inf")
    for rows in (x, clean):
        rows[3, ::2] = float("-inf")
        rows[6, : V - 3] = float("-inf")
    for k, p, t in ((-1, 1.0, 1.0), (-1, 1.0, 0.0), (50, 1.0, 1.0), (-1, 0.9, 0.7), (20, 0.8, 1.0), (900, 1.0, 1.3)):
        outs = []
        for rows in (x, clean):
            full = lambda v, dt: torch.full((7,), v, dtype=dt, device="cuda")  # noqa: E731
            outs.append(ops.sample(rows, temperature=full(t, torch.float32), top_k=full(k, torch.int32), top_p=full(p, torch.float32),
                                   seed=5, step=torch.zeros(1, dtype=torch.long, device="cuda")))
        (tok, lp), (tok_c, lp_c) = outs
        assert bool(((tok >= 0) & (tok < V)).all())
        for r in (3, 5, 6):
            assert int(tok[r]) == int(tok_c[r]) and float(lp[r]) == float(lp_c[r])
        assert int(tok[3]) % 2 == 1 and int(tok[6]) >= V - 3


@pytest.mark.parametrize("B", [3, 30, 75])
def test_sampler_mixed_rows(B):
    """Restricted, free and greedy rows in one call give the bits that each gives among rows of its own kind."""
    from verl_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(B)
    logits = torch.randn(B, 32771, device="cuda", generator=gen) * 2
    kinds = [(1.0, -1, 1.0), (0.0, 50, 0.9), (0.8, 40, 1.0), (1.0, -1, 0.95), (0.7, 2000, 0.99)]  # temperature, top-k, top-p

    def call(of):
        cols = list(zip(*(kinds[i] for i in of)))
        return ops.sample(logits, temperature=torch.tensor(cols[0], device="cuda"), top_k=torch.tensor(cols[1], dtype=torch.int32, device="cuda"),
                          top_p=torch.tensor(cols[2], device="cuda"), seed=1, step=torch.zeros(1, dtype=torch.long, device="cuda"))

    of = [b % len(kinds) for b in range(B)]
    tok, lp = call(of)
    for i in range(len(kinds)):
        t, l = call([i] * B)
        rows = torch.tensor([o == i for o in of], device="cuda")
        assert torch.equal(t[rows], tok[rows]) and torch.equal(l[rows], lp[rows])


def test_sampler_never_takes_a_token_of_no_weight():
    """A uniform draw that rounds up to one must not become infinite noise: 4000 rows of 152 064 tokens hold about 36 such draws."""
    from verl_b200 import ops

    logits = torch.zeros(1, 152064, device="cuda")
    logits[0, 77] = 100.0
    tok, _ = ops.sample(logits.expand(4000, -1), seed=11, step=torch.zeros(1, device="cuda", dtype=torch.long))
    assert bool((tok == 77).all())


@pytest.mark.parametrize("D", [64, 128])
def test_position_tables_off_a_16_byte_boundary(D):
    """They are read 16 bytes at a time: tables that lie 4 bytes off take the separate steps, which give the same bits, and the kernel's
    entry points refuse them."""
    from verl_b200 import ops
    from verl_b200.ops import _lib

    T, Hq, Hk = 9, 4, 2
    qkv = torch.randn(T, (Hq + 2 * Hk) * D, device="cuda").bfloat16()
    pos = torch.arange(T, device="cuda")
    tables = ops.rope_tables(D, 64, 10000.0, "cuda")
    off = []
    for t in tables:
        off.append(torch.empty(t.numel() + 1, device="cuda")[1:].view(t.shape))
        off[-1].copy_(t)
    with torch.no_grad():
        want = ops.rope_qkv(qkv.clone(), pos, *tables, Hq, Hk, D)
        assert ops.qkv_heads(qkv.clone(), pos, *off, Hq, Hk, D, None, 1e-6) is None
        assert not ops.head_norm_rope_(qkv.clone(), pos, *off, Hq, Hk, D, None, 1e-6)
        assert torch.equal(ops.rope_qkv(qkv.clone(), pos, *off, Hq, Hk, D), want)
        q, _, _ = ops.qkv_heads(qkv.clone(), pos, *tables, Hq, Hk, D, None, 1e-6)
        assert torch.equal(q.reshape(T, -1), want[:, : Hq * D])
    out = torch.empty_like(qkv)
    head = (qkv.data_ptr(), qkv.stride(0), out.data_ptr(), out.stride(0), pos.data_ptr())
    tail = (None, None, 1e-6, T, Hq, Hk, D)
    assert _lib.fn("vb_head_norm_rope")(*head, off[0].data_ptr(), off[1].data_ptr(), *tail, None, None, None, 0, _lib.stream()) == -3
    assert _lib.fn("vb_head_norm_rope_bwd")(*(qkv.data_ptr(),) * 3, None, 0, pos.data_ptr(), off[0].data_ptr(), off[1].data_ptr(), *tail,
                                            out.data_ptr(), None, None, None, 0, 0, _lib.stream()) == -3


@pytest.mark.parametrize("T,Hq,Hk,D,bs", [(1, 14, 2, 64, 16), (37, 28, 4, 128, 16), (5, 3, 1, 256, 8), (129, 9, 3, 64, 64)])
@pytest.mark.parametrize("norm", [False, True])
def test_head_norm_rope(T, Hq, Hk, D, bs, norm):
    """Norms, positions and cache writes in one pass against the separate steps in fp64; rows without a slot are not written."""
    from verl_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(T)
    full = torch.randn(T, (Hq + 2 * Hk) * D + 8, device="cuda", generator=gen).bfloat16()
    src = full[:, 4 : 4 + (Hq + 2 * Hk) * D]
    pos = torch.randint(0, 4096, (T,), device="cuda", generator=gen)
    cos_t, sin_t = ops.rope_tables(D, 4096, 1e6, "cuda")
    qw, kw = (1 + 0.1 * torch.randn(D, device="cuda", generator=gen).bfloat16() for _ in range(2))
    NB = T // bs + 2
    slots = torch.randperm(NB * bs, device="cuda", generator=gen)[:T]
    slots[T // 2] = -1 if T > 1 else slots[0]
    kc, vc = (torch.full((NB, Hk, bs, D), 9.0, device="cuda").bfloat16() for _ in range(2))
    x = src.double().view(T, Hq + 2 * Hk, D)
    if norm:
        n = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6)
        x = torch.cat([n[:, :Hq] * qw.double(), n[:, Hq : Hq + Hk] * kw.double(), x[:, Hq + Hk :]], 1)
    c, s = cos_t[pos].double()[:, None], sin_t[pos].double()[:, None]
    a, b = x[:, : Hq + Hk, : D // 2], x[:, : Hq + Hk, D // 2 :]
    ref = torch.cat([torch.cat([a * c - b * s, b * c + a * s], -1), x[:, Hq + Hk :]], 1)
    with torch.no_grad():
        assert ops.head_norm_rope_(src, pos, cos_t, sin_t, Hq, Hk, D, (qw, kw) if norm else None, 1e-6, slots, kc, vc)
    got = src.double().view(T, Hq + 2 * Hk, D)
    # roundings to bf16 of the normed head, carried by the rotation, and of the result, 2^-8 each
    size = torch.cat([(a.abs() + b.abs()).repeat(1, 1, 2), x[:, Hq + Hk :].abs()], 1)
    assert ((got - ref).abs() <= 2.0 ** -7 * size + 1e-5 * ref.abs().max()).all()
    want_k, want_v = torch.full_like(kc, 9.0), torch.full_like(vc, 9.0)
    k, v = (src[:, i : i + Hk * D].clone().view(T, Hk, D) for i in (Hq * D, (Hq + Hk) * D))  # that kernel takes 16-byte boundaries
    ops.kv_cache_write(k, v, slots, want_k, want_v)
    assert torch.equal(kc, want_k) and torch.equal(vc, want_v)


@pytest.mark.parametrize("T,Hq,Hk,D", [(1, 14, 2, 64), (300, 7, 1, 128), (33, 4, 4, 256), (2000, 8, 2, 64)])
@pytest.mark.parametrize("norm", [False, True])
def test_qkv_heads_gradients(T, Hq, Hk, D, norm):
    """Forward as without gradients, bit for bit; gradients of the projection and of the norms against fp64, added to ``main_grad``."""
    from verl_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()  # noqa: E731
    qkv = rnd(T, (Hq + 2 * Hk) * D).requires_grad_(True)
    pos = torch.randint(0, 4096, (T,), device="cuda", generator=gen)
    cos_t, sin_t = ops.rope_tables(D, 4096, 1e6, "cuda")
    w = [(1 + 0.1 * rnd(D)).requires_grad_(True) for _ in range(2)]
    w[1].main_grad = torch.full((D,), 2.0, device="cuda")
    grads = [rnd(T, n, D) for n in (Hq, Hk, Hk)]
    got = ops.qkv_heads(qkv, pos, cos_t, sin_t, Hq, Hk, D, tuple(w) if norm else None, 1e-6)
    with torch.no_grad():
        plain = ops.qkv_heads(qkv.detach().clone(), pos, cos_t, sin_t, Hq, Hk, D, tuple(w) if norm else None, 1e-6)
    assert all(torch.equal(g, p) for g, p in zip(got, plain))
    if not norm:
        with torch.no_grad():
            assert torch.equal(torch.cat(got, 1).view(T, -1), ops.rope_qkv(qkv.detach().clone(), pos, cos_t, sin_t, Hq, Hk, D))
    torch.autograd.backward(got, grads)
    x, (qw, kw) = qkv.detach().double().requires_grad_(True), (t.detach().double().requires_grad_(True) for t in w)
    h = x.view(T, Hq + 2 * Hk, D)
    if norm:
        n = h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-6)
        h = torch.cat([n[:, :Hq] * qw, n[:, Hq : Hq + Hk] * kw, h[:, Hq + Hk :]], 1)
    c, s = cos_t[pos].double()[:, None], sin_t[pos].double()[:, None]
    a, b = h[:, : Hq + Hk, : D // 2], h[:, : Hq + Hk, D // 2 :]
    y = torch.cat([torch.cat([a * c - b * s, b * c + a * s], -1), h[:, Hq + Hk :]], 1)
    y.backward(torch.cat(grads, 1).double())
    # the rotated gradient and the result are rounded, 2^-8 each; the norm's weights and 1 / rms carry the first one by less than 2
    _bf16_close(qkv.grad, x.grad, ulps=3)
    if norm:
        for g, ref, heads in ((w[0].grad.double(), qw.grad, Hq), (w[1].main_grad.double() - 2.0, kw.grad, Hk)):
            # T * heads terms of about 1, their gradient factor rounded (2^-8, of either sign: 6 sigma), and the result in bf16
            bound = 2.0 ** -8 * 6 * (T * heads) ** 0.5 + 2.0 ** -8 * ref.abs()
            assert ((g - ref).abs() <= bound).all()


@pytest.mark.parametrize("B,Hq,Hk,D,bs,maxlen", [(5, 28, 4, 128, 16, 700), (3, 4, 2, 64, 16, 300), (2, 32, 4, 128, 32, 3000),
                                                 (4, 40, 8, 128, 16, 150), (3, 32, 2, 128, 128, 1000),
                                                 (2, 8, 8, 128, 8, 260), (1, 14, 2, 64, 16, 110), (7, 8, 8, 64, 8, 129),
                                                 (3, 32, 2, 64, 32, 1025), (40, 8, 1, 64, 256, 2100), (3, 9, 1, 128, 16, 513),
                                                 # more (sequence, head, split) CTAs than run at once, some of them without keys
                                                 (100, 28, 4, 128, 16, 700), (80, 32, 8, 128, 16, 300)])
def test_paged_decode_attention(B, Hq, Hk, D, bs, maxlen):
    from verl_b200 import ops

    torch.manual_seed(10)
    lens = torch.randint(1, maxlen, (B,), dtype=torch.int32)
    lens[0] = maxlen
    nblk_per = (maxlen + bs - 1) // bs
    NB = B * nblk_per + 3
    kc = torch.zeros(NB, Hk, bs, D, device="cuda", dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    table = torch.randperm(NB)[: B * nblk_per].reshape(B, nblk_per).int().cuda()
    # fill through the cache-write kernel
    for b in range(B):
        L = int(lens[b])
        k_new = torch.randn(L, Hk, D, device="cuda").bfloat16()
        v_new = torch.randn(L, Hk, D, device="cuda").bfloat16()
        pos = torch.arange(L, device="cuda")
        slots = table[b].long()[pos // bs] * bs + pos % bs
        ops.kv_cache_write(k_new, v_new, slots, kc, vc)
    q = torch.randn(B, Hq, D, device="cuda").bfloat16()
    ref = ops.paged_decode_attention(q.cpu().float(), kc.cpu().float(), vc.cpu().float(), table.cpu(), lens)
    from verl_b200.ops import _lib

    impls = ["auto"] + (["simt"] if Hq // Hk <= 8 else [])
    if _lib.fn("vb_paged_decode_tc_supported")(Hq, Hk, D, bs):
        impls.append("tc")
    assert impls
    for impl in impls:
        for splits in sorted({1, 3, ops.decode_workspace(B, Hq, Hk, D, maxlen, "cuda")[0]}):
            out = ops.paged_decode_attention(q, kc, vc, table, lens.cuda(), num_splits=splits, impl=impl)
            assert _lib.read_status("cuda")[0] == 0
            _bf16_close(out, ref, ulps=4)


def test_hooked_projection_keeps_its_result():
    """A forward hook on the projection of a layer with head norms may keep what it is given: the pass without gradients does not write
    over it, and gives the bits that it gives without the hook."""
    from verl_b200.models import PackedBatch, build_model, preset

    model = build_model(preset("tiny-qwen2", model_type="qwen3", head_dim=64), device="cuda")
    ids = torch.arange(3, 40, device="cuda")
    batch = PackedBatch(ids, torch.arange(37, device="cuda"), torch.tensor([0, 37], dtype=torch.int32, device="cuda"), 37)
    kept = []
    with torch.no_grad():
        want = model.forward_hidden(batch)
        handle = model.layers[0].self_attn.qkv_proj.register_forward_hook(lambda m, a, out: kept.append((out, out.clone())) or None)
        got = model.forward_hidden(batch)
        handle.remove()
    assert len(kept) == 1 and torch.equal(*kept[0]) and torch.equal(got, want)


@pytest.mark.parametrize("Hq,Hk,D,bs,lens", [(14, 2, 64, 16, (500, 1, 129)), (8, 8, 64, 8, (3000, 17)), (32, 2, 64, 32, (700, 64)),
                                             (8, 1, 128, 256, (2100, 255, 300)), (9, 1, 128, 512, (513, 30))])
def test_decode_attention_weights_stay_in_fp32(Hq, Hk, D, bs, lens):
    """Heads of 64, and pages above 128 rows: the splits' fp32 results against fp64, before anything is rounded to bf16."""
    from verl_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(Hq + D)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()  # noqa: E731
    B, G, S = len(lens), Hq // Hk, 3
    n = (max(lens) + bs - 1) // bs
    q, kc, vc = rnd(B, Hq, D), rnd(B * n, Hk, bs, D), rnd(B * n, Hk, bs, D)
    table = torch.arange(B * n, device="cuda", dtype=torch.int32).reshape(B, n)
    work = torch.zeros(B * Hq * S * (D + 2), device="cuda")
    ops.paged_decode_attention(q, kc, vc, table, torch.tensor(lens, dtype=torch.int32, device="cuda"), num_splits=S, work=work)
    o, ml = work[: B * Hq * S * D].view(B, Hq, S, D).double(), work[B * Hq * S * D :].view(B, Hq, S, 2).double()
    part = torch.exp(ml[..., 0] - ml[..., 0].amax(-1, keepdim=True))
    got = (o * part[..., None]).sum(2) / (ml[..., 1] * part).sum(-1)[..., None]
    for b, L in enumerate(lens):
        k, v = (c.view(B, n, Hk, bs, D)[b].transpose(0, 1).reshape(Hk, n * bs, D)[:, :L].double() for c in (kc, vc))
        p = torch.softmax(torch.einsum("hgd,hkd->hgk", q[b].view(Hk, G, D).double(), k) * D ** -0.5, -1)
        want = torch.einsum("hgk,hkd->hgd", p, v).reshape(Hq, D)
        # scores of up to about 5 in fp32 and sums of L weights: 2^-24 each, some tens of them together; weights in bf16 would be 2^-10 off
        assert float((got[b] - want).norm() / want.norm()) <= 64 * 2.0 ** -24


@pytest.mark.parametrize("sigmoid", [False, True])
@pytest.mark.parametrize("B,Hq,Hk,D,splits,window", [(160, 8, 2, 128, 1, 0), (120, 8, 2, 64, 3, 150), (75, 40, 8, 96, 2, 0), (310, 3, 1, 128, 4, 70)])
def test_windowed_decode_walks_several_items_per_cta(B, Hq, Hk, D, splits, window, sigmoid):
    """More (sequence, KV head, split) items than CTAs run at once: the tcgen05 kernel of the layer-list models takes one after the
    other, with items in between that have no key (short sequences, windows), and none may see what the one before left."""
    from verl_b200 import ops
    from verl_b200.ops import _lib

    gen = torch.Generator().manual_seed(B + splits)
    bs, most = 16, 700
    assert B * Hk * splits > 2 * torch.cuda.get_device_properties(0).multi_processor_count
    lens = torch.randint(1, most, (B,), generator=gen, dtype=torch.int32)
    lens[::7] = torch.randint(1, 40, (len(lens[::7]),), generator=gen, dtype=torch.int32)
    n = (most + bs - 1) // bs
    q, kc, vc = (torch.randn(*s, generator=gen).bfloat16() for s in ((B, Hq, D), (B * n, Hk, bs, D), (B * n, Hk, bs, D)))
    table = torch.randperm(B * n, generator=gen).int().reshape(B, n)
    scale, opts = D ** -0.5, dict(window=window)
    shift = r1 = r2 = None
    if sigmoid:
        shift, r1, r2 = torch.randn(Hq, generator=gen) - 3, torch.rand(Hq, generator=gen) * 0.3, torch.rand(Hq, generator=gen) * 0.1
        opts.update(shift=shift, log_bias=(r1, r2))
    cu = torch.arange(B + 1, dtype=torch.int32)
    ref = ops.paged_attention(q.float(), kc.float(), vc.float(), table, cu, lens, 1, scale=scale, **opts)
    q, kc, vc, table, lens_d = (t.cuda() for t in (q, kc, vc, table, lens))
    shift, r1, r2 = (None if t is None else t.cuda() for t in (shift, r1, r2))
    work = torch.full((B * Hq * splits * (D + 2),), float("nan"), device="cuda")
    out = torch.full((B, Hq * D), float("nan"), dtype=torch.bfloat16, device="cuda")
    rc = _lib.fn("vb_paged_decode_window")(q.data_ptr(), q.stride(0), kc.data_ptr(), vc.data_ptr(), kc.shape[0], table.data_ptr(),
                                           table.stride(0), lens_d.data_ptr(), B, Hq, Hk, D, D, bs, scale, window, 0, 0, None, 0, 0.0, None,
                                           _lib.ptr(shift), _lib.ptr(r1), _lib.ptr(r2), None, 0, 0, splits, out.data_ptr(), out.stride(0),
                                           work.data_ptr() if splits > 1 else None, _lib.status_word("cuda").data_ptr(), _lib.stream())
    assert rc == 0 and _lib.read_status("cuda")[0] == 0
    _bf16_close(out, ref, ulps=4)


def _attn_ref(q, k, v, cu, causal, scale):
    """fp32 reference, one sequence at a time. Returns (out [T,Hq,D], lse [Hq,T])."""
    T, Hq, D = q.shape
    G = Hq // k.shape[1]
    out = torch.empty(T, Hq, D, device=q.device)
    lse = torch.empty(Hq, T, device=q.device)
    b = cu.tolist()
    for s, e in zip(b[:-1], b[1:]):
        qs = q[s:e].float().transpose(0, 1)
        ks = k[s:e].float().repeat_interleave(G, dim=1).transpose(0, 1)
        vs = v[s:e].float().repeat_interleave(G, dim=1).transpose(0, 1)
        sc = qs @ ks.transpose(1, 2) * scale
        if causal:
            n = e - s
            sc = sc.masked_fill(torch.triu(torch.ones(n, n, device=q.device, dtype=torch.bool), 1), float("-inf"))
        lse[:, s:e] = torch.logsumexp(sc, -1)
        out[s:e] = (torch.softmax(sc, -1) @ vs).transpose(0, 1)
    return out, lse


@pytest.mark.parametrize("lens,Hq,Hk,causal", [([300, 77, 512, 129], 28, 4, True), ([1, 128, 640], 8, 8, True),
                                               ([1000, 333], 16, 2, False), ([2048], 4, 4, True)])
def test_flash_attention_fwd(lens, Hq, Hk, causal):
    from verl_b200.ops import _lib
    from verl_b200.ops.attention import flash_fwd

    torch.manual_seed(11)
    D, T = 128, sum(lens)
    # q / k / v as views of one fused buffer (token stride (Hq + 2 Hk) * D), the way the model produces them
    qkv = torch.randn(T, (Hq + 2 * Hk) * D, device="cuda").bfloat16()
    q = qkv[:, : Hq * D].view(T, Hq, D)
    k = qkv[:, Hq * D : (Hq + Hk) * D].view(T, Hk, D)
    v = qkv[:, (Hq + Hk) * D :].view(T, Hk, D)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")
    scale = D ** -0.5
    out, lse = flash_fwd(q, k, v, cu, max(lens), causal, scale)
    assert _lib.read_status("cuda")[0] == 0
    ref, ref_lse = _attn_ref(q, k, v, cu, causal, scale)
    _bf16_close(out, ref, ulps=4)
    torch.testing.assert_close(lse, ref_lse, atol=2e-3, rtol=1e-4)


@pytest.mark.parametrize("lens,Hq,Hk,causal", [([200, 131, 64], 8, 2, True), ([513, 1], 4, 4, True), ([300, 77], 28, 4, True),
                                               ([260], 4, 2, False)])
def test_flash_attention_autograd_matches_reference(lens, Hq, Hk, causal):
    from verl_b200 import ops
    from verl_b200.ops import _lib

    torch.manual_seed(12)
    D = 128
    T = sum(lens)
    q = torch.randn(T, Hq, D, device="cuda").bfloat16().requires_grad_(True)
    k = torch.randn(T, Hk, D, device="cuda").bfloat16().requires_grad_(True)
    v = torch.randn(T, Hk, D, device="cuda").bfloat16().requires_grad_(True)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")
    do = torch.randn(T, Hq, D, device="cuda").bfloat16()
    ops.attention_varlen(q, k, v, cu, max(lens), causal=causal, impl="native").backward(do)
    assert _lib.read_status("cuda")[0] == 0
    qr, kr, vr = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    ref, _ = _attn_ref(qr, kr, vr, cu, causal, D ** -0.5)
    ref.backward(do.float())
    for got, want in ((q.grad, qr.grad), (k.grad, kr.grad), (v.grad, vr.grad)):
        err = (got.float() - want).abs().max().item()
        assert err <= 2e-2 * max(1.0, want.abs().max().item()), err


def test_flash_attention_fwd_with_cached_prefix():
    """Queries are the last positions of a longer key stream (chunked prefill on top of cached context)."""
    from verl_b200.ops.attention import flash_fwd

    torch.manual_seed(13)
    Hq, Hk, D = 8, 2, 128
    lq, lk = [100, 1, 260], [100, 300, 700]
    q = torch.randn(sum(lq), Hq, D, device="cuda").bfloat16()
    k = torch.randn(sum(lk), Hk, D, device="cuda").bfloat16()
    v = torch.randn(sum(lk), Hk, D, device="cuda").bfloat16()
    cu_q = torch.tensor([0] + list(torch.tensor(lq).cumsum(0)), dtype=torch.int32, device="cuda")
    cu_k = torch.tensor([0] + list(torch.tensor(lk).cumsum(0)), dtype=torch.int32, device="cuda")
    out, _ = flash_fwd(q, k, v, cu_q, max(lq), True, D ** -0.5, cu_seqlens_k=cu_k)
    G = Hq // Hk
    for b in range(len(lq)):
        qs = q[cu_q[b]:cu_q[b + 1]].float().transpose(0, 1)
        ks = k[cu_k[b]:cu_k[b + 1]].float().repeat_interleave(G, 1).transpose(0, 1)
        vs = v[cu_k[b]:cu_k[b + 1]].float().repeat_interleave(G, 1).transpose(0, 1)
        s = qs @ ks.transpose(1, 2) * D ** -0.5
        mask = torch.arange(lk[b], device="cuda")[None, :] <= (torch.arange(lq[b], device="cuda")[:, None] + lk[b] - lq[b])
        ref = (torch.softmax(s.masked_fill(~mask, float("-inf")), -1) @ vs).transpose(0, 1)
        _bf16_close(out[cu_q[b]:cu_q[b + 1]], ref, ulps=4)


def test_moe_grouped_gemm_matches_expert_loop():
    """Grouped GEMM path of the MoE MLP (one launch per projection, device-side routing layout) against the
    per-expert fp32 reference: outputs, input gradients, weight gradients (also fused into main_grad)."""
    from verl_b200 import ops
    from verl_b200.ops.moe import moe_mlp

    torch.manual_seed(14)
    T, H, I, E, k = 300, 256, 192, 8, 2
    x = torch.randn(T, H, device="cuda").bfloat16().requires_grad_(True)
    gate_up = (torch.randn(E, 2 * I, H, device="cuda") * 0.05).bfloat16().requires_grad_(True)
    down = (torch.randn(E, H, I, device="cuda") * 0.05).bfloat16().requires_grad_(True)
    logits = torch.randn(T, E, device="cuda")
    logits[:, 5] = -1e9  # an expert without tokens
    top_w, top_i = torch.topk(torch.softmax(logits, -1), k, -1)
    top_w = (top_w / top_w.sum(-1, keepdim=True)).detach()
    dy = torch.randn(T, H, device="cuda").bfloat16()
    y = moe_mlp(x, top_i, top_w, gate_up, down, ops.swiglu)
    y.backward(dy)
    xr, gr, dr = (t.detach().float().requires_grad_(True) for t in (x, gate_up, down))
    ref = torch.zeros(T, H, device="cuda")
    for j in range(k):
        for e in range(E):
            sel = top_i[:, j] == e
            if sel.any():
                gu = xr[sel] @ gr[e].t()
                h = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
                ref[sel] = ref[sel] + (h @ dr[e].t()) * top_w[sel, j : j + 1].float()
    ref.backward(dy.float())

    def close(a, b, tol):
        err = (a.float() - b).abs().max().item()
        assert err <= tol * max(1.0, b.abs().max().item()), (err, b.abs().max().item())

    close(y, ref.detach(), 2e-2)
    close(x.grad, xr.grad, 3e-2)
    close(gate_up.grad, gr.grad, 3e-2)
    close(down.grad, dr.grad, 3e-2)
    assert float(gate_up.grad[5].abs().sum()) == 0.0
    # fused accumulation into fp32 main_grad
    g2 = gate_up.detach().clone().requires_grad_(True)
    g2.main_grad = torch.ones(g2.shape, device="cuda")
    moe_mlp(x.detach(), top_i, top_w, g2, down.detach(), ops.swiglu).backward(dy)
    assert g2.grad is None
    close(g2.main_grad - 1.0, gr.grad, 3e-2)


@pytest.mark.parametrize("T,E,k,H,I,first,total", [
    (1, 8, 2, 128, 64, 0, 8),        # fewer pairs than experts
    (24, 128, 8, 256, 64, 0, 128),   # a decode step
    (129, 3, 1, 64, 128, 0, 3),      # shares just above one block of rows
    (700, 16, 4, 192, 64, 4, 32),    # experts 4 .. 19 of 32 (a replica's part): other pairs have no row
    (5000, 2, 1, 64, 64, 0, 2),      # several chunks of pairs per expert
])
def test_routed_mlp_forms(T, E, k, H, I, first, total):
    """Places, padding rows, weighted sum and all gradients of the routed MLP against an fp64 loop over the experts, and a buffer
    full of NaN behind every allocation it makes (nothing undefined may reach a result)."""
    from verl_b200 import ops
    from verl_b200.ops.moe import moe_mlp

    gen = torch.Generator(device="cuda").manual_seed(T + E)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    x = rnd(T, H).bfloat16().requires_grad_(True)
    gate_up, down = ((rnd(*s) * 0.1).bfloat16().requires_grad_(True) for s in ((E, 2 * I, H), (E, H, I)))
    top_i = rnd(T, total).topk(k, -1).indices
    top_w = torch.rand(T, k, device="cuda", generator=gen).requires_grad_(True)
    dy = rnd(T, H).bfloat16()
    for n in (T * k * H, (T * k + E * 127) * H, (T * k + E * 127) * 2 * I, T * H):  # freed at once: found again by the next allocations
        torch.full((n,), float("nan"), dtype=torch.bfloat16, device="cuda")
    y = moe_mlp(x, top_i, top_w, gate_up, down, ops.swiglu, expert_offset=first, num_experts=total)
    y.backward(dy)
    xr, wr, gr, dr = (t.detach().double().requires_grad_(True) for t in (x, top_w, gate_up, down))
    ref = torch.zeros(T, H, dtype=torch.float64, device="cuda")
    for e in range(E):
        t, j = (top_i == first + e).nonzero(as_tuple=True)
        gu = xr[t] @ gr[e].t()
        h = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
        ref = ref.index_add(0, t, (h @ dr[e].t()) * wr[t, j][:, None])
    ref.backward(dy.double())
    # three bf16 roundings on the way forward and six back, 2^-9 each, against the largest value
    for got, want, roundings in ((y, ref, 3), (x.grad, xr.grad, 6), (top_w.grad, wr.grad, 6), (gate_up.grad, gr.grad, 6),
                                 (down.grad, dr.grad, 6)):
        want = want.detach()
        err = float((got.detach().double() - want).abs().max())
        assert err <= roundings * 2.0 ** -8 * float(want.abs().max()) + 1e-12, (got.shape, err, float(want.abs().max()))


def test_routed_mlp_of_very_many_experts_and_pairs():
    """Both sides of the line beyond which the places are taken by a sort, against each other."""
    from verl_b200 import ops
    from verl_b200.ops import moe

    gen = torch.Generator(device="cuda").manual_seed(4)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    T, E, k, H, I = 10300, 2048, 8, 64, 64
    x, gate_up, down = rnd(T, H).bfloat16(), rnd(E, 2 * I, H).bfloat16() * 0.1, rnd(E, H, I).bfloat16() * 0.1
    top_i = torch.randint(0, E, (T, k), device="cuda", generator=gen)
    top_w = torch.rand(T, k, device="cuda", generator=gen)
    args = (gate_up, down, ops.swiglu)
    n = 10240
    assert moe._fused_mlp_ok(x[:n], top_i[:n], top_w[:n], *args) and not moe._fused_mlp_ok(x, top_i, top_w, *args)
    got, want = moe.moe_mlp(x[:n], top_i[:n], top_w[:n], *args), moe.moe_mlp(x, top_i, top_w, *args)[:n]
    # weights, terms and sums in bf16 on the general path
    assert float((got.double() - want.double()).abs().max()) <= 4 * 2.0 ** -8 * float(want.abs().max())


def test_routed_mlp_refuses_and_realigns():
    """Routing of another number of tokens is refused before a kernel reads past it; rows and gradients off a 16-byte boundary work."""
    from verl_b200 import ops
    from verl_b200.ops.moe import moe_gate, moe_mlp

    T, E, k, H, I = 20, 4, 2, 64, 64
    gate_up, down = (torch.randn(*s, device="cuda").bfloat16() * 0.1 for s in ((E, 2 * I, H), (E, H, I)))
    z = torch.randn(T, E, device="cuda")
    w, idx = moe_gate(z, k, True)
    x = torch.randn(T * H + 1, device="cuda").bfloat16()
    off = x[1:].view(T, H)
    y = moe_mlp(off, idx, w, gate_up, down, ops.swiglu)
    _bf16_close(y, moe_mlp(off.clone(), idx, w, gate_up, down, ops.swiglu))
    leaf = off.clone().requires_grad_(True)
    out = moe_mlp(leaf, idx, w, gate_up, down, ops.swiglu)
    (want,) = torch.autograd.grad(out, leaf, x[1:].view(T, H).clone(), retain_graph=True)
    (got,) = torch.autograd.grad(out, leaf, x[1:].view(T, H))
    assert torch.equal(got, want)
    assert moe_gate(z, k, False, idx[:7])[0].shape == (7, k)  # as torch.gather does it
    with pytest.raises((RuntimeError, ValueError, IndexError)):
        moe_mlp(off.clone(), idx[:7], w[:7], gate_up, down, ops.swiglu)


@pytest.mark.parametrize("E,k", [(8, 2), (33, 8), (128, 8), (300, 32)])
@pytest.mark.parametrize("renorm", [True, False])
@pytest.mark.parametrize("given", [False, True])
def test_moe_gate_matches_softmax_topk(E, k, renorm, given):
    """Experts (ties included: bf16 logits repeat), weights and gradient of the gate against torch in fp64."""
    from verl_b200.ops.moe import moe_gate

    gen = torch.Generator(device="cuda").manual_seed(E)
    z = torch.randn(37, E, device="cuda", generator=gen).bfloat16().requires_grad_(True)
    fixed = torch.rand(37, E, device="cuda", generator=gen).topk(k, -1).indices if given else None
    w, idx = moe_gate(z, k, renorm, fixed)
    g = torch.randn(37, k, device="cuda", generator=gen)
    w.backward(g)
    zr = z.detach().double().requires_grad_(True)
    want = fixed if given else torch.sort(zr.detach(), dim=-1, descending=True, stable=True).indices[:, :k]
    assert torch.equal(idx, want)
    p = torch.softmax(zr, -1).gather(1, want)
    p = p / p.sum(-1, keepdim=True) if renorm else p
    p.backward(g.double())
    assert float((w.double() - p).abs().max()) < 1e-6
    assert float((z.grad.double() - zr.grad).abs().max()) <= 2.0 ** -8 * float(zr.grad.abs().max()) + 1e-9


@pytest.mark.parametrize("bad", [-1, 8, 1 << 32])
@pytest.mark.parametrize("renorm", [True, False])
def test_experts_outside_the_layer_are_refused(bad, renorm):
    """A given expert that the layer does not have (also one that is 0 in its low 32 bits): the next look raises, once, and until then
    nothing that depends on it is a number; other tokens are as without it. A replica's part takes them for another rank's."""
    from verl_b200 import ops
    from verl_b200.ops import _lib
    from verl_b200.ops.moe import moe_gate, moe_mlp

    T, E, k, H, I = 12, 8, 2, 64, 64
    gen = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    z, x = rnd(T, E), rnd(T, H).bfloat16()
    gate_up, down = (rnd(*s).bfloat16() * 0.1 for s in ((E, 2 * I, H), (E, H, I)))
    good = rnd(T, E).topk(k, -1).indices
    given = good.clone()
    given[4, 1] = bad
    keep = torch.arange(T, device="cuda") != 4
    want = moe_gate(z, k, renorm, good)[0]

    def looked():
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError, match="pair 9 .* outside"):
            _lib.raise_refused()
        _lib.raise_refused()

    got = moe_gate(z, k, renorm, given)[0]
    looked()
    assert bool(got[4, 1].isnan()) and torch.equal(got[keep], want[keep])
    leaf = z.clone().requires_grad_(True)
    w, _ = moe_gate(leaf, k, renorm, given)
    looked()
    w.sum().backward()
    assert bool(leaf.grad[4].isnan().any()) and not bool(leaf.grad[keep].isnan().any())
    y = moe_mlp(x, given, want, gate_up, down, ops.swiglu)
    looked()
    assert bool(y[4].isnan().all()) and torch.equal(y[keep], moe_mlp(x, good, want, gate_up, down, ops.swiglu)[keep])
    part = moe_mlp(x, given, want, gate_up[2:6].contiguous(), down[2:6].contiguous(), ops.swiglu, expert_offset=2, num_experts=E)
    torch.cuda.synchronize()
    _lib.raise_refused()
    assert not bool(part.isnan().any())


@pytest.mark.parametrize("renorm", [True, False])
def test_second_derivatives_of_gate_and_routed_sum(renorm):
    """Gradients taken with ``create_graph`` are those of the kernels, and differentiating them gives what torch gives in fp64 (gate: all
    second derivatives; routed sum: those by the routing weights, its products have a first backward only)."""
    from verl_b200 import ops
    from verl_b200.ops.moe import moe_gate, moe_mlp

    gen = torch.Generator(device="cuda").manual_seed(8)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    T, E, k, H, I = 20, 8, 2, 64, 64
    z, g = rnd(T, E).requires_grad_(True), rnd(T, k).requires_grad_(True)
    w, idx = moe_gate(z, k, renorm)
    (dz,) = torch.autograd.grad(w, z, g, create_graph=True)
    assert float((dz - torch.autograd.grad(w, z, g, retain_graph=True)[0]).abs().max()) < 1e-6
    v = rnd(T, E)
    got = torch.autograd.grad(dz, (z, g), v)
    zr, gr = z.detach().double().requires_grad_(True), g.detach().double().requires_grad_(True)
    p = torch.softmax(zr, -1).gather(1, idx)
    p = p / p.sum(-1, keepdim=True) if renorm else p
    (dzr,) = torch.autograd.grad(p, zr, gr, create_graph=True)
    for a, b in zip(got, torch.autograd.grad(dzr, (zr, gr), v.double())):
        assert float((a.double() - b).abs().max()) <= 64 * 2.0 ** -24 * max(1.0, float(b.abs().max()))
    gate_up, down = (rnd(*s).bfloat16() * 0.1 for s in ((E, 2 * I, H), (E, H, I)))
    x, dy = rnd(T, H).bfloat16(), rnd(T, H).bfloat16().requires_grad_(True)
    top_w = w.detach().t().contiguous().t().requires_grad_(True)  # not contiguous
    y = moe_mlp(x, idx, top_w, gate_up, down, ops.swiglu)
    (first,) = torch.autograd.grad(y, top_w, dy, create_graph=True)
    (plain,) = torch.autograd.grad(y, top_w, dy.detach(), retain_graph=True)
    scale = float(plain.abs().max())
    assert float((first - plain).abs().max()) <= 4 * 2.0 ** -8 * scale  # bf16 terms, summed
    (back,) = torch.autograd.grad(first, dy, torch.ones_like(first))
    # linear in dy: the sum of the experts' rows, weights 1
    want = moe_mlp(x, idx, torch.ones_like(top_w), gate_up, down, ops.swiglu).double()
    assert float((back.double() - want).abs().max()) <= 4 * 2.0 ** -8 * float(want.abs().max())


def test_traces_and_forward_mode_pass_through():
    """A trace of an op without gradients computes new inputs, and a tangent of the routing weights reaches the routed sum, as
    through torch's own operators."""
    from torch.autograd import forward_ad

    from verl_b200 import ops
    from verl_b200.ops.moe import moe_gate, moe_mlp

    gen = torch.Generator(device="cuda").manual_seed(2)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    T, E, k, H, I = 24, 4, 2, 64, 64
    w, wn = rnd(2 * I, H).bfloat16() * 0.1, rnd(H).bfloat16()
    gate_up, down = (rnd(*s).bfloat16() * 0.1 for s in ((E, 2 * I, H), (E, H, I)))
    x, x2 = rnd(T, H).bfloat16(), rnd(T, H).bfloat16()
    router = rnd(E, H).bfloat16() * 0.1

    with torch.no_grad():
        p, idx = moe_gate(rnd(T, E), k, True)
        for op in (lambda v: ops.rmsnorm(v, wn)[0], lambda v: ops.linear(v, w), lambda v: ops.linear_swiglu(v, w), ops.swiglu,
                   lambda v: moe_gate(ops.linear(v, router), k, True)[0], lambda v: moe_mlp(v, idx, p, gate_up, down, ops.swiglu)):
            got, want = torch.jit.trace(op, x, check_trace=False)(x2).double(), op(x2).double()
            # the routed sum has its terms and its sum in bf16 then, 2^-9 each of the largest
            assert float((got - want).abs().max()) <= 4 * 2.0 ** -9 * float(want.abs().max())
        dp = rnd(T, k)
        with forward_ad.dual_level():
            y = moe_mlp(x, idx, forward_ad.make_dual(p, dp), gate_up, down, ops.swiglu)
            tangent = forward_ad.unpack_dual(y).tangent
            z = forward_ad.make_dual(rnd(T, E), rnd(T, E))
            assert forward_ad.unpack_dual(moe_gate(z, k, True)[0]).tangent is not None
        assert tangent is not None
        # the sum is linear in the weights: two bf16 roundings of the terms and one of the sum
        want = moe_mlp(x, idx, dp, gate_up, down, ops.swiglu).double()
        assert float((tangent.double() - want).abs().max()) <= 3 * 2.0 ** -8 * float(want.abs().max())


def test_bounded_device_wait_reports_status_and_context_survives():
    """A cross-rank barrier whose peer never arrives: the kernel gives up after its time limit, records the wait in
    the status word and returns; the host reads the code and the context keeps working."""
    import ctypes
    import time

    from verl_b200.ops import _lib, gemm

    lib = _lib.load()
    lib.vb_peer_barrier.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_uint, ctypes.c_void_p,
                                    ctypes.c_void_p]
    lib.vb_peer_barrier.restype = ctypes.c_int
    _lib.clear_status("cuda")
    mine = torch.zeros(1024, dtype=torch.int32, device="cuda")
    absent = torch.zeros(1024, dtype=torch.int32, device="cuda")  # stands for a peer that never writes its slot
    pads = (ctypes.c_void_p * 2)(mine.data_ptr(), absent.data_ptr())
    t0 = time.perf_counter()
    rc = lib.vb_peer_barrier(pads, 0, 2, 3, 1, _lib.status_word("cuda").data_ptr(), _lib.stream())
    assert rc == 0
    torch.cuda.synchronize()
    dt = time.perf_counter() - t0
    code, _, detail = _lib.read_status("cuda")
    assert code == 5 and detail == 1, (code, detail)   # ERR_WAIT_FLAG, waiting for rank 1
    assert 1.0 < dt < 10.0
    _lib.clear_status("cuda")
    a = torch.randn(256, 256, device="cuda").bfloat16()
    _bf16_close(gemm(a, a), a.float() @ a.float().t())


@pytest.mark.parametrize("M,N,K,pow2", [(128, 512, 1024, False), (300, 384 + 64, 640, True), (1000, 256, 3584, False),
                                        # decode: every width of the tile, one CTA and up to eight per tile, uneven shares of K
                                        (1, 128, 128, False), (16, 200, 1040, False), (17, 1152, 896, False), (32, 64, 4864, False),
                                        (33, 3584, 3584, False), (48, 4608, 3584, False), (49, 130, 144, False),
                                        (64, 896, 18944, False), (65, 37888, 512, False), (65, 520, 3584, False),
                                        (127, 3584, 3600, False)])
def test_fp8_blockscale_quant_and_gemm(M, N, K, pow2):
    from verl_b200.ops import _lib, fp8

    torch.manual_seed(15)
    x = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
    bias = torch.randn(N, device="cuda").bfloat16()
    wq, sw = fp8.quantize_weight(w, pow2)
    xq, sx = fp8.quantize_activation(x, pow2)
    # quantisation agrees with the plain PyTorch statement of the scheme
    wq_ref, sw_ref = fp8.quantize_weight(w.cpu(), pow2)
    xq_ref, sx_ref = fp8.quantize_activation(x.cpu(), pow2)
    torch.testing.assert_close(sw.cpu(), sw_ref, rtol=1e-6, atol=0)
    torch.testing.assert_close(sx.cpu(), sx_ref, rtol=1e-6, atol=0)
    for got, want in ((wq, wq_ref), (xq, xq_ref)):
        a, b = got.cpu().float(), want.float()
        # the kernel multiplies by a fast reciprocal: values next to a rounding boundary may land on the neighbouring
        # e4m3 code (one step = 1/8 relative), nothing may be further off
        assert (a != b).float().mean() < 0.02
        assert ((a - b).abs() <= 0.126 * torch.maximum(a.abs(), b.abs()) + 2 ** -9).all()
    if pow2:
        assert torch.equal(torch.log2(sw), torch.log2(sw).round())
    # GEMM against the dequantised fp32 product, and loosely against the unquantised one
    out = fp8.fp8_gemm(xq, sx, wq, sw, bias)
    assert _lib.read_status("cuda")[0] == 0
    ref = fp8.dequantize(xq, sx, False) @ fp8.dequantize(wq, sw, True).t() + bias.float()
    _bf16_close(out, ref, ulps=4)
    full = x.float() @ w.float().t() + bias.float()
    rel = (out.float() - full).norm() / full.norm()
    assert rel < 0.06, float(rel)
    _bf16_close(fp8.fp8_linear(x, wq, sw, bias, pow2), ref, ulps=4)


@pytest.mark.parametrize("T", [8, 128, 1000])
def test_programmatic_dependent_launch_chain_is_bit_identical(T):
    """A decode-layer-shaped chain (norm -> GEMM -> rope -> cache write -> paged attention -> GEMM -> norm -> GEMM ->
    swiglu -> GEMM) gives the same bits whether each kernel waits for the one before it at launch (the ordinary
    stream order) or only before its first global access (programmatic dependent launch), eagerly and in a graph."""
    from verl_b200 import ops
    from verl_b200.ops import _lib

    torch.manual_seed(3)
    H, Hq, Hk, D, I, bs = 1024, 8, 2, 128, 2048, 16
    dev = "cuda"
    x0 = torch.randn(T, H, device=dev).bfloat16()
    wn = torch.randn(H, device=dev).bfloat16()
    wqkv = (torch.randn((Hq + 2 * Hk) * D, H, device=dev) * 0.03).bfloat16()
    wo = (torch.randn(H, Hq * D, device=dev) * 0.03).bfloat16()
    wgu = (torch.randn(2 * I, H, device=dev) * 0.03).bfloat16()
    wd = (torch.randn(H, I, device=dev) * 0.03).bfloat16()
    ctx = 200
    nblk = (ctx + bs) // bs + 1
    kc = torch.randn(T * nblk, Hk, bs, D, device=dev).bfloat16()
    vc = torch.randn_like(kc)
    table = torch.arange(T * nblk, device=dev, dtype=torch.int32).reshape(T, nblk)
    lens = torch.full((T,), ctx + 1, device=dev, dtype=torch.int32)
    pos = torch.full((T,), ctx, device=dev, dtype=torch.long)
    slots = table[:, ctx // bs].long() * bs + ctx % bs
    cos, sin = ops.rope_tables(D, 4096, 10000.0, dev)

    def chain(x):
        for _ in range(3):
            h, res = ops.rmsnorm(x, wn, 1e-6, None)
            qkv = ops.gemm(h, wqkv)
            qkv = ops.rope_qkv(qkv, pos, cos, sin, Hq, Hk, D)
            q = qkv[:, : Hq * D].view(T, Hq, D)
            k = qkv[:, Hq * D : (Hq + Hk) * D].view(T, Hk, D)
            v = qkv[:, (Hq + Hk) * D :].view(T, Hk, D)
            ops.kv_cache_write(k, v, slots, kc, vc)
            a = ops.paged_decode_attention(q, kc, vc, table, lens)
            o = ops.gemm(a.reshape(T, Hq * D), wo)
            h, res = ops.rmsnorm(o, wn, 1e-6, res)
            x = ops.gemm(ops.swiglu(ops.gemm(h, wgu)), wd)
        return x

    outs = {}
    try:
        for on in (False, True):
            _lib.set_pdl(on)
            outs[on, "eager"] = chain(x0).clone()
            g = torch.cuda.CUDAGraph()
            static_in = x0.clone()
            s = torch.cuda.Stream()
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                chain(static_in)
            torch.cuda.current_stream().wait_stream(s)
            with torch.cuda.graph(g):
                static_out = chain(static_in)
            for _ in range(3):
                g.replay()
            torch.cuda.synchronize()
            outs[on, "graph"] = static_out.clone()
    finally:
        _lib.set_pdl(True)
    ref = outs[False, "eager"]
    assert torch.isfinite(ref.float()).all()
    for key, val in outs.items():
        assert torch.equal(val, ref), f"{key} differs from the ordinary stream order"


def test_kernels_write_inside_their_buffers():
    """Every output and workspace that the ops allocate sits between canary bands while a battery of kernels runs on
    tile-edge shapes; no band may change (the sanitizer-free memory-safety check of this code base)."""
    from verl_b200 import ops
    from verl_b200.utils.debug.guard_bands import guard_allocations

    torch.manual_seed(5)
    dev = "cuda"
    with guard_allocations() as g:
        for M, N, K in [(1, 72, 64), (127, 136, 200), (129, 264, 72), (300, 4608, 512), (8, 3584, 1024)]:
            a = torch.randn(M, K, device=dev).bfloat16()
            w = torch.randn(N, K, device=dev).bfloat16()
            ops.gemm(a, w)
            ops.gemm(a, w, out_dtype=torch.float32)
        for T, H in [(1, 64), (37, 1000), (130, 3584)]:
            x = torch.randn(T, H, device=dev).bfloat16()
            wn = torch.randn(H, device=dev).bfloat16()
            y, r = ops.rmsnorm(x, wn, 1e-6, x)
            ops.swiglu(torch.randn(T, 2 * 256, device=dev).bfloat16())
        Hq, Hk, D, bs = 8, 2, 128, 16
        for T in (1, 33, 200):
            qkv = torch.randn(T, (Hq + 2 * Hk) * D, device=dev).bfloat16()
            cos, sin = ops.rope_tables(D, 2048, 10000.0, dev)
            qkv = ops.rope_qkv(qkv, torch.arange(T, device=dev), cos, sin, Hq, Hk, D)
            q = qkv[:, : Hq * D].view(T, Hq, D)
            k = qkv[:, Hq * D : (Hq + Hk) * D].view(T, Hk, D)
            v = qkv[:, (Hq + Hk) * D :].view(T, Hk, D)
            cu = torch.tensor([0, T], dtype=torch.int32, device=dev)
            ops.attention_varlen(q.contiguous(), k.contiguous(), v.contiguous(), cu, T, causal=True)
        B, ctx = 5, 77
        nblk = (ctx + bs - 1) // bs
        kc = torch.zeros(B * nblk + 2, Hk, bs, D, device=dev, dtype=torch.bfloat16)
        vc = torch.zeros_like(kc)
        table = torch.arange(B * nblk, device=dev, dtype=torch.int32).reshape(B, nblk)
        lens = torch.tensor([ctx, 1, 16, 17, 64], device=dev, dtype=torch.int32)
        knew = torch.randn(B, Hk, D, device=dev).bfloat16()
        slots = table[torch.arange(B, device=dev), ((lens - 1) // bs).long()].long() * bs + ((lens - 1) % bs).long()
        ops.kv_cache_write(knew, knew, slots, kc, vc)
        q1 = torch.randn(B, Hq, D, device=dev).bfloat16()
        for splits in (1, 3):
            ops.paged_decode_attention(q1, kc, vc, table, lens, num_splits=splits)
        logits = torch.randn(7, 1001, device=dev)
        ops.sample(logits, temperature=torch.ones(7, device=dev), seed=3)
        h = torch.randn(100, 256, device=dev).bfloat16()
        wl = (torch.randn(1000, 256, device=dev) * 0.05).bfloat16()
        ops.lmhead_logprob_entropy(h, wl, torch.randint(0, 1000, (100,), device=dev), 1.0)
        n_checked = g.check()
    assert n_checked >= 30


def test_fused_kernels_write_inside_their_buffers():
    """The same for the few-row and fp8 decode products, gated units, head norms with positions, routed experts, column sums, decode
    attention of heads of 64 and restricted sampling, forward and backward, on ragged sizes."""
    from verl_b200 import ops
    from verl_b200.ops import fp8
    from verl_b200.ops.gemm import colsum
    from verl_b200.ops.moe import moe_gate, moe_mlp
    from verl_b200.utils.debug.guard_bands import guard_allocations

    torch.manual_seed(6)
    dev = "cuda"
    rnd = lambda *s: torch.randn(*s, device=dev).bfloat16()  # noqa: E731
    with guard_allocations() as g:
        with torch.no_grad():
            for M in (1, 9, 17, 31):
                ops.gemm(rnd(M, 520), rnd(1153, 520))
                ops.gemm(rnd(M, 72), rnd(33, 72), out_dtype=torch.float32)
            for M, I, K in ((3, 24, 72), (16, 296, 136), (601, 4872, 264)):
                ops.linear_swiglu(rnd(M, K), rnd(2 * I, K))
            for M, N, K in ((1, 136, 144), (33, 200, 1040), (65, 520, 3584)):
                wq, sw = fp8.quantize_weight(rnd(N, K))
                fp8.fp8_linear(rnd(M, K), wq, sw, None)
        for T, Hq, Hk, D in ((1, 14, 2, 64), (37, 5, 1, 128), (3, 2, 2, 256)):
            pos, tables = torch.arange(T, device=dev), ops.rope_tables(D, 512, 10000.0, dev)
            for norms in (None, (rnd(D).requires_grad_(True), rnd(D).requires_grad_(True))):
                qkv = rnd(T, (Hq + 2 * Hk) * D).requires_grad_(True)
                heads = ops.qkv_heads(qkv, pos, *tables, Hq, Hk, D, norms, 1e-6)
                torch.autograd.backward(heads, [torch.randn_like(h) for h in heads])
                with torch.no_grad():
                    ops.qkv_heads(qkv, pos, *tables, Hq, Hk, D, norms, 1e-6, in_place=False)
        for T, E, k, H, I in ((1, 8, 2, 64, 64), (45, 33, 8, 192, 64), (300, 4, 1, 128, 128)):
            z = rnd(T, E).requires_grad_(True)
            w, idx = moe_gate(z, k, True)
            leaves = [t.requires_grad_(True) for t in (rnd(T, H), rnd(E, 2 * I, H), rnd(E, H, I))]
            moe_mlp(leaves[0], idx, w, leaves[1], leaves[2], ops.swiglu).backward(rnd(T, H))
        for T, N in ((7, 34), (513, 1026)):
            colsum(rnd(T, N))
        B, Hq, Hk, D, bs, ctx = 5, 14, 2, 64, 16, 77
        n = (ctx + bs - 1) // bs
        table = torch.arange(B * n, device=dev, dtype=torch.int32).reshape(B, n)
        lens = torch.tensor([ctx, 1, 16, 17, 64], device=dev, dtype=torch.int32)
        for splits in (1, 3):
            ops.paged_decode_attention(rnd(B, Hq, D), rnd(B * n, Hk, bs, D), rnd(B * n, Hk, bs, D), table, lens, num_splits=splits)
        for rows, V in ((3, 5003), (150, 1025)):
            full = lambda v, dt: torch.full((rows,), v, dtype=dt, device=dev)  # noqa: B023,E731
            ops.sample(torch.randn(rows, V, device=dev), top_k=full(20, torch.int32), top_p=full(0.9, torch.float32), seed=3)
        n_checked = g.check()
    assert n_checked >= 60
