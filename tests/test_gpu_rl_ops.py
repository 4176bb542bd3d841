"""Fused RL-step kernels against their PyTorch twins: the token-mean GRPO objective (loss, statistics, gradient), the
mixture-of-experts routing decision, and the expert FFN whose grouped-GEMM tile tables are built on the device."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kl", [None, "low_var_kl", "kl", "mse", "abs"])
@pytest.mark.parametrize("weighted", [False, True])
def test_grpo_token_loss_matches_the_composed_torch_ops(kl, weighted):
    from arctic_platform_b200.ops import _lib, rl_ops
    from arctic_platform_b200.rl.processors.functional import agg_loss, kl_penalty, ppo_clip_token_loss
    g = torch.Generator(device="cuda").manual_seed(5)
    n = 10_007
    lp = (torch.randn(n, generator=g, device="cuda") * 0.7 - 2.0).requires_grad_(True)
    old = lp.detach() + torch.randn(n, generator=g, device="cuda") * 0.5
    old[::97] -= 30.0                                         # beyond the +-20 clamp of the log ratio
    ref = lp.detach() + torch.randn(n, generator=g, device="cuda") * 0.3
    adv = torch.randn(n, generator=g, device="cuda")
    mask = torch.rand(n, generator=g, device="cuda") > 0.2
    w = torch.rand(n, generator=g, device="cuda") + 0.5 if weighted else None
    dp, ntok, coef = 2, 12345.0, 0.01
    # twin
    lp2 = lp.detach().clone().requires_grad_(True)
    tok, d, clipped, lower = ppo_clip_token_loss(lp2, old, adv, 0.2, 0.2, 3.0)
    if w is not None:
        tok = tok * w
    want = agg_loss(tok, mask, "token-mean", dp_size=dp, batch_num_tokens=ntok)
    if kl:
        kld = kl_penalty(lp2, ref, kl)
        want = want + coef * agg_loss(kld, mask, "token-mean", dp_size=dp, batch_num_tokens=ntok)
    want.backward()
    # fused
    loss, sums = rl_ops.grpo_token_loss(lp, old, adv, mask, dp / ntok, ref_lp=ref if kl else None, kl_kind=kl,
                                        kl_coef=coef if kl else 0.0, weight=w)
    (loss * 3.0).backward()
    _lib.check_status("grpo kernel")
    assert float(loss) == pytest.approx(float(want), rel=2e-5, abs=1e-7)
    assert torch.allclose(lp.grad / 3.0, lp2.grad, rtol=2e-4, atol=1e-9)
    mf = mask.float()
    s = sums.tolist()
    assert s[0] == float(mf.sum()) and s[1] == float((clipped.float() * mf).sum()) and s[3] == float((lower.float() * mf).sum())
    assert s[2] == pytest.approx(float((-d.detach() * mf).sum()), rel=1e-4)
    assert s[4] == pytest.approx(float((tok.detach() * mf).sum()), rel=1e-4)


@pytest.mark.parametrize("E,k,score", [(128, 8, "softmax"), (64, 6, "sigmoid"), (8, 2, "softmax"), (384, 8, "softmax")])
def test_route_kernel_picks_the_same_experts_as_topk(E, k, score):
    from arctic_platform_b200.ops import _lib, rl_ops
    g = torch.Generator(device="cuda").manual_seed(E)
    T = 777
    logits = torch.randn(T, E, generator=g, device="cuda") * 2.0
    bias = torch.randn(E, generator=g, device="cuda") * 0.1
    counts = torch.zeros(E, device="cuda", dtype=torch.int32)
    idx = rl_ops.moe_route(logits, k, score, bias, counts)
    _lib.check_status("route")
    scores = torch.softmax(logits, -1) if score == "softmax" else torch.sigmoid(logits)
    want = torch.topk(scores + bias, k, dim=-1).indices
    assert torch.equal(idx.sort(-1).values, want.sort(-1).values)
    assert torch.equal(idx, want)                                            # best first, like topk
    assert torch.equal(counts.long(), torch.bincount(want.reshape(-1), minlength=E))


def test_moe_layer_forward_and_backward_with_device_built_tiles():
    """The expert FFN with tile tables written by a kernel (no copy of the expert histogram to the host in the forward)
    against the per-expert fp32 loop, values and gradients; skewed routing with empty experts."""
    import dataclasses
    from arctic_platform_b200.models.config import PRESETS
    from arctic_platform_b200.models.moe import MoEFeedForward, grouped_ffn
    from arctic_platform_b200.ops import _lib
    name = next((n for n in PRESETS if PRESETS[n].is_moe and PRESETS[n].moe_activation == "swiglu"
                 and not PRESETS[n].layer_types), None)
    if name is None:
        pytest.skip("no plain MoE preset")
    cfg = dataclasses.replace(PRESETS[name], hidden_size=256, moe_intermediate_size=128, num_experts=16,
                              num_experts_per_tok=4, shared_expert_intermediate_size=0)
    torch.manual_seed(0)
    moe = MoEFeedForward(cfg, "cuda", torch.bfloat16)
    for p in moe.parameters():
        p.data.normal_(0, 0.05)
    R = 700
    counts = torch.tensor([300, 0, 5, 128, 129, 0, 0, 1, 37, 0, 100, 0, 0, 0, 0, 0], device="cuda")
    x = (torch.randn(R, cfg.hidden_size, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_(True)
    y = grouped_ffn(x, moe.wgu, moe.wdown, counts)
    y.float().pow(2).sum().backward()
    _lib.check_status("moe device tiles")
    xr = x.detach().float().requires_grad_(True)
    outs, row = [], 0
    for e, c in enumerate(counts.tolist()):
        gu = xr[row:row + c] @ moe.wgu[e].float().t()
        outs.append((torch.nn.functional.silu(gu[:, 0::2]) * gu[:, 1::2]) @ moe.wdown[e].float().t())
        row += c
    ref = torch.cat(outs)
    ref.pow(2).sum().backward()
    assert (y.float() - ref).abs().max() < 3e-2 * ref.abs().max() + 1e-3
    assert (x.grad.float() - xr.grad).abs().max() < 5e-2 * xr.grad.abs().max() + 1e-3


@pytest.mark.parametrize("tokens,experts,top_k", [(300, 16, 4), (37, 8, 2), (1024, 64, 8)])
def test_moe_layer_padded_plan_backward_matches_per_expert_fp32(tokens, experts, top_k):
    """Training path of the expert layer: padded expert-major rows, forward, data gradients and weight gradients as
    grouped GEMMs planned by a kernel (no expert count reaches the host) against an fp32 per-expert loop; skewed
    routing leaves some experts without tokens."""
    import dataclasses
    from arctic_platform_b200.models.config import PRESETS
    from arctic_platform_b200.models.moe import MoEFeedForward
    from arctic_platform_b200.ops import _lib
    cfg = dataclasses.replace(PRESETS["qwen3-moe-tiny"], hidden_size=256, moe_intermediate_size=192, num_experts=experts,
                              num_experts_per_tok=top_k, shared_expert_intermediate_size=0)
    torch.manual_seed(1)
    moe = MoEFeedForward(cfg, "cuda", torch.bfloat16)
    for p in moe.parameters():
        p.data.normal_(0, 0.05)
    moe.router.data[experts // 2:] -= 1.0                          # starve the upper half of the experts
    x = (torch.randn(tokens, 256, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_(True)
    from arctic_platform_b200.models.moe import route_topk
    route = lambda lg, forced: route_topk(lg, top_k, cfg.norm_topk_prob, cfg.moe_score_func, cfg.moe_route_scale, None,
                                          forced, cfg.moe_n_group, cfg.moe_topk_group)
    with torch.no_grad():
        _, idx = route((x.float() @ moe.router.float().t()), None)
    moe.routed_experts = idx                                       # both sides route identically
    y = moe(x)
    (y.float() * torch.linspace(-1, 1, 256, device="cuda")).sum().backward()
    _lib.check_status("moe padded plan")
    # oracle: same routing decision, fp32 math (the routing weights carry gradient to x through the router)
    xr = x.detach().float().requires_grad_(True)
    wgu = moe.wgu.detach().float().requires_grad_(True)
    wdn = moe.wdown.detach().float().requires_grad_(True)
    w, _ = route(xr @ moe.router.detach().float().t(), idx)
    out = torch.zeros(tokens, 256, device="cuda")
    for e in range(experts):
        tok, slot = (idx == e).nonzero(as_tuple=True)
        if tok.numel() == 0:
            continue
        gu = xr[tok] @ wgu[e].t()
        ye = (torch.nn.functional.silu(gu[:, 0::2]) * gu[:, 1::2]) @ wdn[e].t()
        out = out.index_add(0, tok, ye * w[tok, slot, None].float())
    (out * torch.linspace(-1, 1, 256, device="cuda")).sum().backward()
    tol = lambda ref: 4e-2 * ref.abs().max() + 1e-3
    assert (y.float() - out).abs().max() < tol(out)
    assert (x.grad.float() - xr.grad).abs().max() < tol(xr.grad)
    g_gu = moe.wgu.grad_f32 if getattr(moe.wgu, "grad_f32", None) is not None else moe.wgu.grad.float()
    g_dn = moe.wdown.grad_f32 if getattr(moe.wdown, "grad_f32", None) is not None else moe.wdown.grad.float()
    assert (g_gu - wgu.grad).abs().max() < tol(wgu.grad)
    assert (g_dn - wdn.grad).abs().max() < tol(wdn.grad)
    starved = (torch.bincount(idx.reshape(-1), minlength=experts) == 0).nonzero().flatten().tolist()
    for e in starved:                                              # experts without tokens: exactly zero gradient
        assert float(g_gu[e].abs().max()) == 0.0 and float(g_dn[e].abs().max()) == 0.0


@pytest.mark.parametrize("E,k", [(8, 2), (60, 4), (128, 8), (512, 10), (33, 33)])
@pytest.mark.parametrize("score", ["softmax", "sigmoid"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_route_without_gradients_has_the_bits_of_the_pass_with_them(E, k, score, dtype):
    """Decision and weights from one kernel where no gradient is wanted: those of the softmax, gather and division behind a decision, to
    the bit, with and without a bias, normalised and scaled; rows with a stride."""
    from arctic_platform_b200.models.moe import route_topk
    torch.manual_seed(E)
    x = (torch.randn(1037, E + 3, device="cuda") * 3).to(dtype)[:, :E]
    bias = torch.randn(E, device="cuda")
    for b, renorm, scale in ((None, True, 1.0), (bias, False, 2.5), (bias, True, 0.5)):
        w0, i0 = route_topk(x.clone().requires_grad_(), k, renorm, score, scale, b)
        w1, i1 = route_topk(x, k, renorm, score, scale, b)
        assert torch.equal(i0, i1) and torch.equal(w0.detach(), w1)


@pytest.mark.parametrize("E,k", [(8, 3), (33, 33), (40, 6), (512, 10)])
@pytest.mark.parametrize("grad", [False, True])
def test_route_names_experts_whatever_the_logits_are(E, k, grad):
    """NaN, infinities and a bias that leaves fewer experts than are chosen: every choice is one of the experts, none twice; scores that
    are left are chosen in their order, ahead of the others; rows of plain numbers next to them choose as by themselves."""
    from arctic_platform_b200.models.moe import route_topk
    nan, inf = float("nan"), float("inf")
    torch.manual_seed(E)
    x = torch.randn(64, E, device="cuda")
    plain = x.clone()
    x[1::8] = nan
    x[2::8, ::3] = nan
    x[3::8] = -inf
    x[4::8, 1] = inf
    x[5::8, 2:] = -inf
    shut = torch.full((E,), -inf, device="cuda")
    shut[-2:] = 0
    with torch.set_grad_enabled(grad):
        for score in ("softmax", "sigmoid"):
            for bias in (None, shut):
                idx = route_topk(x.clone().requires_grad_(grad), k, True, score, 1.0, bias)[1]
                assert ((idx >= 0) & (idx < E)).all() and (idx.sort(1).values.diff(dim=1) > 0).all()
                alone = route_topk(plain[::8].clone().requires_grad_(grad), k, True, score, 1.0, bias)[1]
                assert torch.equal(idx[::8], alone)
                if bias is not None:
                    assert torch.equal(alone[:, :2].sort(1).values, torch.tensor([[E - 2, E - 1]] * 8, device="cuda"))
            if k <= E - (E + 2) // 3:
                some = route_topk(x[2::8].clone().requires_grad_(grad), k, True, "sigmoid")[1]
                assert torch.equal(some, x[2::8].nan_to_num(-1e9).topk(k, dim=1).indices)


@pytest.mark.parametrize("score", ["softmax", "sigmoid"])
@pytest.mark.parametrize("grad", [False, True])
def test_route_keeps_a_forward_mode_tangent(score, grad):
    """Weights of logits that carry a tangent carry one too, with and without gradients enabled: the derivative of scores, gather and
    division in 64 bits (fp32 sums of up to 40 terms: 1e-5)."""
    import torch.autograd.forward_ad as fw
    from arctic_platform_b200.models.moe import route_topk
    torch.manual_seed(4)
    x, t = torch.randn(31, 40, device="cuda") * 2, torch.randn(31, 40, device="cuda")
    with torch.set_grad_enabled(grad), fw.dual_level():
        w, idx = route_topk(fw.make_dual(x, t), 5, True, score, 1.5)
        got = fw.unpack_dual(w)
        assert got.tangent is not None and got.tangent.dtype == torch.float32

        def weights(y):
            s = (torch.softmax(y, -1) if score == "softmax" else torch.sigmoid(y)).gather(-1, idx)
            return s / s.sum(-1, keepdim=True) * 1.5

    want, slope = torch.func.jvp(weights, (x.double(),), (t.double(),))
    assert (got.primal - want).abs().max() <= 1e-5 and (got.tangent - slope).abs().max() <= 1e-5 * slope.abs().max()
    with torch.set_grad_enabled(grad):
        w0, idx0 = route_topk(x, 5, True, score, 1.5)
    assert torch.equal(idx, idx0) and torch.equal(got.primal, w0)


@pytest.mark.parametrize("E", [1, 2, 7, 64, 129, 511, 512])
def test_group_tiles_of_any_number_of_experts(E):
    """Prefix sums of two experts a thread: odd and even numbers, experts without rows, more than a block of rows."""
    from arctic_platform_b200.models.moe import build_group_tiles, device_group_tiles
    g = torch.Generator().manual_seed(E)
    counts = torch.randint(0, 300, (E,), generator=g)
    counts[::3] = 0
    t1, t2, n, _, _ = device_group_tiles(counts.to(torch.int32).cuda(), int(counts.sum()), 384, 200)
    for got, live, width in ((t1, int(n[0]), 384), (t2, int(n[1]), 200)):
        assert torch.equal(got[:live].cpu(), build_group_tiles(counts, width, "cpu"))
