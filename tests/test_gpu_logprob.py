"""Fused lm_head log-prob / entropy kernel against the fp32 chunked reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,H,V", [(300, 256, 32000), (129, 512, 151936), (5, 128, 1000)])
@pytest.mark.parametrize("per_row_temp", [False, True])
def test_logprob_forward_backward(N, H, V, per_row_temp):
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops.logprob import lm_head_logprobs, logprobs_entropy_ref
    torch.manual_seed(0)
    hidden = torch.randn(N, H, device="cuda").bfloat16().requires_grad_()
    weight = (torch.randn(V, H, device="cuda") * 0.05).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (N,), device="cuda")
    it = (0.5 + torch.rand(N, device="cuda")) if per_row_temp else 0.7
    lp, ent = lm_head_logprobs(hidden, weight, labels, it, with_entropy=True, bwd_chunk=128)
    g1, g2 = torch.randn(N, device="cuda"), torch.randn(N, device="cuda") * 0.1
    ((lp * g1).sum() + (ent * g2).sum()).backward()
    _lib.check_status("lmhead")
    hr, wr = hidden.detach().float().requires_grad_(), weight.detach().float().requires_grad_()
    lpr, entr = logprobs_entropy_ref(hr, wr, labels, it, True)
    ((lpr * g1).sum() + (entr * g2).sum()).backward()
    assert torch.allclose(lp, lpr.detach(), atol=3e-2, rtol=1e-2), (lp - lpr).abs().max()
    assert torch.allclose(ent, entr.detach(), atol=3e-2, rtol=1e-2), (ent - entr).abs().max()
    for got, ref, nm in ((hidden.grad, hr.grad, "dh"), (weight.grad, wr.grad, "dw")):
        err = (got.float() - ref).abs().max().item()
        sc = ref.abs().max().item()
        assert err <= 3e-2 * sc + 1e-3, f"{nm}: {err} vs scale {sc}"


@pytest.mark.parametrize("N,H,V", [(129, 64, 1032), (256, 72, 1280), (385, 2560, 4232), (700, 1024, 136)])
def test_row_and_column_remainders_of_pair_tiles(N, H, V):
    """More than one 128-row tile runs on CTA pairs of 256 x 256: odd rows, a last tile of 8, 128 or 136 columns.  The logits of
    both sides have the same bf16 operands, so log-probabilities differ by fp32 rounding of sums and exponentials (V terms of
    2^-22 relative, 1e-4 with room); gradients pass through bf16 once per d(logits) and once per result (2^-8 at most each, half of that in the mean)."""
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops.logprob import lm_head_logprobs, logprobs_entropy_ref
    g = torch.Generator(device="cuda").manual_seed(N)
    hidden = torch.randn(N, H, device="cuda", generator=g).bfloat16().requires_grad_()
    weight = (torch.randn(V, H, device="cuda", generator=g) * 2 * H ** -0.5).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (N,), device="cuda", generator=g)
    labels[:2] = torch.tensor([0, V - 1], device="cuda")
    g1, g2 = (torch.randn(N, device="cuda", generator=g) for _ in range(2))
    lp, ent = lm_head_logprobs(hidden, weight, labels)
    ((lp * g1).sum() + 0.1 * (ent * g2).sum()).backward()
    _lib.check_status("lmhead")
    hr, wr = (t.detach().double().requires_grad_() for t in (hidden, weight))
    z = torch.log_softmax(hr @ wr.T, -1)
    lpr, entr = z.gather(1, labels[:, None])[:, 0], -(z.exp() * z).sum(-1)
    ((lpr * g1).sum() + 0.1 * (entr * g2).sum()).backward()
    for got, ref in ((lp, lpr), (ent, entr)):
        assert (got - ref).abs().max() <= 1e-4 * max(1.0, ref.abs().max().item())
    for got, ref in ((hidden.grad, hr.grad), (weight.grad, wr.grad)):
        assert (got.double() - ref).norm() <= 2 ** -7 * ref.norm()


def test_gradients_where_memory_is_short():
    """Without memory to spare d(logits) takes 4096 rows at a time; the gradients are those of one chunk but for the order of the
    sums.  The tensor cores cut each step of 16 rows to the 24 bits of the running fp32 sum: N / 16 steps of 2^-23 at most.  The
    hidden gradient is rounded to bf16 once on each side, 2^-9."""
    from arctic_platform_b200.ops.logprob import lm_head_logprobs
    from arctic_platform_b200.utils import memory_budget
    N, H, V = 9000, 128, 32000
    g = torch.Generator(device="cuda").manual_seed(2)
    hidden = torch.randn(N, H, device="cuda", generator=g).bfloat16()
    weight = (torch.randn(V, H, device="cuda", generator=g) * H ** -0.5).bfloat16()
    labels = torch.randint(0, V, (N,), device="cuda", generator=g)
    spare, got = memory_budget.spare_bytes, []
    try:
        for free in (0, 1 << 40):
            memory_budget.spare_bytes = lambda device, wanted: free
            h, w = hidden.clone().requires_grad_(), weight.clone().requires_grad_()
            w.grad_f32 = torch.zeros(V, H, device="cuda")
            lp, _ = lm_head_logprobs(h, w, labels)
            torch.cuda.synchronize()
            before = torch.cuda.memory_allocated()
            torch.cuda.reset_peak_memory_stats()
            lp.sum().backward()
            got.append((h.grad, w.grad_f32, torch.cuda.max_memory_allocated() - before))
    finally:
        memory_budget.spare_bytes = spare
    short, long = got
    assert short[2] <= 4096 * V * 2 + (32 << 20) < long[2]
    assert (short[1] - long[1]).norm() <= N / 16 * 2 ** -23 * long[1].norm()
    assert (short[0].double() - long[0].double()).norm() <= 2 ** -8 * long[0].double().norm()
