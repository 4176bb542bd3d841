"""RMSNorm / qk-norm+RoPE / SwiGLU kernels against fp32 PyTorch expressions."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(shape, scale=1.0):
    return (torch.randn(shape, device="cuda", dtype=torch.float32) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("T,H", [(7, 256), (513, 2560), (64, 8192)])
@pytest.mark.parametrize("with_res", [False, True])
def test_rmsnorm_fwd_bwd(T, H, with_res):
    from arctic_platform_b200.ops import _lib, norm
    x = _rand((T, H)).requires_grad_()
    res = _rand((T, H)).requires_grad_() if with_res else None
    w = (1 + 0.1 * torch.randn(H, device="cuda")).to(torch.bfloat16).requires_grad_()
    y, stream = norm.rmsnorm(x, w, 1e-6, res)
    dy, ds = _rand((T, H)), _rand((T, H))
    (y.float() * dy.float()).sum().add((stream.float() * ds.float()).sum() if with_res else 0).backward()
    _lib.check_status("rmsnorm")
    xr = x.detach().float().requires_grad_()
    rr = res.detach().float().requires_grad_() if with_res else None
    wr = w.detach().float().requires_grad_()
    xs = xr + rr if with_res else xr
    if with_res:
        xs_q = xs.detach().to(torch.bfloat16).float()
        xs = xs + (xs_q - xs).detach()
    yr = xs * torch.rsqrt(xs.pow(2).mean(-1, keepdim=True) + 1e-6) * wr
    ((yr * dy.float()).sum() + ((xs * ds.float()).sum() if with_res else 0)).backward()
    assert torch.allclose(y.float(), yr.detach(), atol=3e-2, rtol=2e-2)
    assert torch.allclose(x.grad.float(), xr.grad, atol=6e-2, rtol=3e-2)
    if with_res:
        assert torch.allclose(res.grad.float(), rr.grad, atol=6e-2, rtol=3e-2)
    rel = (w.grad.float() - wr.grad).abs().max() / (wr.grad.abs().max() + 1e-6)
    assert rel < 2e-2, rel


@pytest.mark.parametrize("D", [64, 128])
def test_qknorm_rope_fwd_bwd(D):
    from arctic_platform_b200.ops import _lib, norm
    T, Hq, Hkv = 131, 8, 2
    qkv = _rand((T, (Hq + 2 * Hkv) * D)).requires_grad_()
    wq = (1 + 0.1 * torch.randn(D, device="cuda")).to(torch.bfloat16).requires_grad_()
    wk = (1 + 0.1 * torch.randn(D, device="cuda")).to(torch.bfloat16).requires_grad_()
    cos_t, sin_t = norm.rope_tables(4096, D, 1e6, "cuda")
    pos = torch.randint(0, 4096, (T,), device="cuda", dtype=torch.int32)
    q, k, v = norm.qknorm_rope(qkv, wq, wk, cos_t, sin_t, pos, Hq, Hkv, D)
    gq, gk, gv = _rand(q.shape), _rand(k.shape), _rand(v.shape)
    ((q.float() * gq.float()).sum() + (k.float() * gk.float()).sum() + (v.float() * gv.float()).sum()).backward()
    _lib.check_status("qknorm_rope")
    qkvr = qkv.detach().float().requires_grad_()
    wqr, wkr = wq.detach().float().requires_grad_(), wk.detach().float().requires_grad_()
    q0 = qkvr[:, :Hq * D].reshape(T, Hq, D)
    k0 = qkvr[:, Hq * D:(Hq + Hkv) * D].reshape(T, Hkv, D)
    v0 = qkvr[:, (Hq + Hkv) * D:].reshape(T, Hkv, D)
    qr, kr = norm.qknorm_rope_ref(q0, k0, wqr, wkr, cos_t, sin_t, pos, 1e-6)
    ((qr * gq.float()).sum() + (kr * gk.float()).sum() + (v0 * gv.float()).sum()).backward()
    assert torch.allclose(q.float(), qr.detach(), atol=3e-2, rtol=2e-2)
    assert torch.allclose(k.float(), kr.detach(), atol=3e-2, rtol=2e-2)
    assert torch.equal(v, v0.detach().to(torch.bfloat16))
    assert torch.allclose(qkv.grad.float(), qkvr.grad, atol=8e-2, rtol=3e-2)
    for g, gr in ((wq.grad, wqr.grad), (wk.grad, wkr.grad)):
        rel = (g.float() - gr).abs().max() / (gr.abs().max() + 1e-6)
        assert rel < 2e-2, rel


def test_swiglu_fwd_bwd():
    from arctic_platform_b200.ops import _lib, norm
    gu = _rand((257, 2 * 688)).requires_grad_()
    act = norm.swiglu(gu)
    d = _rand(act.shape)
    act.backward(d)
    _lib.check_status("swiglu")
    gr = gu.detach().float().requires_grad_()
    ar = torch.nn.functional.silu(gr[:, 0::2]) * gr[:, 1::2]
    ar.backward(d.float())
    assert torch.allclose(act.float(), ar.detach(), atol=3e-2, rtol=2e-2)
    assert torch.allclose(gu.grad.float(), gr.grad, atol=5e-2, rtol=3e-2)


@pytest.mark.parametrize("T,H,Dk,Dv", [(200, 4, 128, 128), (64, 2, 32, 48), (1000, 3, 64, 128)])
def test_delta_rule_scan_kernel_matches_the_token_by_token_recurrence(T, H, Dk, Dv):
    """The chunk recurrence of the gated delta rule as one kernel (no-grad passes) against the token-by-token oracle
    and against the differentiable PyTorch loop, with and without a carried-in state."""
    from arctic_platform_b200.models.linear_attention import gated_delta_rule_chunked, gated_delta_rule_recurrent
    from arctic_platform_b200.ops import _lib
    g = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn(T, H, Dk, device="cuda", generator=g)
    k = torch.randn(T, H, Dk, device="cuda", generator=g)
    v = torch.randn(T, H, Dv, device="cuda", generator=g)
    gate = -torch.rand(T, H, device="cuda", generator=g) * 0.3
    beta = torch.rand(T, H, device="cuda", generator=g)
    S0 = torch.randn(H, Dk, Dv, device="cuda", generator=g) * 0.1
    for state in (None, S0):
        want_o, want_S = gated_delta_rule_recurrent(q, k, v, gate, beta, state)
        with torch.no_grad():
            got_o, got_S = gated_delta_rule_chunked(q, k, v, gate, beta, state)            # kernel
        _lib.check_status("delta rule scan")
        with torch.enable_grad():
            loop_o, loop_S = gated_delta_rule_chunked(q, k, v, gate, beta, state)          # PyTorch loop
        for a, b in ((got_o, want_o), (got_S, want_S), (got_o, loop_o), (got_S, loop_S)):
            assert (a - b).abs().max() < 2e-3 * b.abs().max() + 1e-4


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("T,Hq,Hkv", [(1, 4, 2), (37, 3, 1), (513, 8, 2)])
def test_qknorm_rope_of_rows_off_a_16_byte_boundary(D, T, Hq, Hkv):
    """Rows, weights and tables that begin anywhere have the results of aligned ones, to the bit, with and without weights; both agree
    with fp32 (bf16 outputs: 2^-8 of a value and a little for the sums)."""
    from arctic_platform_b200.ops import norm
    torch.manual_seed(D + T)
    width = (Hq + 2 * Hkv) * D
    wide = torch.randn(T, width + 13, device="cuda").bfloat16()
    off = wide[:, 3:3 + width]
    w = [torch.randn(2 * D + 5, device="cuda").bfloat16()[i * D + 1:(i + 1) * D + 1] for i in (0, 1)]
    cos_t, sin_t = norm.rope_tables(700, D, 1e4, "cuda")
    shift = [torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view_as(t) for t in (cos_t, sin_t)]
    pos = torch.randint(0, 700, (T,), device="cuda", dtype=torch.int32)
    for wq, wk in (w, (None, None)):
        q0, k0, _ = norm.qknorm_rope(off.contiguous(), *(None if x is None else x.clone() for x in (wq, wk)), cos_t, sin_t, pos, Hq, Hkv, D)
        q1, k1, _ = norm.qknorm_rope(off, wq, wk, *shift, pos, Hq, Hkv, D)
        assert torch.equal(q0, q1) and torch.equal(k0, k1)
        ref = norm.qknorm_rope_ref(off[:, :Hq * D].reshape(T, Hq, D).float(), off[:, Hq * D:(Hq + Hkv) * D].reshape(T, Hkv, D).float(),
                                   wq, wk, cos_t, sin_t, pos, 1e-6)
        for got, want in zip((q0, k0), ref):
            assert (got.float() - want).abs().max() <= 2 ** -8 * want.abs().max() + 1e-4


@pytest.mark.parametrize("H", [8, 1024, 2048, 2056, 2560, 4104, 8192])
@pytest.mark.parametrize("T", [1, 1185, 2400])
def test_rows_after_rows_in_one_block(H, T):
    """RMSNorm forward and backward where a block walks several rows (1184 blocks and fewer), at the widths where the vectors per thread
    change: as single rows give it, to the bit."""
    from arctic_platform_b200.ops import norm
    torch.manual_seed(H)
    x, res, dy, dst = (torch.randn(T, H, device="cuda").bfloat16() for _ in range(4))
    w = torch.randn(H, device="cuda").bfloat16()

    def run(rows):
        a, b = x[rows].clone().requires_grad_(), res[rows].clone().requires_grad_()
        y, stream = norm.rmsnorm(a, w, 1e-6, b)
        torch.autograd.backward([y, stream], [dy[rows], dst[rows]])
        return y.detach(), stream.detach(), a.grad

    whole = run(slice(0, T))
    for r in {0, T // 2, T - 1}:
        for got, want in zip(run(slice(r, r + 1)), whole):
            assert torch.equal(got[0], want[r])


@pytest.mark.parametrize("T,I", [(1, 8), (3, 1000), (700, 4864), (2049, 2056)])
def test_swiglu_backward_two_sets_a_thread(T, I):
    """Odd numbers of sets, fewer than threads and more than two rounds; bf16 results against fp32."""
    from arctic_platform_b200.ops import norm
    torch.manual_seed(T)
    gu = torch.randn(T, 2 * I, device="cuda").bfloat16().requires_grad_()
    d = torch.randn(T, I, device="cuda").bfloat16()
    norm.swiglu(gu).backward(d)
    ref = gu.detach().float().requires_grad_()
    (torch.nn.functional.silu(ref[:, 0::2]) * ref[:, 1::2]).backward(d.float())
    assert (gu.grad.float() - ref.grad).abs().max() <= 2 ** -8 * ref.grad.abs().max()
