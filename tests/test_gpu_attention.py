"""tcgen05 segment attention (varlen causal + ZoRRo shared prefix) against the dense fp32 reference."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(shape, scale=1.0):
    return (torch.randn(shape, device="cuda", dtype=torch.float32) * scale).to(torch.bfloat16)


def _layouts():
    from arctic_platform_b200.ops.attention import AttnLayout
    varlen = AttnLayout.from_cu_seqlens([0, 1, 130, 386, 700, 1212])
    # two groups: prompt 300 with responses 70 / 130 / 1, prompt 129 with responses 256 / 40
    segs, t = [], 0
    for plen, rlens in ((300, (70, 130, 1)), (129, (256, 40))):
        p0 = t
        segs.append([p0, plen, 0, 0, p0, plen])
        t += plen
        for r in rlens:
            segs.append([t, r, p0, plen, t, r])
            t += r
    zorro = AttnLayout(np.array(segs, dtype=np.int32), t)
    return {"varlen": varlen, "zorro": zorro}


@pytest.mark.parametrize("name", ["varlen", "zorro"])
@pytest.mark.parametrize("Hq,Hkv,D", [(4, 2, 128), (8, 2, 128), (2, 2, 128), (4, 2, 64)])
def test_attention_forward(name, Hq, Hkv, D):
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops.attention import attention_fwd_cuda, attention_ref
    layout = _layouts()[name]
    T = layout.total_tokens
    q, k, v = _rand((T, Hq, D)), _rand((T, Hkv, D)), _rand((T, Hkv, D))
    o, lse = attention_fwd_cuda(q, k, v, layout, D ** -0.5)
    _lib.check_status("attn fwd")
    o_ref, lse_ref = attention_ref(q, k, v, layout, D ** -0.5, return_lse=True)
    assert torch.allclose(o.float(), o_ref.float(), atol=2e-2, rtol=2e-2), (o.float() - o_ref.float()).abs().max()
    assert torch.allclose(lse, lse_ref, atol=2e-2, rtol=1e-3)


@pytest.mark.parametrize("name", ["varlen", "zorro"])
@pytest.mark.parametrize("Hq,Hkv", [(4, 2), (8, 2), (2, 2)])
def test_attention_backward(name, Hq, Hkv):
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops.attention import attention_ref, segment_attention
    D = 128
    layout = _layouts()[name]
    T = layout.total_tokens
    q, k, v = (_rand((T, Hq, D)).requires_grad_(), _rand((T, Hkv, D)).requires_grad_(),
               _rand((T, Hkv, D)).requires_grad_())
    d_o = _rand((T, Hq, D))
    o = segment_attention(q, k, v, layout)
    o.backward(d_o)
    _lib.check_status("attn bwd")
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    o_ref = attention_ref(qr, kr, vr, layout)
    o_ref.backward(d_o.float())
    for got, ref, nm in ((q.grad, qr.grad, "dq"), (k.grad, kr.grad, "dk"), (v.grad, vr.grad, "dv")):
        err = (got.float() - ref).abs().max().item()
        scale = ref.abs().max().item()
        assert err <= 2e-2 * scale + 2e-2, f"{nm}: err {err} scale {scale}"


def test_zorro_matches_replicated_layout():
    """Shared-prefix attention equals ordinary causal attention on [prompt || response] copies."""
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops.attention import AttnLayout, attention_fwd_cuda
    Hq, Hkv, D, P = 4, 2, 128, 333
    rl = (100, 57)
    T = P + sum(rl)
    q, k, v = _rand((T, Hq, D)), _rand((T, Hkv, D)), _rand((T, Hkv, D))
    segs, t = [[0, P, 0, 0, 0, P]], P
    for r in rl:
        segs.append([t, r, 0, P, t, r])
        t += r
    o, _ = attention_fwd_cuda(q, k, v, AttnLayout(np.array(segs, dtype=np.int32), T), D ** -0.5)
    t = P
    for r in rl:
        idx = torch.cat([torch.arange(P), torch.arange(t, t + r)]).cuda()
        o2, _ = attention_fwd_cuda(q[idx].contiguous(), k[idx].contiguous(), v[idx].contiguous(),
                                   AttnLayout.from_cu_seqlens([0, P + r]), D ** -0.5)
        assert torch.allclose(o2[P:].float(), o[t:t + r].float(), atol=1e-2, rtol=1e-2)
        t += r
    _lib.check_status("attn zorro")


@pytest.mark.parametrize("Hq,Hkv", [(3, 3), (4, 1), (10, 2), (16, 2)])
@pytest.mark.parametrize("sharp", [1.0, 4.0])
def test_tile_edges_and_sharp_scores_against_64_bits(Hq, Hkv, sharp):
    """Lengths around the 128-row tiles, prompts shared by several responses, every number of query heads per key head, and scores
    wide enough that running maxima and references move.  o, P and dS are bf16 operands (2^-8 at most each) of sums that cancel in
    dS: a few times that of a gradient's norm."""
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops.attention import AttnLayout, attention_ref, segment_attention
    segs, t = [], 0
    for plen, rlens in ((127, ()), (128, ()), (129, (1, 127)), (257, (128, 129, 33)), (64, (65,)), (1, (1,)), (384, (300,))):
        p0 = t
        segs.append([p0, plen, 0, 0, p0, plen])
        t += plen
        for r in rlens:
            segs.append([t, r, p0, plen, t, r])
            t += r
    layout = AttnLayout(np.array(segs, dtype=np.int32), t)
    torch.manual_seed(Hq)
    q, k, v = _rand((t, Hq, 128), sharp).requires_grad_(), _rand((t, Hkv, 128)).requires_grad_(), _rand((t, Hkv, 128)).requires_grad_()
    d_o = _rand((t, Hq, 128))
    o = segment_attention(q, k, v, layout)
    o.backward(d_o)
    _lib.check_status("attention")
    qr, kr, vr = (x.detach().double().requires_grad_() for x in (q, k, v))
    ref = _attention64(qr, kr, vr, layout)
    ref.backward(d_o.double())
    assert (o.double() - ref).norm() <= 2 ** -7 * ref.norm()
    for got, want in ((q.grad, qr.grad), (k.grad, kr.grad), (v.grad, vr.grad)):
        assert (got.double() - want).norm() <= 2 ** -6 * want.norm()


def _attention64(q, k, v, layout):
    rep, out = q.shape[1] // k.shape[1], []
    for qs, ql, ps, pl, os_, ol in layout.segs.tolist():
        kk, vv = (torch.cat([x[ps:ps + pl], x[os_:os_ + ol]]).repeat_interleave(rep, 1) for x in (k, v))
        s = torch.einsum("qhd,khd->hqk", q[qs:qs + ql], kk) * q.shape[-1] ** -0.5
        seen = torch.arange(pl + ol, device=q.device)[None] <= pl + ol - ql + torch.arange(ql, device=q.device)[:, None]
        out.append(torch.einsum("hqk,khd->qhd", torch.softmax(s.masked_fill(~seen, float("-inf")), -1), vv))
    return torch.cat(out)


@pytest.mark.parametrize("scale", [0.0, -0.05])
def test_scales_that_are_not_positive(scale):
    """A scale of zero weighs all visible keys alike, a negative one turns the order of the scores: blocks with and without masks,
    forward and backward.  Tolerances as above (bf16 operands o, P and dS)."""
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops.attention import AttnLayout, attention_ref, segment_attention
    segs = np.array([[0, 200, 0, 0, 0, 200], [200, 70, 0, 200, 200, 70], [270, 129, 0, 0, 270, 129]], dtype=np.int32)
    layout = AttnLayout(segs, 399)
    torch.manual_seed(8)
    q, k, v = (_rand((399, h, 128)).requires_grad_() for h in (4, 2, 2))
    d_o = _rand((399, 4, 128))
    o = segment_attention(q, k, v, layout, scale)
    o.backward(d_o)
    _lib.check_status("attention")
    qr, kr, vr = (x.detach().double().requires_grad_() for x in (q, k, v))
    ref = attention_ref(qr, kr, vr, layout, scale)
    ref.backward(d_o.double())
    assert (o.double() - ref.double()).norm() <= 2 ** -7 * ref.double().norm()
    for got, want in ((q.grad, qr.grad), (k.grad, kr.grad), (v.grad, vr.grad)):
        assert (got.double() - want.double()).norm() <= 2 ** -6 * want.double().norm() + 1e-6


@pytest.mark.parametrize("name", ["varlen", "zorro"])
@pytest.mark.parametrize("Hq,Hkv,D,growth", [(4, 2, 128, 1), (3, 1, 128, 40), (4, 2, 64, 12)])
def test_forward_with_the_output_in_tensor_memory(name, Hq, Hkv, D, growth):
    """Rows whose maximum moves late, in some blocks and not in others (``growth`` multiplies some keys), and rows whose first key is the
    largest: as near to 64 bits as with the output in registers, within a hundredth for the luck of the last roundings.  With a scale that
    is not positive both are the same kernel."""
    from arctic_platform_b200.ops import _lib
    from arctic_platform_b200.ops.attention import attention_fwd_cuda, attention_ref
    layout = _layouts()[name]
    T = layout.total_tokens
    torch.manual_seed(D + growth)
    q, k, v = _rand((T, Hq, D)), _rand((T, Hkv, D)), _rand((T, Hkv, D))
    k[40::97] *= growth
    q[::3] *= 2
    ref, ref_lse = attention_ref(q.double(), k.double(), v.double(), layout, D ** -0.5, return_lse=True)
    errs = []
    for tmem_o in (False, True):
        o, lse = attention_fwd_cuda(q, k, v, layout, D ** -0.5, tmem_o=tmem_o)
        _lib.check_status("attn fwd")
        assert torch.isfinite(o.float()).all()
        errs.append(((o.double() - ref).norm() / ref.norm()).item())
        assert torch.allclose(lse, ref_lse.float(), atol=2e-2, rtol=1e-3)
    assert errs[1] <= 1.01 * errs[0], errs
    a, b = (attention_fwd_cuda(q, k, v, layout, -0.01, tmem_o=tmem_o) for tmem_o in (False, True))
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
