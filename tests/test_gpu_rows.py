"""Gradients of row look-ups (rows.cu) against sums in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,table", [(1, 8, 3), (257, 72, 5), (1000, 2560, 40000)])
def test_rows_are_added_where_they_were_taken(rows, cols, table):
    """Repeated rows included.  fp32: sums of at most `rows` bf16 values, 2^-24 each; bf16: one rounding of 2^-9 per addition."""
    from arctic_platform_b200.ops import rows as ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    index = torch.randint(0, table, (rows,), device="cuda", generator=g)
    dy = torch.randn(rows, cols, device="cuda", generator=g).bfloat16()
    start = torch.randn(table, cols, device="cuda", generator=g)
    most = int(torch.bincount(index).max())
    size = torch.zeros(table, cols, device="cuda", dtype=torch.float64).index_add_(0, index, dy.double().abs())
    weight = torch.nn.Parameter(torch.randn(table, cols, device="cuda", generator=g).bfloat16())
    weight.grad_f32 = start.clone()
    y = ops.embedding(index, weight)
    assert torch.equal(y, weight.detach()[index])
    y.backward(dy)
    assert weight.grad is None
    want = start.double().index_add(0, index, dy.double())
    assert ((weight.grad_f32 - want).abs() <= 2 ** -23 * most * (size + start.abs())).all()
    x = torch.randn(table, cols, device="cuda", generator=g).bfloat16().requires_grad_()
    ops.gather_rows(x, index).backward(dy)
    want = torch.zeros(table, cols, device="cuda", dtype=torch.float64).index_add_(0, index, dy.double())
    assert ((x.grad.double() - want).abs() <= 2 ** -8 * most * size).all()


def test_embedding_without_a_gradient_buffer_is_torchs():
    from arctic_platform_b200.ops import rows as ops
    weight = torch.nn.Parameter(torch.randn(50, 64, device="cuda").bfloat16())
    index = torch.randint(0, 50, (20,), device="cuda")
    ops.embedding(index, weight).float().sum().backward()
    assert weight.grad is not None and weight.grad.float().sum() == 20 * 64


@pytest.mark.parametrize("tokens,k,experts,cols,pad", [(1, 1, 1, 8, 1), (3, 8, 128, 72, 64), (1025, 2, 5, 264, 64), (700, 8, 512, 2048, 1)])
def test_rows_to_experts_and_back(tokens, k, experts, cols, pad):
    """Places are those of a stable sort by expert; weighted sums and all gradients against 64 bits: bf16 roundings of a weight, of a
    weighted row and of a result (8 significant bits: 2^-8 of a term each, three of them below 2^-6), the weights' gradients are fp32 sums of `cols` products."""
    from arctic_platform_b200.ops import rows as ops
    g = torch.Generator(device="cuda").manual_seed(tokens)
    chosen = torch.stack([torch.randperm(experts, device="cuda", generator=g)[:k] for _ in range(tokens)])
    counts, place = ops.moe_place(chosen, experts, pad)
    flat = chosen.reshape(-1)
    want = torch.bincount(flat, minlength=experts)
    assert torch.equal(counts.long(), want)
    start = torch.cat([want.new_zeros(1), ((want + pad - 1) // pad * pad).cumsum(0)])
    order = torch.argsort(flat, stable=True)
    rank = torch.empty_like(flat)
    rank[order] = torch.arange(flat.numel(), device="cuda") - (want.cumsum(0) - want)[flat[order]]
    assert torch.equal(place.long().reshape(-1), start[flat] + rank)
    n = int(start[-1])
    x = torch.randn(tokens, cols, device="cuda", generator=g).bfloat16().requires_grad_()
    w = torch.rand(tokens, k, device="cuda", generator=g).requires_grad_()
    y = ops.moe_spread(x, place, n, pad > 1)
    assert torch.equal(y[place.long()], x.detach()[:, None].expand(-1, k, -1))
    if pad > 1:
        assert int((y != 0).any(1).sum()) <= flat.numel()
    z = (y.float() * 1.5).bfloat16().detach().requires_grad_()
    out = ops.moe_collect(z, place, w, pad > 1)
    d = torch.randn(tokens, cols, device="cuda", generator=g).bfloat16()
    out.backward(d)
    dy = torch.randn(n, cols, device="cuda", generator=g).bfloat16()
    y.backward(dy)
    zr, wr, at = z.detach().double(), w.detach().double(), place.long()
    near = lambda got, ref, size: ((got.double() - ref).abs() <= 2 ** -6 * size + 1e-30).all()
    terms = wr[..., None] * zr[at]
    assert near(out, terms.sum(1), terms.abs().sum(1))
    dz = torch.zeros(n, cols, device="cuda", dtype=torch.float64)
    dz[at.reshape(-1)] = (wr[..., None] * d.double()[:, None]).reshape(-1, cols)
    assert near(z.grad, dz, dz.abs())
    dw = d.double()[:, None] * zr[at]
    assert ((w.grad - dw.sum(-1)).abs() <= cols * 2 ** -23 * dw.abs().sum(-1)).all()
    assert near(x.grad, dy.double()[at].sum(1), dy.double()[at].abs().sum(1))


def test_rows_that_begin_anywhere():
    """Views that start off a 16-byte boundary, a lone row with an odd stride: the same sums as aligned copies of them."""
    from arctic_platform_b200.ops import rows as ops
    g = torch.Generator(device="cuda").manual_seed(6)
    off = lambda r, c: torch.randn(r * c + 1, device="cuda", generator=g).bfloat16()[1:].view(r, c)
    x, d, index = off(40, 64), off(25, 64), torch.randperm(40, device="cuda", generator=g)[:25]
    base = torch.randn(40, 64, device="cuda", generator=g).bfloat16().requires_grad_()
    ops.gather_rows(base, index).backward(d)
    assert torch.equal(base.grad[index], d)
    weight = torch.nn.Parameter(torch.randn(40, 64, device="cuda", generator=g).bfloat16())
    weight.grad_f32 = torch.zeros(40, 64, device="cuda")
    ops.embedding(index, weight).backward(d)
    assert torch.equal(weight.grad_f32[index], d.float())
    chosen = torch.randint(0, 5, (40, 1), device="cuda", generator=g)
    lone = torch.randn(1, 67, device="cuda", generator=g).bfloat16()[:, :64]
    for src, c in ((x, chosen), (lone, chosen[:1])):
        _, place = ops.moe_place(c, 5)
        y = ops.moe_spread(src, place, len(c))
        assert torch.equal(y[place[:, 0].long()], src)
        w = torch.ones(len(c), 1, device="cuda")
        z = off(len(c), 64)
        z.copy_(y)
        z.requires_grad_()
        out = ops.moe_collect(z, place, w)
        assert torch.equal(out, src)
        out.backward(x[:len(c)])
        assert torch.equal(z.grad[place[:, 0].long()], x[:len(c)])
