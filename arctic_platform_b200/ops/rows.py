"""Row look-ups whose gradients are added in place (``rows.cu``): the token embedding and the choice of predicting rows.

Forward is PyTorch's row gather.  The backward differs from autograd's: an embedding whose weight has an fp32 gradient buffer
(``grad_f32``) receives its rows there directly, and gathered rows go back through vector reductions instead of scalar ones."""
from __future__ import annotations

import ctypes

import torch

from . import _lib

_ADD = None


def rows_add(src: torch.Tensor, index: torch.Tensor, dst: torch.Tensor) -> None:
    """``dst[index[r]] += src[r]``; ``src [R, H]`` bf16, ``dst [N, H]`` bf16 or fp32, ``index [R]`` int64 within ``[0, N)``."""
    global _ADD
    if _ADD is None:
        c = ctypes
        _ADD = _lib.declare("apb_rows_add", [c.c_void_p, c.c_longlong, c.c_void_p, c.c_void_p, c.c_longlong, c.c_longlong, c.c_int,
                                             c.c_int, c.c_int, c.c_void_p])
    _lib.check(_ADD(_lib.ptr(src), _ld(src), _lib.ptr(index), _lib.ptr(dst), dst.stride(0), dst.shape[0],
                    int(dst.dtype == torch.float32), src.shape[0], src.shape[1], _lib.stream_ptr()), "apb_rows_add")


def _fits(t: torch.Tensor) -> bool:
    """Rows that the kernel addresses: whole vectors of 8 columns at 16-byte boundaries."""
    return t.is_cuda and t.dim() == 2 and t.stride(1) == 1 and t.shape[1] % 8 == 0 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0


def _whole(t: torch.Tensor) -> torch.Tensor:
    """Rows one behind the other from a 16-byte boundary on; a copy where a view is laid out otherwise."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _ld(t: torch.Tensor) -> int:
    """Elements between rows; a lone row may come with any stride."""
    return t.stride(0) if t.shape[0] > 1 else t.shape[1]


class _EmbeddingFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, ids, weight):
        ctx.save_for_backward(ids)
        ctx.weight = weight                 # for its gradient buffer; the values are not needed again
        return torch.nn.functional.embedding(ids, weight)

    @staticmethod
    def backward(ctx, dy):
        (ids,) = ctx.saved_tensors
        rows_add(_whole(dy), ids, ctx.weight.grad_f32)
        return None, None


def embedding(ids: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """``weight[ids]`` for ``ids [T]``.  With an fp32 gradient buffer on a bf16 CUDA weight the gradient is added there and autograd
    sees none, as for every other weight of the model."""
    acc = getattr(weight, "grad_f32", None)
    if (acc is not None and torch.is_grad_enabled() and weight.requires_grad and weight.dtype == torch.bfloat16
            and acc.dtype == torch.float32 and ids.dtype == torch.int64 and ids.dim() == 1 and ids.is_contiguous()
            and _fits(weight) and _fits(acc)):
        return _EmbeddingFn.apply(ids, weight)
    return torch.nn.functional.embedding(ids, weight)


class _GatherFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, index):
        ctx.save_for_backward(index)
        ctx.shape = x.shape
        return x.index_select(0, index)

    @staticmethod
    def backward(ctx, dy):
        (index,) = ctx.saved_tensors
        dx = torch.zeros(ctx.shape, device=dy.device, dtype=dy.dtype)
        rows_add(_whole(dy), index, dx)
        return dx, None


def gather_rows(x: torch.Tensor, index: torch.Tensor) -> torch.Tensor:
    """``x[index]`` for ``x [N, H]``; a row that is taken several times receives the sum of its gradients."""
    if (torch.is_grad_enabled() and x.requires_grad and x.dtype == torch.bfloat16 and _fits(x) and index.dtype == torch.int64
            and index.dim() == 1 and index.is_contiguous()):
        return _GatherFn.apply(x, index)
    return x.index_select(0, index)


# ------------------------------------------------------------------------------------------------- rows to experts and back
_MOE = {}


def _moe(name: str):
    if not _MOE:
        c = ctypes
        vp, i, ll = c.c_void_p, c.c_int, c.c_longlong
        _MOE["place"] = _lib.declare("apb_moe_place", [vp, i, i, i, vp, vp, vp])
        _MOE["spread"] = _lib.declare("apb_moe_spread", [vp, ll, vp, i, i, i, vp, ll, vp])
        _MOE["collect"] = _lib.declare("apb_moe_collect", [vp, ll, vp, vp, i, i, i, vp, ll, vp])
        _MOE["collect_bwd"] = _lib.declare("apb_moe_collect_bwd", [vp, ll, vp, ll, vp, vp, i, i, i, vp, vp, vp])
    return _MOE[name]


def moe_rows_supported(x: torch.Tensor, experts: int) -> bool:
    """What the kernels below take: bf16 rows of whole 16-byte vectors on the GPU, at most 512 experts."""
    return x.is_cuda and x.dtype == torch.bfloat16 and x.shape[1] % 8 == 0 and experts <= 512


def moe_place(chosen: torch.Tensor, experts: int, pad: int = 1):
    """Expert-major places of the routed pairs ``chosen [T, k]`` (int64): ``(counts [experts], place [T, k])``, both int32 on the GPU.
    Expert ``e`` owns rows from ``sum(roundup(counts[:e], pad))`` on, its pairs in the order of the tokens."""
    chosen = chosen.contiguous()
    counts = torch.empty(experts, device=chosen.device, dtype=torch.int32)
    place = torch.empty(chosen.shape, device=chosen.device, dtype=torch.int32)
    _lib.check(_moe("place")(_lib.ptr(chosen), chosen.numel(), experts, pad, _lib.ptr(counts), _lib.ptr(place), _lib.stream_ptr()),
               "apb_moe_place")
    return counts, place


def _spread(x, place, rows: int, pad_rows: bool):
    x = _whole(x)
    out = (torch.zeros if pad_rows else torch.empty)((rows, x.shape[1]), device=x.device, dtype=x.dtype)
    _lib.check(_moe("spread")(_lib.ptr(x), _ld(x), _lib.ptr(place), place.shape[0], place.shape[1], x.shape[1], _lib.ptr(out),
                              out.stride(0), _lib.stream_ptr()), "apb_moe_spread")
    return out


def _collect(y, place, weight):
    y = _whole(y)
    out = torch.empty((place.shape[0], y.shape[1]), device=y.device, dtype=y.dtype)
    _lib.check(_moe("collect")(_lib.ptr(y), _ld(y), _lib.ptr(place), _lib.ptr(weight), place.shape[0], place.shape[1], y.shape[1],
                               _lib.ptr(out), out.stride(0), _lib.stream_ptr()), "apb_moe_collect")
    return out


class _SpreadFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, place, rows, pad_rows):
        ctx.save_for_backward(place)
        return _spread(x, place, rows, pad_rows)

    @staticmethod
    def backward(ctx, d):
        (place,) = ctx.saved_tensors
        return _collect(d, place, None), None, None, None


class _CollectFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, y, place, weight, pad_rows):
        y, weight = _whole(y), weight.contiguous()
        ctx.save_for_backward(y, place, weight)
        ctx.pad_rows = pad_rows
        return _collect(y, place, weight)

    @staticmethod
    def backward(ctx, d):
        y, place, weight = ctx.saved_tensors
        d = _whole(d)
        dy = (torch.zeros_like if ctx.pad_rows else torch.empty_like)(y)
        dw = torch.empty_like(weight)
        _lib.check(_moe("collect_bwd")(_lib.ptr(d), _ld(d), _lib.ptr(y), _ld(y), _lib.ptr(place), _lib.ptr(weight),
                                       place.shape[0], place.shape[1], y.shape[1], _lib.ptr(dy), _lib.ptr(dw), _lib.stream_ptr()),
                   "apb_moe_collect_bwd")
        return dy, None, dw, None


def moe_spread(x: torch.Tensor, place: torch.Tensor, rows: int, pad_rows: bool = False) -> torch.Tensor:
    """``[rows, H]`` with row ``place[t, j]`` equal to ``x[t]``; the rows that no pair has are zero with ``pad_rows`` (and are not
    written without)."""
    return _SpreadFn.apply(x, place, rows, pad_rows)


def moe_collect(y: torch.Tensor, place: torch.Tensor, weight: torch.Tensor, pad_rows: bool = False) -> torch.Tensor:
    """``out[t] = sum_j weight[t, j] y[place[t, j]]``: bf16 products, summed in fp32; gradients in fp32.  ``pad_rows``: ``y`` has rows that no pair has, whose
    gradient is zero."""
    return _CollectFn.apply(y, place, weight.float(), pad_rows)
