"""Row reductions over a kernel map (warpconvnet/ops/reductions.py:13-70).

The reference reduces a CSR of gathered rows with ``torch_scatter.segment_csr``; here the
reduction runs straight over the dense neighbour table in one native launch
(``wcn_row_reduce``): output row m reduces the input rows ``nbr[k][m] >= 0``.  The reductions
are differentiable like the reference's (its ``segment_csr`` is an autograd op): sum and mean
send the output gradient back through the transposed table with the same kernel, max and min
send it to the row that attained the extremum.
"""
from __future__ import annotations

from enum import Enum
from typing import Union

import torch
from torch import Tensor

from .._native import check, device_status, dtype_code, lib, ptr, require_cuda, stream_ptr
from ..geometry.coords.search.search_results import IntSearchResult


class REDUCTIONS(Enum):
    MIN = "min"
    MAX = "max"
    MEAN = "mean"
    SUM = "sum"
    MUL = "mul"
    VAR = "var"
    STD = "std"
    RANDOM = "random"


_NATIVE_OP = {REDUCTIONS.MIN: 0, REDUCTIONS.MAX: 1, REDUCTIONS.SUM: 2, REDUCTIONS.MEAN: 3, REDUCTIONS.MUL: 4}
_EXTREMA = (_NATIVE_OP[REDUCTIONS.MIN], _NATIVE_OP[REDUCTIONS.MAX])


def _native_reduce(features: Tensor, nbr: Tensor, op: int) -> Tensor:
    K, M = nbr.shape
    dev = features.device
    out = torch.empty((M, features.shape[1]), dtype=features.dtype, device=dev)
    check(lib().wcn_row_reduce(ptr(features), features.shape[0], ptr(nbr), M, K, features.shape[1],
                               dtype_code(features.dtype), op, ptr(out), ptr(device_status(dev)), stream_ptr(dev)),
          "wcn_row_reduce")
    return out


class _RowReduce(torch.autograd.Function):
    """``wcn_row_reduce`` with a backward pass: sum and mean send the output gradient (over the number of
    neighbours) to every neighbour, max and min send it, per channel, to the first neighbour (ascending
    offset) that attained the result, as ``segment_csr``'s arg-extremum does.  The forward kernel leaves
    that offset (or the counts) behind; mul has no backward here."""

    @staticmethod
    def forward(ctx, features: Tensor, kernel_map: IntSearchResult, num_out: int, op: int) -> Tensor:
        x = features.contiguous()
        nbr = kernel_map.neighbor_table(num_out)
        K, M, C, dev = nbr.shape[0], num_out, x.shape[1], x.device
        out = torch.empty((M, C), dtype=x.dtype, device=dev)
        arg = count = None
        if op in _EXTREMA:
            arg = torch.empty((M, C), dtype=torch.uint8 if K <= 255 else torch.int16, device=dev)
        elif op == _NATIVE_OP[REDUCTIONS.MEAN]:
            count = torch.empty(M, dtype=torch.float32, device=dev)
        check(lib().wcn_row_reduce_train(ptr(x), x.shape[0], ptr(nbr), M, K, C, dtype_code(x.dtype), op, ptr(out),
                                         ptr(arg), arg.element_size() if arg is not None else 0, ptr(count),
                                         ptr(device_status(dev)), stream_ptr(dev)), "wcn_row_reduce_train")
        ctx.kernel_map, ctx.num_in, ctx.op = kernel_map, x.shape[0], op
        ctx.save_for_backward(arg, count)
        return out

    @staticmethod
    def backward(ctx, grad_out: Tensor):
        if ctx.op == _NATIVE_OP[REDUCTIONS.MUL]:
            raise NotImplementedError("the 'mul' reduction has no backward pass")
        arg, count = ctx.saved_tensors
        return _RowReduceBackward.apply(grad_out, ctx.kernel_map, ctx.num_in, arg, count), None, None, None


def _attained(nbr: Tensor, arg: Tensor):
    """(input row, whether there is one) per element ``[M, C]`` of the outputs, from the offset that attained its extremum."""
    at = arg.long() & (255 if arg.dtype == torch.uint8 else 65535)
    rows = nbr.t().gather(1, at.clamp(max=nbr.shape[0] - 1)).long()
    return rows.clamp(min=0), (at < nbr.shape[0]) & (rows >= 0)


class _RowReduceBackward(torch.autograd.Function):
    """The gradient of :class:`_RowReduce`, linear in the output gradient and differentiable with respect to it."""

    @staticmethod
    def forward(ctx, grad_out: Tensor, kernel_map: IntSearchResult, num_in: int, arg, count) -> Tensor:
        g = grad_out.contiguous()
        M, C, dev = g.shape[0], g.shape[1], g.device
        ctx.kernel_map, ctx.num_out = kernel_map, M
        ctx.save_for_backward(arg, count)
        facts = getattr(kernel_map, "_output_rows", {})
        if arg is not None and not (facts.get("distinct") or facts.get("unique")):
            # Output rows with the same coordinates (or a caller's own map): an input row may have several at one offset,
            # of which a transposed table holds one.  Added up where the extremum was instead.
            rows, live = _attained(kernel_map.neighbor_table(M), arg)
            gx = torch.zeros((num_in, C), dtype=torch.float32, device=dev)
            return gx.scatter_add_(0, rows, torch.where(live, g.float(), 0.0)).to(g.dtype)
        nbr_t = kernel_map.swapped(num_in=num_in).neighbor_table(num_in)
        gx = torch.empty((num_in, C), dtype=g.dtype, device=dev)
        check(lib().wcn_row_reduce_backward(ptr(g), M, ptr(nbr_t), num_in, nbr_t.shape[0], C, dtype_code(g.dtype),
                                            ptr(arg), arg.element_size() if arg is not None else 0, ptr(count),
                                            ptr(gx), ptr(device_status(dev)), stream_ptr(dev)),
              "wcn_row_reduce_backward")
        return gx

    @staticmethod
    def backward(ctx, gg: Tensor):
        arg, count = ctx.saved_tensors
        nbr = ctx.kernel_map.neighbor_table(ctx.num_out)
        if arg is None:
            total = _native_reduce(gg.contiguous(), nbr, _NATIVE_OP[REDUCTIONS.SUM])
            return (total if count is None else (total / count.unsqueeze(1)).to(gg.dtype)), None, None, None, None
        rows, live = _attained(nbr, arg)
        return torch.where(live, gg.gather(0, rows), torch.zeros((), dtype=gg.dtype, device=gg.device)), None, None, None, None


def neighbor_reduction(features: Tensor, kernel_map: IntSearchResult, num_out: int,
                       reduction: Union[REDUCTIONS, str], eps: float = 1e-6) -> Tensor:
    """``out[m] = reduction over the neighbours of output row m`` (rows without a neighbour: 0).
    ``var`` / ``std`` follow the reference: mean of squares minus squared mean (+ eps under the root);
    ``random`` picks one neighbour per row uniformly.  Differentiable with respect to ``features``."""
    if isinstance(reduction, str):
        reduction = REDUCTIONS(reduction)
    require_cuda(features, "features")
    if features.dtype not in (torch.float32, torch.float16, torch.bfloat16):
        raise ValueError(f"unsupported feature dtype {features.dtype}")
    tracked = torch.is_grad_enabled() and features.requires_grad

    def native(x: Tensor, red: REDUCTIONS) -> Tensor:
        if tracked:
            return _RowReduce.apply(x, kernel_map, num_out, _NATIVE_OP[red])
        return _native_reduce(x.contiguous(), kernel_map.neighbor_table(num_out), _NATIVE_OP[red])

    if reduction in _NATIVE_OP:
        return native(features, reduction)
    if reduction in (REDUCTIONS.VAR, REDUCTIONS.STD):
        mean = native(features, REDUCTIONS.MEAN)
        var = native(features * features, REDUCTIONS.MEAN) - mean * mean
        return var if reduction == REDUCTIONS.VAR else torch.sqrt(var + eps)
    if reduction == REDUCTIONS.RANDOM:
        with torch.no_grad():
            nbr = kernel_map.neighbor_table(num_out)
            present = nbr >= 0
            count = present.sum(0)
            pick = (torch.rand(num_out, device=features.device) * count).floor().long().clamp_(min=0)
            rank = present.long().cumsum(0) - 1                      # rank of each present neighbour in its column
            chosen = (present & (rank == pick.unsqueeze(0))).float().argmax(0)
            idx = nbr.gather(0, chosen.unsqueeze(0)).squeeze(0).long().clamp_(min=0)
        out = features[idx]                                          # differentiable gather
        return out * (count > 0).to(out.dtype).unsqueeze(1)
    raise ValueError(f"Invalid reduction: {reduction}")
