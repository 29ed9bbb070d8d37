"""Training-mode BatchNorm of feature rows with the residual addition and the ReLU that follow it, two native launches
per direction (``csrc/batch_norm.cu``).  An addition to the reference, whose blocks run ``nn.BatchNorm1d``, the addition
and ``nn.ReLU`` one after the other (examples/mink_unet.py:36-47, 129-141); values are rounded where those round."""
from __future__ import annotations

import functools
import struct
from typing import Optional

import torch
import torch.nn as nn
import torch.nn.modules.module as _module
from torch import Tensor
from torch.autograd import forward_ad

from ..._native import check, dtype_code, lib, ptr, query_bytes, stream_ptr

_DTYPES = (torch.float32, torch.float16, torch.bfloat16)
_counters: dict = {}


def _counter(device: torch.device, stream: int) -> Tensor:
    """The block counter of the reductions: zero between launches of one stream.  A launch that is being captured gets one
    of its own, zeroed by the graph: graphs replay in any order and on any stream, and the capture's memory is theirs."""
    if torch.cuda.is_current_stream_capturing():
        return torch.zeros(1, dtype=torch.int32, device=device)
    key = (device.index, stream)
    hit = _counters.get(key)
    if hit is None:
        if len(_counters) >= 256:  # streams come and go; the memory of a counter returns to its own stream
            _counters.pop(next(iter(_counters)), None)
        hit = _counters[key] = torch.zeros(1, dtype=torch.int32, device=device)
    return hit


def reverse_mode_only() -> bool:
    """Whether neither forward-mode differentiation nor a function transform is on: autograd functions take part in plain
    backward passes only, torch's own operations in all of them."""
    return forward_ad._current_level < 0 and not torch._C._are_functorch_transforms_active()


def bare(*modules: nn.Module) -> bool:
    """Whether calling these modules runs their class's ``forward`` and nothing else: no hooks, on them or on all modules,
    and no ``forward`` of the instance's own."""
    if (_module._global_forward_hooks or _module._global_forward_pre_hooks or _module._global_backward_hooks
            or _module._global_backward_pre_hooks):
        return False
    for m in modules:
        d = m.__dict__  # (a training step asks this of every block: no attribute protocol)
        if (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"]
                or "forward" in d):
            return False
    return True


def can_fuse(bn: nn.Module, x: Tensor) -> bool:
    """Whether ``batch_norm_act`` computes what ``bn(x)`` would (training mode, running statistics kept)."""
    return (x.is_cuda and x.dim() == 2 and x.is_contiguous() and x.data_ptr() % 16 == 0
            and fusable(bn, x.shape[0], x.shape[1], x.dtype, x.device))


def fusable(bn: nn.Module, n: int, c: int, dtype: torch.dtype, device: torch.device) -> bool:
    """:func:`can_fuse` for contiguous rows that do not exist yet."""
    if type(bn) is not nn.BatchNorm1d or not bn.training or not bn.track_running_stats or bn.momentum is None:
        return False
    if not bare(bn) or not reverse_mode_only():
        return False
    if (device.type != "cuda" or dtype not in _DTYPES or n < 2 or c != bn.num_features or c > 1024
            or c % (4 if dtype == torch.float32 else 8)):
        return False
    buffers, params = bn._buffers, bn._parameters
    tracked = buffers["num_batches_tracked"]
    if tracked is None or tracked.device != device or tracked.dtype != torch.int64:
        return False
    for t in (buffers["running_mean"], buffers["running_var"], params["weight"], params["bias"]):
        if t is not None and (t.dtype != torch.float32 or t.device != device or not t.is_contiguous() or t.numel() != c):
            return False
    return buffers["running_mean"] is not None


def train_forward(x: Tensor, gamma, beta, residual, bn: nn.BatchNorm1d, relu: bool):
    """(the rows, mean and 1 / std) of one training step; the running statistics advance."""
    n, c = x.shape
    dev, dc, st = x.device, dtype_code(x.dtype), stream_ptr(x.device)
    y = torch.empty_like(x)
    saved = torch.empty((2, c), dtype=torch.float32, device=dev)
    ws = torch.empty(query_bytes("wcn_batch_norm_workspace_bytes", n, c, dc), dtype=torch.uint8, device=dev)
    at, counter = saved.data_ptr(), _counter(dev, st)
    check(lib().wcn_batch_norm_train(ptr(x), n, c, dc, ptr(gamma), ptr(beta), _bits(bn.eps), _bits(bn.momentum),
                                     ptr(bn.running_mean), ptr(bn.running_var), ptr(bn.num_batches_tracked), ptr(residual),
                                     int(relu), ptr(y), at, at + 4 * c, ptr(ws), ptr(counter), st),
          "wcn_batch_norm_train")
    torch.autograd.graph.increment_version([bn.running_mean, bn.running_var, bn.num_batches_tracked])
    return y, saved


def _aligned_rows(t: Optional[Tensor]) -> Optional[Tensor]:
    """``t`` contiguous on a 16-byte boundary (a gradient may be a view into a flat buffer, a saved tensor whatever a
    saved-tensor hook made of it)."""
    if t is not None:
        t = t.contiguous()
        if t.data_ptr() % 16:
            t = t.clone()
    return t


def train_backward(dy: Tensor, x: Tensor, gamma, beta, saved: Tensor, y: Optional[Tensor], relu: bool, need_x: bool,
                   need_res: bool):
    """(dx, (d beta, d gamma), d residual); ``y`` only with a residual under a ReLU."""
    x, dy, y = _aligned_rows(x), _aligned_rows(dy), _aligned_rows(y)
    n, c = x.shape
    dev, dc, st = x.device, dtype_code(x.dtype), stream_ptr(x.device)
    want_res = need_res and relu
    dx = torch.empty_like(x) if need_x or want_res else None
    dres = torch.empty_like(x) if want_res else None
    sums = torch.empty((2, c), dtype=torch.float32, device=dev)
    ws = torch.empty(query_bytes("wcn_batch_norm_workspace_bytes", n, c, dc), dtype=torch.uint8, device=dev)
    at, counter = saved.data_ptr(), _counter(dev, st)
    check(lib().wcn_batch_norm_backward(ptr(x), ptr(dy), ptr(y), n, c, dc, ptr(gamma), ptr(beta), at, at + 4 * c, int(relu),
                                        ptr(dx), ptr(dres), ptr(sums), ptr(ws), ptr(counter), st),
          "wcn_batch_norm_backward")
    return dx, sums, (dres if relu else dy) if need_res else None


def formula(x: Tensor, gamma, beta, residual, eps: float, relu: bool) -> Tensor:
    """The same through torch, for a graph of the gradient (running statistics untouched)."""
    z = torch.nn.functional.batch_norm(x, None, None, gamma, beta, True, 0.0, eps)
    z = z if residual is None else z + residual
    return torch.relu(z) if relu else z


class _BatchNormAct(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x: Tensor, gamma: Optional[Tensor], beta: Optional[Tensor], residual: Optional[Tensor], bn, relu: bool):
        y, saved = train_forward(x, gamma, beta, residual, bn, relu)
        ctx.relu, ctx.eps = relu, bn.eps
        ctx.save_for_backward(x, gamma, beta, residual, saved, y if relu and residual is not None else None)
        return y

    @staticmethod
    def backward(ctx, dy: Tensor):
        x, gamma, beta, residual, saved, y = ctx.saved_tensors
        if torch.is_grad_enabled():  # a graph of the gradient is wanted: the same formulas through torch
            z = formula(x, gamma, beta, residual, ctx.eps, ctx.relu)
            wanted = [t for t, need in zip((x, gamma, beta, residual), ctx.needs_input_grad) if need]
            got = iter(torch.autograd.grad(z, wanted, dy, create_graph=True))
            return tuple(next(got) if need else None for need in ctx.needs_input_grad[:4]) + (None, None)
        need_x, need_g, need_b, need_res = ctx.needs_input_grad[:4]
        dx, sums, dres = train_backward(dy, x, gamma, beta, saved, y, ctx.relu, need_x, need_res)
        return dx if need_x else None, sums[1] if need_g else None, sums[0] if need_b else None, dres, None, None


@functools.lru_cache(maxsize=64)
def _bits(value: float) -> int:
    """A float argument as the 32 bits the C function reinterprets (calls pass integers only)."""
    return struct.unpack("<I", struct.pack("<f", value))[0]


def aligned_residual(residual: Optional[Tensor], shape, dtype: torch.dtype) -> Optional[Tensor]:
    if residual is not None:
        assert residual.shape == shape, f"residual {tuple(residual.shape)} != {tuple(shape)}"
        residual = _aligned_rows(residual.to(dtype))
    return residual


def batch_norm_act(x: Tensor, bn: nn.BatchNorm1d, relu: bool = False, residual: Optional[Tensor] = None) -> Tensor:
    """``relu(bn(x) + residual)`` of a training step (see :func:`can_fuse`)."""
    residual = aligned_residual(residual, x.shape, x.dtype)
    return _BatchNormAct.apply(x, bn.weight, bn.bias, residual, bn, relu)
