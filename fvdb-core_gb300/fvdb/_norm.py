"""Group normalisation of jagged features (fvdb.nn.GroupNorm): the CUDA kernels of csrc/norm.cu
behind a torch.autograd.Function, and the same map composed of torch operations."""

from __future__ import annotations

import torch

from . import _lib
from ._dispatch import has_memory, plain_cuda

_DTYPES = (torch.float32, torch.float64, torch.bfloat16, torch.float16)


def _acc(dtype: torch.dtype) -> torch.dtype:
    return torch.float64 if dtype == torch.float64 else torch.float32


def group_norm_composed(x: torch.Tensor, jidx: torch.Tensor, num_grids: int, groups: int, eps: float, weight=None,
                        bias=None) -> torch.Tensor:
    """Normalises each (grid, group) of x [n, C] with differentiable torch operations: segment
    sums keyed by the rows' grid index (int64 jidx), the variance about the mean, FP32 or wider."""
    n, c = x.shape
    acc = _acc(x.dtype)
    xg = x.to(acc).reshape(n, groups, c // groups)
    counts = torch.bincount(jidx, minlength=num_grids).to(acc) * (c // groups)
    denom = counts.clamp(min=1)[:, None]
    mean = torch.zeros(num_grids, groups, dtype=acc, device=x.device).index_add_(0, jidx, xg.sum(2)) / denom
    d = xg - mean[jidx][:, :, None]
    var = torch.zeros(num_grids, groups, dtype=acc, device=x.device).index_add_(0, jidx, (d * d).sum(2)) / denom
    y = (d * torch.rsqrt(var + eps)[jidx][:, :, None]).reshape(n, c)
    if weight is not None:
        y = y * weight.to(acc) + bias.to(acc)
    return y.to(x.dtype)


def group_norm_kernel_takes(x: torch.Tensor, weight, bias) -> bool:
    """Whether the kernels serve this call: plain CUDA tensors outside function transforms,
    forward-mode differentiation and tracing (where composed operations carry the derivative)."""
    params = [p for p in (weight, bias) if p is not None]
    if not plain_cuda(x, weight, bias) or x.dtype not in _DTYPES or x.shape[1] > 65535:
        return False
    return (weight is None) == (bias is None) and all(p.is_floating_point() and p.device == x.device for p in params)


class GroupNormFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias, joffsets, groups: int, eps: float):
        acc = _acc(x.dtype)
        w = None if weight is None else weight.to(acc).contiguous()
        b = None if bias is None else bias.to(acc).contiguous()
        y, mean, rstd = _lib.load().group_norm_forward(x, joffsets, groups, w, b, eps)
        ctx.save_for_backward(x, weight, bias, mean, rstd)
        # the grid's own offsets, which carry no gradient; a grid built in inference mode has an
        # inference tensor there, which cannot be saved
        ctx.joffsets, ctx.groups, ctx.eps = joffsets, groups, eps
        return y

    @staticmethod
    def backward(ctx, dy):
        x, weight, bias, mean, rstd = ctx.saved_tensors
        joffsets = ctx.joffsets
        create_graph = torch.is_grad_enabled()
        if create_graph or not has_memory(dy):  # a gradient to differentiate again, or one per batch entry
            need = [t for t, n in zip((x, weight, bias), ctx.needs_input_grad) if n]
            counts = joffsets[1:] - joffsets[:-1]
            jidx = torch.repeat_interleave(torch.arange(counts.numel(), device=x.device), counts)
            with torch.enable_grad():
                y = group_norm_composed(x, jidx, counts.numel(), ctx.groups, ctx.eps, weight, bias)
            g = iter(torch.autograd.grad(y, need, dy, create_graph=create_graph))
            return (*(next(g) if n else None for n in ctx.needs_input_grad[:3]), None, None, None)
        w = None if weight is None else weight.to(mean.dtype).contiguous()
        dx, dw, db = _lib.load().group_norm_backward(dy, x, joffsets, ctx.groups, w, mean, rstd, ctx.needs_input_grad[0])
        return (dx if ctx.needs_input_grad[0] else None, dw.to(weight.dtype) if ctx.needs_input_grad[1] else None,
                db.to(bias.dtype) if ctx.needs_input_grad[2] else None, None, None, None)
