"""The torch.autograd.Function of one sparse convolution.

Forward and backward bodies run in the C++ extension (conv_forward / conv_backward), which
launches the hand-written kernels through the C ABI: forward = fused gather-GEMM over the
kernel map; dgrad = the same contraction over the transposed map with W^T; wgrad = the
per-offset reduction with an FP64 cross-CTA sum.  Semantics follow
src/fvdb/detail/autograd/SparseConvolutionKernelMap.cpp:18-191 (weight permutes, checks,
gradient layout).
"""

from __future__ import annotations

import torch

from . import _lib
from ._dispatch import has_memory, plain_cuda, wants_grad


class SparseConvFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, features: torch.Tensor, weights: torch.Tensor, pack_impl, transposed: bool, bias=None,
                relu: bool = False, scale=None):
        C = _lib.load()
        # a data gradient to come reuses the kernel map (and may share its row order)
        ctx.announced = ctx.needs_input_grad[0]
        y, wkio = C.conv_forward(features, weights, pack_impl, transposed, bias, relu, scale, ctx.announced)
        ctx.scaled = scale is not None
        if relu:
            ctx.save_for_backward(features, wkio, y)
        else:
            ctx.save_for_backward(features, wkio)
        ctx.pack_impl = pack_impl
        ctx.transposed = transposed
        ctx.relu = relu
        ctx.bias_dtype = bias.dtype if bias is not None else None
        return y

    @staticmethod
    def backward(ctx, grad_out: torch.Tensor):
        C = _lib.load()
        features, wkio = ctx.saved_tensors[:2]
        need_dx, need_dw, need_db = ctx.needs_input_grad[0], ctx.needs_input_grad[1], ctx.needs_input_grad[4]
        if grad_out is None or not (need_dx or need_dw or need_db):
            return None, None, None, None, None, None, None
        if ctx.scaled:
            raise RuntimeError("a convolution with a folded batch norm (out_scale) is inference-only")
        # fused ReLU: the gradient passes where the output is positive (torch.relu's rule); bias
        # gradient = column sum of dy, accumulated in at least FP32 (FP64 stays FP64)
        y = ctx.saved_tensors[2] if ctx.relu else None
        dx = dw = db = None
        if torch.is_grad_enabled() or not has_memory(grad_out):
            # create_graph or batched gradients: operations that record their own gradient and batch
            if ctx.relu:
                grad_out = grad_out * (y > 0)
            if need_db:
                db = grad_out.sum(0, dtype=torch.promote_types(grad_out.dtype, torch.float32))
        else:
            grad_out, db = C.bias_relu_backward(grad_out, y, need_db)
        if need_dx or need_dw:
            dx, dw = C.conv_backward(grad_out, features, wkio, ctx.pack_impl, ctx.transposed, need_dx, need_dw,
                                     ctx.announced)
        if need_db:
            db = db.to(ctx.bias_dtype)
        return (dx if need_dx else None), (dw if need_dw else None), None, None, db, None, None


def sparse_conv(features: torch.Tensor, weights: torch.Tensor, pack_impl, transposed: bool, bias=None,
                relu: bool = False, scale=None) -> torch.Tensor:
    """One sparse convolution with autograd; `bias` ([C_out], optional) is added, and with `relu`
    the output clamped at zero, in the contraction's epilogue on the tensor-core path (one pass
    over the output instead of two or three).  `scale` ([C_out], optional, inference only)
    multiplies the contraction before the bias: an eval-mode batch norm folded into the layer."""
    if not wants_grad(features, weights, bias, scale) and plain_cuda(features, weights, bias, scale):
        return _lib.load().conv_forward(features, weights, pack_impl, transposed, bias, relu, scale)[0]
    return SparseConvFunction.apply(features, weights, pack_impl, transposed, bias, relu, scale)
