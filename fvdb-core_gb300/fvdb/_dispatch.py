"""Which calls may go straight to a kernel: plain CUDA tensors outside tracing, function transforms
and forward-mode differentiation.  Everything else keeps the route through autograd or torch
operations, which carry those mechanisms (or refuse them)."""

from __future__ import annotations

import torch


def plain_cuda(*tensors) -> bool:
    """True when every tensor (None entries skipped) is an ordinary CUDA tensor and nothing records
    or transforms the operations on it."""
    for t in tensors:
        if t is not None and not (t.is_cuda and type(t) in (torch.Tensor, torch.nn.Parameter)):
            return False
    return not (torch.jit.is_tracing() or torch.compiler.is_compiling() or
                torch._C._are_functorch_transforms_active() or torch.autograd.forward_ad._current_level >= 0)


def wants_grad(*tensors) -> bool:
    """Whether autograd would record an operation on these tensors."""
    return torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors)


def has_memory(t: torch.Tensor) -> bool:
    """Whether a kernel can read the tensor: not so for the batched gradients of
    autograd.grad(is_grads_batched=True) and of torch.func.vmap over a backward pass, which look like
    ordinary tensors to the checks above (and reach a backward function with no transform active)."""
    return torch._C._has_storage(t)
