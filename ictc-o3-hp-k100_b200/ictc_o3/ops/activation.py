"""Scaled SiLU with fused first and second derivatives (reference: modes 0 to 2 of
ictc_o3/backends/k100/hip_activation.py:27-38)."""
from __future__ import annotations

import torch

from .. import _lib


def runs_eagerly(x) -> bool:
    """A plain float32 CUDA tensor in eager reverse-mode differentiation.  Everything else stays with the framework's operators:
    traced calls and dispatch modes, forward mode, tensors without a storage of their own (a batched backward pass is not
    announced by any mode) and lazily negated ones."""
    return (type(x) in (torch.Tensor, torch.nn.Parameter) and x.is_cuda and x.dtype == torch.float32
            and x.layout == torch.strided and torch._C._has_storage(x) and not x.is_neg()
            and not torch._C._are_functorch_transforms_active() and torch._C._len_torch_dispatch_stack() == 0
            and torch.autograd.forward_ad._current_level < 0 and not torch.compiler.is_compiling()
            and not torch.jit.is_tracing() and not torch.is_autocast_enabled("cuda"))


def kernel_takes(x) -> bool:
    return runs_eagerly(x) and x.is_contiguous()


def kernels_take(*tensors):
    """The tensors made contiguous, or None when one of them is not for the kernels (looked at again in every backward pass:
    what arrives there, cotangents and what saved-tensor hooks hand back, need not look like the forward's operands)."""
    return [t.contiguous() for t in tensors] if all(runs_eagerly(t) for t in tensors) else None


def _first(x, scale):
    s = torch.sigmoid(x)
    return scale * s * (1 + x * (1 - s))


def _launch(name, x, scale, *buffers):
    with _lib.on_device(x.device):
        _lib.check(getattr(_lib.load(), name)(x.numel(), scale, _lib.ptr(x), *[_lib.ptr(b) for b in buffers],
                                              _lib.stream(x.device)), name)


class _Silu(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, scale):
        ctx.scale = scale
        ctx.save_for_backward(x)
        y = torch.empty_like(x)
        _launch("ictc_silu_forward", x, scale, y)
        return y

    @staticmethod
    def backward(ctx, grad):
        (x,) = ctx.saved_tensors
        rows = kernels_take(x, grad)
        return _SiluGrad.apply(*rows, ctx.scale) if rows else grad * _first(x, ctx.scale), None


class _SiluGrad(torch.autograd.Function):
    """grad * scale * silu'(x) for a contiguous grad; differentiable in x and grad."""

    @staticmethod
    def forward(ctx, x, grad, scale):
        ctx.set_materialize_grads(False)
        ctx.scale = scale
        ctx.save_for_backward(x, grad)
        dx = torch.empty_like(x)
        _launch("ictc_silu_backward", x, scale, grad, dx)
        return dx

    @staticmethod
    def backward(ctx, h):
        if h is None:
            return None, None, None
        x, grad = ctx.saved_tensors
        rows = None if torch.is_grad_enabled() else kernels_take(x, grad, h)
        if rows is None:                             # third order and above, batched passes: plain operators
            s = torch.sigmoid(x)
            second = ctx.scale * s * (1 - s) * (2 + x * (1 - 2 * s))
            return h * grad * second, h * _first(x, ctx.scale), None
        x, grad, h = rows
        gx = torch.empty_like(x) if ctx.needs_input_grad[0] else None
        gg = torch.empty_like(x) if ctx.needs_input_grad[1] else None
        _launch("ictc_silu_second", x, ctx.scale, grad, h, gx, gg)
        return gx, gg, None


def scaled_silu(x, scale):
    return _Silu.apply(x, scale)
