"""Scaled SiLU with fused first and second derivatives (reference: modes 0 to 2 of
ictc_o3/backends/k100/hip_activation.py:27-38)."""
from __future__ import annotations

import torch

from .. import _lib


def kernel_takes(x) -> bool:
    """The kernels take contiguous float32 CUDA tensors in eager reverse-mode differentiation; everything else stays with the
    framework's operators."""
    return (type(x) in (torch.Tensor, torch.nn.Parameter) and x.is_cuda and x.dtype == torch.float32
            and x.layout == torch.strided and x.is_contiguous() and not torch._C._are_functorch_transforms_active()
            and torch.autograd.forward_ad._current_level < 0 and not torch.compiler.is_compiling()
            and not torch.is_autocast_enabled("cuda"))


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
        return _SiluGrad.apply(x, grad.contiguous(), ctx.scale), None


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
        if torch.is_grad_enabled():                  # third order and above: plain operators
            s = torch.sigmoid(x)
            first = ctx.scale * s * (1 + x * (1 - s))
            second = ctx.scale * s * (1 - s) * (2 + x * (1 - 2 * s))
            return h * grad * second, h * first, None
        gx = torch.empty_like(x) if ctx.needs_input_grad[0] else None
        gg = torch.empty_like(x) if ctx.needs_input_grad[1] else None
        _launch("ictc_silu_second", x, ctx.scale, grad, h.contiguous(), gx, gg)
        return gx, gg, None


def scaled_silu(x, scale):
    return _Silu.apply(x, scale)
