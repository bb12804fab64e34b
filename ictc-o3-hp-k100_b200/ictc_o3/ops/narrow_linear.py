"""Bias-free linear map from 8 to 64 columns over many rows (the first radial layer in training).  The three functions are
closed under differentiation: each one's derivatives are the other two."""
from __future__ import annotations

import torch

from .. import _lib
from .activation import kernel_takes, runs_eagerly


def narrow_takes(rows, weight) -> bool:
    return (rows.ndim == 2 and tuple(weight.shape) == (64, 8) and rows.shape[1] == 8 and rows.shape[0] > 0
            and kernel_takes(rows) and kernel_takes(weight) and rows.device == weight.device)


def _aligned(t):
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _launch(name, *args):
    device = args[1].device
    with _lib.on_device(device):
        _lib.check(getattr(_lib.load(), name)(args[0], *[t.data_ptr() for t in args[1:]], _lib.stream(device)), name)


def _may_run(*tensors):
    """Looked at again in every backward pass, as in ``activation``; plain products otherwise."""
    return all(runs_eagerly(t) for t in tensors)


class NarrowLinear(torch.autograd.Function):
    """x [R, 8], w [64, 8] -> x w^T [R, 64]"""

    @staticmethod
    def forward(ctx, x, w):
        ctx.save_for_backward(x, w)
        y = torch.empty(x.shape[0], 64, dtype=x.dtype, device=x.device)
        _launch("ictc_narrow_linear_forward", x.shape[0], _aligned(x), _aligned(w), y)
        return y

    @staticmethod
    def backward(ctx, g):
        x, w = ctx.saved_tensors
        run = _may_run(x, w, g)
        dx = dw = None
        if ctx.needs_input_grad[0]:
            dx = _InputGrad.apply(g, w) if run else g @ w
        if ctx.needs_input_grad[1]:
            dw = _WeightGrad.apply(g, x) if run else g.transpose(-2, -1) @ x
        return dx, dw


class _InputGrad(torch.autograd.Function):
    """g [R, 64], w [64, 8] -> g w [R, 8]"""

    @staticmethod
    def forward(ctx, g, w):
        ctx.save_for_backward(g, w)
        dx = torch.empty(g.shape[0], 8, dtype=g.dtype, device=g.device)
        _launch("ictc_narrow_linear_input_grad", g.shape[0], _aligned(g), _aligned(w), dx)
        return dx

    @staticmethod
    def backward(ctx, h):
        g, w = ctx.saved_tensors
        run = _may_run(g, w, h)
        dg = dw = None
        if ctx.needs_input_grad[0]:
            dg = NarrowLinear.apply(h, w) if run else h @ w.transpose(-2, -1)
        if ctx.needs_input_grad[1]:
            dw = _WeightGrad.apply(g, h) if run else g.transpose(-2, -1) @ h
        return dg, dw


class _WeightGrad(torch.autograd.Function):
    """g [R, 64], x [R, 8] -> g^T x [64, 8]"""

    @staticmethod
    def forward(ctx, g, x):
        ctx.save_for_backward(g, x)
        rows = g.shape[0]
        dw = torch.empty(64, 8, dtype=g.dtype, device=g.device)
        work = torch.empty(_lib.load().ictc_narrow_linear_workspace(rows) // 4, dtype=g.dtype, device=g.device)
        _launch("ictc_narrow_linear_weight_grad", rows, _aligned(g), _aligned(x), dw, work)
        return dw

    @staticmethod
    def backward(ctx, h):
        g, x = ctx.saved_tensors
        run = _may_run(g, x, h)
        dg = dx = None
        if ctx.needs_input_grad[0]:
            dg = NarrowLinear.apply(x, h) if run else x @ h.transpose(-2, -1)
        if ctx.needs_input_grad[1]:
            dx = _InputGrad.apply(g, h) if run else g @ h
        return dg, dx
