"""Scaled SiLU and its derivatives against float64, at sizes around the 16-byte pieces and on shifted buffers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
# value and derivatives are a few rounded operations and one expf (2 ulp) per element; near the zeros of the derivatives the
# rounding of their terms stays, which is why the bound is on the difference
TOL = 2e-6


@pytest.mark.parametrize("n,shift", [(1, 0), (3, 0), (4, 1), (1023, 0), (1024, 0), (65541, 0), (65541, 1)])
def test_derivatives_up_to_third_order(n, shift):
    from ictc_o3 import normalized_silu
    gen = torch.Generator("cuda").manual_seed(n)
    store = [4 * torch.randn(n + 1, device="cuda", generator=gen) for _ in range(3)]
    x, g, h = (t[shift:shift + n].requires_grad_(True) for t in store)
    wide = [t.detach().double().requires_grad_(True) for t in (x, g, h)]

    def chain(x, g, h, f):
        y = f(x)
        (d,) = torch.autograd.grad(y, x, g, create_graph=True)
        first = torch.autograd.grad(d, [x, g], h, retain_graph=True)
        second = torch.autograd.grad(d, [x, g], h, create_graph=True)
        return [y, d, *first, *torch.autograd.grad((second[0] * g + second[1]).sum(), [x, g])]

    got = chain(x, g, h, lambda t: normalized_silu(t, 1.7))
    want = chain(*wide, lambda t: 1.7 * torch.nn.functional.silu(t))
    for a, b in zip(got, want):
        scale = max(1.0, float(b.detach().abs().max()))
        assert float((a.detach().double() - b.detach()).abs().max()) < TOL * scale


def test_batched_traced_and_forward_mode_calls_keep_the_framework_operators():
    """Forms in which no kernel can run, decided at the forward call or only in the backward pass."""
    from ictc_o3 import normalized_silu
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils.flop_counter import FlopCounterMode
    x = torch.randn(6, device="cuda", requires_grad=True)
    v = torch.randn(4, 6, device="cuda")
    ours, plain = (lambda t: normalized_silu(t, 1.7)), (lambda t: 1.7 * torch.nn.functional.silu(t))

    def close(a, b):
        assert a.shape == b.shape and float((a - b).detach().abs().max()) < 8 * TOL      # eight: double backward of sums

    for f in (lambda g: torch.autograd.grad(g(x), x, v, is_grads_batched=True)[0],
              lambda g: torch.autograd.grad(torch.autograd.grad(g(x), x, v[0], create_graph=True)[0], x, v, is_grads_batched=True)[0],
              lambda g: torch.autograd.grad(torch.autograd.grad(g(x), x, v, create_graph=True, is_grads_batched=True)[0].sum(), x)[0],
              lambda g: torch.autograd.functional.jacobian(g, x, vectorize=True),
              lambda g: torch.autograd.functional.hessian(lambda t: g(t).sum(), x, vectorize=True),
              lambda g: torch.func.vmap(lambda u, y=g(x): torch.autograd.grad(y, x, u, retain_graph=True)[0])(v),
              lambda g: torch.func.jacfwd(g)(x.detach()), lambda g: torch.func.vmap(torch.func.grad(lambda t: g(t).sum()))(v),
              lambda g: g(torch._neg_view(x.detach()))):
        close(f(ours), f(plain))

    def hooked(g):                                  # hooks that hand other strides back
        turned = torch.randn(7, 5, device="cuda", generator=torch.Generator("cuda").manual_seed(1)).requires_grad_(True)
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t.t().contiguous(), lambda t: t.t()):
            y = g(turned)
        return torch.autograd.grad(y, turned, torch.ones_like(turned))[0]
    close(hooked(ours), hooked(plain))

    graph = make_fx(ours)(v)
    close(graph(v + 1), ours(v + 1))
    close(torch.jit.trace(ours, v)(v + 1), ours(v + 1))
    with FlopCounterMode(display=False):
        close(ours(v), plain(v))
