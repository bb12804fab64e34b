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
