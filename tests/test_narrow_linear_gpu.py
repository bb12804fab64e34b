"""The 8 -> 64 linear map and its first and second derivatives against float64, around its blocks and on shifted buffers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


@pytest.mark.parametrize("rows,shift", [(1, 0), (15, 1), (17, 0), (129, 0), (18945, 0), (100003, 0)])
def test_value_and_derivatives(rows, shift):
    from ictc_o3.ops.narrow_linear import NarrowLinear, narrow_takes
    gen = torch.Generator("cuda").manual_seed(rows)
    make = lambda *s: torch.randn(s[0] * s[1] + shift, device="cuda", generator=gen)[shift:].reshape(s)     # noqa: E731
    x, w, g, hx, hw = make(rows, 8), make(64, 8), make(rows, 64), make(rows, 8), make(64, 8)
    assert narrow_takes(x, w)

    def chain(f, x, w, g, hx, hw):
        x, w, g = (t.clone() if t.dtype == torch.float64 else t for t in (x, w, g))
        x, w, g = (t.detach().requires_grad_(True) for t in (x, w, g))
        y = f(x, w)
        first = torch.autograd.grad(y, [x, w], g, create_graph=True)
        return [y.detach(), *(t.detach() for t in first), *torch.autograd.grad(first, [x, w, g], [hx, hw])]

    got = chain(NarrowLinear.apply, x, w, g, hx, hw)
    d = [t.double() for t in (x, w, g, hx, hw)]
    want = chain(lambda a, b: a @ b.t(), *d)
    size = chain(lambda a, b: a @ b.t(), *[t.abs() for t in d])          # sums of the terms' magnitudes
    # a sum of n terms in 32 bits is off by at most n half-units of that; random signs leave far less: 8 + sqrt(rows)
    for a, b, s in zip(got, want, size):
        assert float(((a.double() - b).abs() - (16 + rows ** 0.5) * EPS * s).max()) <= 0.0


def test_batched_backward_passes_and_hooks_with_other_strides():
    from ictc_o3.ops.narrow_linear import NarrowLinear
    gen = torch.Generator("cuda").manual_seed(4)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen)     # noqa: E731
    x, w = make(33, 8).requires_grad_(True), make(64, 8).requires_grad_(True)
    v, hx, hw = make(3, 33, 64), make(3, 33, 8), make(3, 64, 8)

    def chain(f):
        y = f(x, w)
        first = torch.autograd.grad(y, [x, w], v, is_grads_batched=True, retain_graph=True)
        single = torch.autograd.grad(y, [x, w], v[0], create_graph=True)
        second = torch.autograd.grad(single, [x, w], [hx, hw], is_grads_batched=True)
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t.t().contiguous(), lambda t: t.t()):
            y = f(x, w)
        return [*first, *second, *torch.autograd.grad(y, [x, w], v[1])]

    for a, b in zip(chain(NarrowLinear.apply), chain(lambda a, b: a @ b.t())):
        assert a.shape == b.shape and float((a - b).abs().max()) < 64 * EPS * float(b.abs().max())      # sums of 64 terms


def test_the_first_radial_layer_honours_replaced_forwards_and_global_hooks():
    from mace_ictc.model import MaceIctcModel
    inter = MaceIctcModel(channels=64).cuda().interactions[0]
    rows = torch.rand(40, 8, device="cuda")
    plain = inter.radial_gates(rows)
    inter.fc[0].forward = lambda t: 0.5 * torch.nn.functional.linear(t, inter.fc[0].weight)
    halved = inter.radial_gates(rows)
    del inter.fc[0].forward
    assert float((halved - plain).abs().max()) > 0.01 * float(plain.abs().max())
    seen = []
    handle = torch.nn.modules.module.register_module_forward_hook(lambda module, *_: seen.append(module))
    inter.radial_gates(rows)
    handle.remove()
    assert inter.fc[0] in seen
    assert torch.equal(inter.radial_gates(rows), plain)
