"""Graph messages at row counts around the point where the edges of a row are no longer shared among warps, with rows of 0 to
70 edges, unsorted edge lists and edge masks: against the plain sum in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-5               # one operator in 32-bit sums; the sum of a row of 70 edges is split in four


@pytest.mark.parametrize("channels,rows,masked,ordered", [(64, 1, False, True), (64, 3, True, False), (64, 1776, False, False),
                                                          (64, 1777, True, True), (32, 888, True, False), (32, 889, False, True),
                                                          (64, 3552, False, True), (32, 3553, True, False)])
@pytest.mark.parametrize("degrees", [(2, 2, 2), (0, 2, 2)])
def test_message_and_gradients(channels, rows, masked, ordered, degrees):
    from ictc_o3 import PackedGraphMessage
    from oracle import ictc_oracle as O
    gen = torch.Generator().manual_seed(rows + channels)
    op = PackedGraphMessage.create(channels=channels, input_lmax=degrees[0], edge_lmax=2, output_lmax=2)
    ends = 24                                  # the oracle sees a block of rows; the others have no edges among them
    edges = 400 if rows > 3 else 70 * rows
    pick = torch.randperm(rows, generator=gen)[:ends]
    src, dst = (pick[torch.randint(0, len(pick), (edges,), generator=gen)] for _ in range(2))
    if rows > 3:
        dst[:70] = pick[0]
        src[70:140] = pick[1]
    if ordered:
        dst = dst.sort()[0]
    x = torch.randn(rows, channels * (degrees[0] + 1) ** 2, generator=gen)
    sh, g = torch.randn(edges, 9, generator=gen), torch.randn(edges, op.gate_width, generator=gen)
    mask = (torch.rand(edges, generator=gen) > 0.2).float() if masked else None
    xd, sd, gd = (t.cuda().requires_grad_(True) for t in (x, sh, g))
    out = op(xd, sd, gd, src.cuda(), dst.cuda(), None if mask is None else mask.cuda())
    v = torch.randn(out.shape, generator=gen)
    grads = torch.autograd.grad(out, [xd, sd, gd], v.cuda())
    tp = O.TensorProduct(channels, 2, [tuple(p) for p in op.edge.paths])
    small = torch.full((rows,), -1)
    small[pick] = torch.arange(len(pick))
    xr, sr, gr = (t.double().requires_grad_(True) for t in (x[pick], sh, g))
    ref = O.graph_message(tp, xr, sr, gr.reshape(edges, -1, channels), torch.ones(op.edge.tp.num_paths, channels, dtype=torch.float64),
                          small[src], small[dst], None if mask is None else mask.double(), degrees[0], 2)
    wants = torch.autograd.grad(ref, [xr, sr, gr], v[pick].double())
    rest = torch.ones(rows, dtype=torch.bool)
    rest[pick] = False
    assert float(out.detach().cpu()[rest].abs().sum()) == 0.0 and float(grads[0].cpu()[rest].abs().sum()) == 0.0
    pairs = [(out.detach().cpu()[pick], ref.detach()), (grads[0].cpu()[pick], wants[0]), (grads[1].cpu(), wants[1]),
             (grads[2].cpu(), wants[2])]
    for got, want in pairs:
        assert float((got.double() - want).abs().max()) < TOL * float(want.abs().max())
