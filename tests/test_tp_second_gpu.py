"""Fused second derivatives of the graph message against the composition of forward and adjoint launches (what autograd runs
while it records) and against float64, with empty and long rows, unsorted lists, masks and path weights."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-5               # sums of 32-bit products, two derivatives deep


@pytest.mark.parametrize("degrees", [(2, 2, 2), (0, 2, 2), (1, 1, 1), (2, 2, 0)])
@pytest.mark.parametrize("channels,rows,edges,masked,weighted,ordered",
                         [(64, 1, 1, False, False, True), (64, 7, 2, True, False, False), (64, 40, 300, True, True, False),
                          (32, 23, 150, False, True, True), (32, 5, 200, True, False, False)])
def test_second_derivatives(degrees, channels, rows, edges, masked, weighted, ordered):
    from ictc_o3 import PackedGraphMessage
    from ictc_o3.ops.tensor_product import TpCall
    from oracle import ictc_oracle as O
    lin, ledge, _ = degrees
    gen = torch.Generator().manual_seed(rows * edges + channels)
    op = PackedGraphMessage.create(channels=channels, input_lmax=lin, edge_lmax=ledge, output_lmax=degrees[2])
    if weighted:
        op.tp.weight.copy_(torch.randn(op.tp.weight.shape, generator=gen))
    src, dst = (torch.randint(0, rows, (edges,), generator=gen) for _ in range(2))
    dst[: edges // 3] = 0                      # a long row
    if ordered:
        dst = dst.sort()[0]
    mask = (torch.rand(edges, generator=gen) > 0.3).float() if masked else None
    if masked:
        mask[0] = 1.0
    shapes = [(rows, channels * (lin + 1) ** 2), (edges, (ledge + 1) ** 2), (edges, op.gate_width)]
    args, tangents = ([torch.randn(s, generator=gen) for s in shapes] for _ in range(2))
    v = torch.randn(rows, op.output_width, generator=gen)
    used = []
    plain = TpCall.second
    TpCall.second = lambda self, *a: used.append(1) or plain(self, *a)

    def second(call, args, tangents, v, record):
        args, v = [t.requires_grad_(True) for t in args], v.requires_grad_(True)
        first = torch.autograd.grad(call(*args), args, v, create_graph=True)
        return [t.detach() for t in torch.autograd.grad(first, [*args, v], tangents, create_graph=record)]

    def run(record):
        cuda = lambda ts: [t.clone().cuda() for t in ts]                                      # noqa: E731
        return second(lambda x, sh, g: op(x, sh, g, src.cuda(), dst.cuda(), None if mask is None else mask.cuda()),
                      cuda(args), cuda(tangents), v.clone().cuda(), record)

    try:
        fused = run(False)
        assert used == [1]
        composed = run(True)
        assert used == [1]
    finally:
        TpCall.second = plain
    tp = O.TensorProduct(channels, op.tp.lmax, [tuple(p) for p in op.edge.paths])
    weight = op.tp.weight.detach().cpu().double().reshape(-1, channels)
    want = second(lambda x, sh, g: O.graph_message(tp, x, sh, g.reshape(edges, -1, channels), weight, src, dst,
                                                   None if mask is None else mask.double(), lin, ledge),
                  [t.double() for t in args], [t.double() for t in tangents], v.double(), False)
    for a, b, c in zip(fused, composed, want):
        scale = float(c.abs().max()) + 1e-30
        assert float((a - b).abs().max()) <= TOL * scale and float((a.double().cpu() - c).abs().max()) <= TOL * scale
