"""C entry points that the Python packages do not call themselves (a C or C++ host does): fixed-capacity edge buffers, position
gradient, graph message over ranges of owner rows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _lib():
    from ictc_o3 import _lib as L
    return L, L.load(), L.stream(torch.device("cuda"))


@pytest.mark.parametrize("capacity", [0, 5, 700, 1000])
def test_clamp_and_pad(capacity):
    L, lib, st = _lib()
    rng = np.random.default_rng(capacity)
    counts = rng.integers(0, 5, 300)
    rows = np.concatenate([[0], np.cumsum(counts)])
    rowptr = torch.as_tensor(rows).cuda()
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    L.check(lib.ictc_neighbor_clamp(rowptr.data_ptr(), 300, capacity, flag.data_ptr(), st), "clamp")
    assert np.array_equal(rowptr.cpu().numpy(), np.minimum(rows, capacity)) and int(flag) == int(rows[-1] > capacity)
    src, dst = (torch.full((capacity,), 9, dtype=torch.int64, device="cuda") for _ in range(2))
    shifts = torch.ones(capacity, 3, device="cuda")
    over = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    L.check(lib.ictc_neighbor_pad(rowptr.data_ptr() + 8 * 300, capacity, 123, 4, L.ptr(src), L.ptr(dst), L.ptr(shifts),
                                  over.data_ptr(), st), "pad")
    live = min(int(rows[-1]), capacity)
    assert bool((src[:live] == 9).all()) and bool((src[live:] == 123).all()) and bool((dst[live:] == 4).all())
    assert bool((shifts[:live] == 1).all()) and bool((shifts[live:] == 0).all()) and int(over) == 0


@pytest.mark.parametrize("nodes,owned", [(1, 1), (70, 70), (300, 120)])
def test_position_gradient(nodes, owned):
    from ictc_o3.ops.topology import build_csr
    L, lib, st = _lib()
    gen = torch.Generator("cuda").manual_seed(nodes)
    e = 20 * nodes
    dst = torch.sort(torch.randint(0, owned, (e,), device="cuda", generator=gen))[0]
    src = torch.randint(0, nodes, (e,), device="cuda", generator=gen)
    dvec = torch.randn(e, 3, device="cuda", generator=gen)
    rows = build_csr(dst, owned, True)[0]
    out_rows, order = build_csr(src, nodes, False)
    grad = torch.empty(nodes, 3, device="cuda")
    L.check(lib.ictc_position_gradient(nodes, owned, rows.data_ptr(), out_rows.data_ptr(), order.data_ptr(), dvec.data_ptr(),
                                       grad.data_ptr(), st), "position_gradient")
    want = torch.zeros(nodes, 3, dtype=torch.float64, device="cuda").index_add_(0, dst, dvec.double()).index_add_(0, src, -dvec.double())
    assert float((grad.double() - want).abs().max()) < 1e-5


@pytest.mark.parametrize("channels", [32, 64])
def test_graph_message_over_ranges_of_rows(channels):
    """Gates and gate gradients of a range in buffers of its own: the same rows as the whole table gives, in the one-warp-per-row
    order that a range of unknown context has (the whole call is large enough to use it, too)."""
    from ictc_o3 import _lib as L
    from ictc_o3.ops.topology import build_csr
    _, lib, st = _lib()
    spec = L.tp_spec(2, 2, 2)
    n, e, c = 4000, 12000, channels                       # beyond the limits of the split rows
    gen = torch.Generator("cuda").manual_seed(c)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen)     # noqa: E731
    dst = torch.sort(torch.randint(0, n, (e,), device="cuda", generator=gen))[0]
    src = torch.randint(0, n, (e,), device="cuda", generator=gen)
    x, sh, g, v = make(n, 9 * c), make(e, 9), make(e, 11 * c), make(n, 35 * c)
    (rows, _), (out_rows, order) = build_csr(dst, n, True), build_csr(src, n, False)
    want = torch.empty(n, 35 * c, device="cuda")
    L.check(lib.ictc_tp_graph_forward(spec, c, n, e, x.data_ptr(), sh.data_ptr(), None, g.data_ptr(), src.data_ptr(),
                                      rows.data_ptr(), None, None, want.data_ptr(), st), "forward")
    dx, dsh, dg = torch.empty_like(x), torch.empty_like(sh), torch.empty_like(g)
    L.check(lib.ictc_tp_graph_adjoint(spec, c, n, e, x.data_ptr(), sh.data_ptr(), None, g.data_ptr(), dst.data_ptr(),
                                      out_rows.data_ptr(), order.data_ptr(), None, v.data_ptr(), dx.data_ptr(), dsh.data_ptr(),
                                      dg.data_ptr(), st), "adjoint")
    got, got_dx, got_dsh, got_dg = torch.empty_like(want), torch.empty_like(x), torch.empty_like(sh), torch.empty_like(g)
    cuts = [0, 1, 1500, n]
    at, out_at = rows.tolist(), out_rows.tolist()
    for a, b in zip(cuts[:-1], cuts[1:]):
        part = g[at[a]:at[b]].clone()
        L.check(lib.ictc_tp_graph_forward_chunk(spec, c, b - a, x.data_ptr(), sh.data_ptr(), None, part.data_ptr() or x.data_ptr(),
                                                None, rows.data_ptr() + 8 * a, max(at[b] - at[a], 1), src.data_ptr(),
                                                rows.data_ptr() + 8 * a, None, None, got.data_ptr() + 4 * a * 35 * c, st), "chunk")
        ids = order[out_at[a]:out_at[b]]
        part, grads = torch.cat((g[ids], g[:1])), torch.empty(len(ids) + 1, 11 * c, device="cuda")
        L.check(lib.ictc_tp_graph_adjoint_chunk(spec, c, b - a, x.data_ptr() + 4 * a * 9 * c, sh.data_ptr(), None,
                                                part.data_ptr(), None, 1, out_rows.data_ptr() + 8 * a, len(ids) + 1,
                                                dst.data_ptr(), out_rows.data_ptr() + 8 * a, order.data_ptr(), None, v.data_ptr(),
                                                got_dx.data_ptr() + 4 * a * 9 * c, got_dsh.data_ptr(), grads.data_ptr(),
                                                out_rows.data_ptr() + 8 * a, len(ids) + 1, st), "chunk adjoint")
        got_dg[ids] = grads[:-1]
    for a, b in ((got, want), (got_dx, dx), (got_dsh, dsh), (got_dg, dg)):
        assert torch.equal(a, b)
