"""``ictc_neighbor_build`` (whole list in one call) against the brute-force oracle and the separate entry points: rows
longer than the staging buffer, one to three cells per axis, an atom that is its own neighbour (box = cutoff), centres
that are a prefix of the rows, and a capacity that just fits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CUTOFF = 4.5


@pytest.mark.parametrize("n,box,periodic,centres,extra", [
    (1, (4.5, 4.5, 4.5), (1, 1, 1), 1, 7),              # six images of itself exactly at the cutoff
    (2, (4.5, 9.0, 13.5), (1, 1, 1), 2, 64),
    (200, (5.0, 9.1, 14.0), (1, 1, 1), 200, 1),         # 1 x 2 x 3 cells, about 120 neighbours: both staging routes
    (300, (9.5, 9.5, 9.5), (1, 1, 1), 300, 1),          # rows of 130 keys
    (333, (14.0, 18.2, 23.0), (1, 0, 1), 120, 500),     # centres are a prefix: some senders are not centres
    (2100, (30.0, 27.0, 26.0), (0, 0, 0), 2100, 1),     # more than one tile of rows
])
def test_list_pairs_and_sender_order(n, box, periodic, centres, extra):
    from mace_ictc.md import StaticNeighborList, edge_pairs, neighbor_list
    from oracle import ictc_oracle as O
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 3)) * np.array(box)).astype(np.float32)
    rs, rd, rsh = O.neighbor_list_bruteforce(pos, centres, box, periodic, CUTOFF)
    p = torch.as_tensor(pos).cuda()
    e = len(rs)
    nl = StaticNeighborList(n, box, CUTOFF, e + extra, p.device, num_centres=centres, periodic=periodic,
                            pair_fraction=1.0)
    nl.build(torch.cat((p, torch.full((1, 3), -1.0e6, device="cuda"))))
    edges, pairs, over = nl.counts()
    assert (edges, over) == (e, False)
    assert np.array_equal(nl.src[:e].cpu().numpy(), rs) and np.array_equal(nl.dst[:e].cpu().numpy(), rd)
    assert np.array_equal(nl.shifts[:e].cpu().numpy(), np.asarray(rsh, dtype=np.float32))
    assert bool((nl.src[e:] == n).all()) and bool((nl.dst[e:] == 0).all()) and bool((nl.gate_row[e:] == 0).all())
    assert np.array_equal(nl.rowptr.cpu().numpy(), np.searchsorted(rd, np.arange(centres + 1)))
    # the pair table of the entry point that scans over the edges
    src, dst, _, rowptr, keys = neighbor_list(p, centres, [0, 0, 0], box, box, periodic, CUTOFF, True)
    gate_row, rep, other = edge_pairs(rowptr, dst, keys, centres)
    assert pairs == rep.numel()
    assert torch.equal(nl.gate_row[:e], gate_row)
    assert torch.equal(nl.rep[:pairs], rep) and torch.equal(nl.other[:pairs], other)
    assert bool((nl.rep[pairs:] == e + extra - 1).all()) and bool((nl.other[pairs:] == -1).all())
    if centres == n:            # every edge has its reverse: rev is an involution that swaps the ends
        rev = nl.rev[:e]
        assert torch.equal(rev[rev], torch.arange(e, device="cuda"))
        assert torch.equal(src[rev], dst) and torch.equal(dst[rev], src)


def test_capacity_that_does_not_fit_is_flagged():
    from mace_ictc.md import StaticNeighborList
    rng = np.random.default_rng(5)
    p = torch.as_tensor((rng.random((150, 3)) * 11.0).astype(np.float32)).cuda()
    nl = StaticNeighborList(150, (11.0,) * 3, CUTOFF, 37, p.device, dummy_row=False)
    nl.build(p)
    edges, _, over = nl.counts()
    assert over and edges == 36
    for t, top in ((nl.src, 150), (nl.dst, 150), (nl.rev, 37), (nl.gate_row, nl.ucap), (nl.rep, 37)):
        assert int(t.min()) >= 0 and int(t.max()) < top


@pytest.mark.parametrize("use_engine", [True, False])
def test_eager_steps_follow_a_changed_box_cutoff_and_atom_count(use_engine):
    """The buffers of the eager list outlive a step, what they were built for must not."""
    from mace_ictc import synthetic as S
    from mace_ictc.hp import create_model
    from mace_ictc.md import MolecularDynamics, neighbor_list
    torch.manual_seed(2)
    model = create_model(channels=64, lmax=2, cutoff=CUTOFF, avg_num_neighbors=32.0)
    pos, box, species = S.jittered_lattice(6, 7, 8, 2.15, 0.1, 3)
    z = np.array([1, 6, 8])[species]
    md = MolecularDynamics(model, pos, z, box, seed=1, use_engine=use_engine)
    md.compute_forces()

    def check():
        fresh = MolecularDynamics(model, md.pos.cpu().numpy(), md.z.cpu().numpy(), md.box.numpy(), seed=1, sort_atoms=False,
                                  use_engine=use_engine)
        fresh.cutoff = md.cutoff
        want = fresh.compute_forces()
        assert md.compute_forces().shape == want.shape and md.num_edges == fresh.num_edges
        assert torch.equal(md.forces, want) or not use_engine and float((md.forces - want).abs().max()) < 1e-4 * float(want.abs().max())

    check()
    for factor in (1.04, 0.97):                     # a barostat's changes, below and above the first box
        md.box *= factor
        md.box_f = md.box.to(md.device, torch.float32)
        md.pos *= factor
        check()
    md.cutoff = 3.0
    check()
    md.pos, md.z, md.species = (t[:-9].contiguous() for t in (md.pos, md.z, md.species))
    check()
    md.pos = md.pos.t().contiguous().t()            # other strides
    check()
    rows = neighbor_list(md.pos, md.pos.shape[0], [0, 0, 0], md.box.tolist(), md.box.tolist(), (1, 1, 1), md.cutoff)
    assert md.num_edges == rows[0].numel()
