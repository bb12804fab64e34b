"""The native force sweep behind ``energy_and_forces`` and the MD drivers: against the autograd route (every edge order,
general cells, batches of graphs, masks, sizes around the kernels' blocks), stage by stage around an exchange of ghost
rows, after parameter updates, and its error cases."""
import copy

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-5          # fp32 against fp32 over two layers: the two routes each hold 1e-5 against the float64 oracle
ELEMENTS = (1, 6, 8)


def _model(seed=1):
    from mace_ictc.hp import create_model
    torch.manual_seed(seed)
    model = create_model(channels=64, lmax=2, cutoff=4.5, avg_num_neighbors=32.0)
    with torch.no_grad():
        for name, p in model.named_parameters():
            if "linear_up" in name or "self_connection" in name:
                p.add_(0.05 * torch.randn_like(p))
    return model


def _autograd(model, graph, mask=None):
    """The tape route (what training uses)."""
    from mace_ictc.hp import energy_and_forces
    return {k: v.detach() for k, v in energy_and_forces(model, *graph, training=True, owned_mask=mask).items()}


def _close(got, want, tol=TOL):
    for key in want:
        err = float((got[key] - want[key]).abs().max()) / float(want[key].abs().max())
        assert err < tol, (key, err)


def _graph(rng, sizes, skewed):
    """Random gases, one cell each (skewed or rectangular), every edge within 5 A: some lie beyond the cutoff."""
    pos, z, batch, src, dst, shifts, cells = [], [], [], [], [], [], []
    first = 0
    for g, n in enumerate(sizes):
        side = max(10.0, (n / 0.05) ** (1.0 / 3.0))
        cell = np.diag([side, side * 1.1, side * 0.95])
        if skewed:
            cell += rng.normal(0.0, 0.6, (3, 3))
        p = rng.random((n, 3)) @ cell
        images = np.stack(np.meshgrid(*[[-1, 0, 1]] * 3, indexing="ij"), -1).reshape(-1, 3)
        for image in images:
            vec = p[None, :, :] - p[:, None, :] + image @ cell           # [src, dst]
            near = (np.linalg.norm(vec, axis=-1) < 5.0) & (np.linalg.norm(vec, axis=-1) > 0.7)
            j, i = np.nonzero(near)
            src.append(j + first)
            dst.append(i + first)
            shifts.append(np.repeat(image[None], len(j), 0))
        pos.append(p)
        z.append(rng.choice(ELEMENTS, n))
        batch.append(np.full(n, g))
        cells.append(cell)
        first += n
    src, dst, shifts = np.concatenate(src), np.concatenate(dst), np.concatenate(shifts)
    order = rng.permutation(len(src))
    t = lambda a, d: torch.as_tensor(np.asarray(a), dtype=d, device="cuda")       # noqa: E731
    return [t(np.concatenate(pos), torch.float32), t(np.concatenate(z), torch.int64), t(np.concatenate(batch), torch.int64),
            t(src[order], torch.int64), t(dst[order], torch.int64), t(shifts[order], torch.int64), t(cells, torch.float32)]


@pytest.mark.parametrize("sizes,skewed", [((2,), False), ((33,), True), ((70, 1, 40), True), ((129,) * 3, False), ((700,), True)])
def test_against_the_autograd_route(sizes, skewed):
    from mace_ictc.hp import energy_and_forces
    model = _model()
    graph = _graph(np.random.default_rng(sum(sizes)), sizes, skewed)
    _close(energy_and_forces(model, *graph), _autograd(model, graph))
    order = torch.argsort(graph[4], stable=True)
    for k in (3, 4, 5):
        graph[k] = graph[k][order]
    model.preserve_edge_order = True
    model.skip_input_validation = True
    mask = (torch.arange(sum(sizes), device="cuda") % 3 != 1).float()
    want = _autograd(model, graph, mask)
    got = energy_and_forces(model, *graph, owned_mask=mask)
    _close(got, want)
    assert torch.equal(got["forces"], energy_and_forces(model, *graph, owned_mask=mask)["forces"])


def test_parameter_updates_replacement_copies_and_hooks():
    from mace_ictc.hp import energy_and_forces
    model = _model()
    graph = _graph(np.random.default_rng(3), (50,), False)
    before = energy_and_forces(model, *graph)
    twin = copy.deepcopy(model)
    with torch.no_grad():
        model.products[0].linear["1"].mul_(1.5)
    _close(energy_and_forces(model, *graph), _autograd(model, graph))
    model.interactions[1].fc[0].weight = torch.nn.Parameter(model.interactions[1].fc[0].weight * 0.9)
    _close(energy_and_forces(model, *graph), _autograd(model, graph))
    model.interactions[0].avg_num_neighbors = 20.0
    after = energy_and_forces(model, *graph)
    _close(after, _autograd(model, graph))
    assert float((after["forces"] - before["forces"]).abs().max()) > 1e-3 * float(before["forces"].abs().max())
    assert torch.equal(energy_and_forces(twin, *graph)["forces"], before["forces"])
    seen = []
    handle = model.products[1].register_forward_hook(lambda *_: seen.append(1))
    energy_and_forces(model, *graph)
    assert seen == [1]
    handle.remove()
    model.products[0].linear["2"].data.mul_(0.7)              # no version counter moves
    model.last_layer_energy_readout.linear_2.weight.data.copy_(torch.randn(1, 16, device="cuda"))
    _close(energy_and_forces(model, *graph), _autograd(model, graph))
    model.interactions[1].fc[1] = torch.nn.Tanh()             # a module that the sweep does not know
    _close(energy_and_forces(model, *graph), _autograd(model, graph))


def test_parameters_at_any_word_of_a_flattened_buffer():
    from mace_ictc.hp import energy_and_forces
    model = _model()
    graph = _graph(np.random.default_rng(11), (30,), False)
    want = energy_and_forces(model, *graph)
    params = list(model.parameters())
    flat = torch.empty(sum(p.numel() + 2 for p in params) + 2, device="cuda")
    at = 1
    for p in params:
        view = flat[at:at + p.numel()].view_as(p)
        p.data = view.copy_(p.data)
        at += p.numel() + 1 + (at + p.numel()) % 2        # every parameter at an odd word
    assert all(p.data_ptr() % 8 == 4 for p in params)
    got = energy_and_forces(model, *graph)
    assert torch.equal(got["forces"], want["forces"]) and torch.equal(got["atomic_energy"], want["atomic_energy"])
    _close(got, _autograd(model, graph))


def test_models_with_other_readouts_answer_through_their_own_forward():
    from mace_ictc.hp import energy_and_forces
    from mace_ictc.md import MolecularDynamics
    from mace_ictc.model import MLPReadout
    graph = _graph(np.random.default_rng(8), (45,), False)

    def linear(rows, cols, bias):
        return torch.nn.Linear(cols, rows, bias=bias, device="cuda")

    changes = [lambda m: setattr(m.last_layer_energy_readout, "linear_2", linear(1, 16, True)),
               lambda m: setattr(m.last_layer_energy_readout, "linear_1", linear(16, 64, True)),
               lambda m: setattr(m.layer_energy_readouts[0], "readout", linear(1, 64, True)),
               lambda m: setattr(m.last_layer_energy_readout, "linear_2", linear(3, 16, False)),
               lambda m: setattr(m.last_layer_energy_readout, "activation", torch.nn.Sequential()),
               lambda m: m.interactions[1].fc.__setitem__(1, torch.nn.Sequential()),
               lambda m: m.layer_energy_readouts.__setitem__(0, MLPReadout(9 * 64).cuda())]
    for change in changes:
        model = _model()
        stock = energy_and_forces(model, *graph)
        change(model)
        got, want = energy_and_forces(model, *graph), _autograd(model, graph)
        _close(got, want)
        assert float((got["atomic_energy"] - stock["atomic_energy"]).abs().max()) > 1e-3      # the change does something
        box = np.full(3, 12.0)
        md = MolecularDynamics(model, graph[0].cpu().numpy() % 12.0, graph[1].cpu().numpy(), box)
        ref = MolecularDynamics(model, graph[0].cpu().numpy() % 12.0, graph[1].cpu().numpy(), box, use_engine=False)
        md.compute_forces(), ref.compute_forces()
        assert abs(float(md.energy) - float(ref.energy)) < TOL * abs(float(ref.energy))


def test_weights_laid_out_on_another_stream():
    from mace_ictc.hp import energy_and_forces
    model = _model()
    graph = _graph(np.random.default_rng(5), (60,), False)
    want = _autograd(model, graph)
    for _ in range(3):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.no_grad():
            model.products[0].linear["1"].mul_(1.0)           # laid out again, here on the current stream
        energy_and_forces(model, *graph)
        with torch.cuda.stream(side):
            got = energy_and_forces(model, *graph)
        torch.cuda.current_stream().wait_stream(side)
        _close(got, want)


def test_unknown_atoms_and_bad_edges_raise_and_the_next_call_works():
    from mace_ictc.hp import energy_and_forces
    model = _model()
    graph = _graph(np.random.default_rng(4), (40,), False)
    good = energy_and_forces(model, *graph)
    for index, value in ((1, 7), (1, 500), (2, 1), (2, -1), (3, 40), (4, -1)):
        bad = list(graph)
        bad[index] = bad[index].clone()
        bad[index][5] = value
        with pytest.raises(ValueError):
            energy_and_forces(model, *bad)
    for index in (3, 5):                                      # one row short: refused before anything is launched
        bad = list(graph)
        bad[index] = bad[index][:-1]
        with pytest.raises(ValueError):
            energy_and_forces(model, *bad)
    with pytest.raises((ValueError, RuntimeError)):
        energy_and_forces(model, *graph, owned_mask=torch.ones(40))
    assert torch.equal(energy_and_forces(model, *graph)["forces"], good["forces"])


def test_small_sweeps_queued_behind_each_other_do_not_see_each_other():
    """Launches of about one wave start before the previous one has ended: sweeps of other sizes (pair rows, CSR offsets, chunk
    bounds, features) right behind each other give what each gives alone."""
    from mace_ictc import synthetic as S
    from mace_ictc.hp import energy_and_forces
    from mace_ictc.md import MolecularDynamics
    model = _model()
    model.skip_input_validation = True
    graphs = [_graph(np.random.default_rng(k), (n,), False) for k, n in enumerate((33, 150, 45, 90))]
    runs = []
    for k, (side, chunk) in enumerate(((6, None), (7, 64), (6, 100))):
        pos, box, species = S.jittered_lattice(side, side, side, 2.15, 0.1, k)
        md = MolecularDynamics(model, pos, np.array(ELEMENTS)[species], box, seed=k, chunk_rows=chunk, stream_gates=chunk == 64)
        md.compute_forces()
        runs.append(md)
    alone = []
    for graph in graphs:
        alone.append(energy_and_forces(model, *graph)["forces"])
        torch.cuda.synchronize()
    steps = []
    for md in runs:
        steps.append(md.compute_forces().clone())
        torch.cuda.synchronize()
    for _ in range(10):
        got = [energy_and_forces(model, *graph)["forces"] for graph in graphs]
        forces = [md.compute_forces() for md in runs]
        assert all(torch.equal(a, b) for a, b in zip(got + forces, alone + steps))


@pytest.mark.parametrize("share_gates,chunk_rows,stream_gates", [(True, None, None), (False, None, None), (True, 1, True)])
def test_atoms_without_any_neighbour(share_gates, chunk_rows, stream_gates):
    from mace_ictc.hp import energy_and_forces
    from mace_ictc.md import MolecularDynamics
    model = _model()
    pos, z = np.array([[1.0, 1.0, 1.0], [9.0, 9.0, 9.0], [1.0, 9.0, 17.0]]), np.array([1, 6, 8])
    md = MolecularDynamics(model, pos, z, np.full(3, 24.0), velocities=np.zeros((3, 3)), share_gates=share_gates,
                           chunk_rows=chunk_rows, stream_gates=stream_gates)
    assert md.engine is not None and bool((md.compute_forces() == 0).all()) and md.num_edges == 0
    empty = torch.zeros(0, dtype=torch.int64, device="cuda")
    graph = [torch.as_tensor(pos, dtype=torch.float32).cuda(), torch.as_tensor(z).cuda(), torch.zeros(3, dtype=torch.int64, device="cuda"),
             empty, empty, torch.zeros(0, 3, device="cuda"), 24.0 * torch.eye(3, device="cuda").unsqueeze(0)]
    alone = energy_and_forces(model, *graph)
    assert bool((alone["forces"] == 0).all()) and torch.isfinite(alone["energy"]).all()
    assert abs(float(md.energy) - float(alone["energy"])) < 1e-5 * abs(float(alone["energy"]))
    tape = energy_and_forces(model, *graph, training=True)
    tape["energy"].sum().backward()
    assert all(p.grad is None or torch.isfinite(p.grad).all() for p in model.parameters())
    md.step()
    md.enable_graph()
    md.run(2)
    assert bool((md.forces == 0).all()) and abs(float(md.energy) - float(alone["energy"])) < 1e-5 * abs(float(alone["energy"]))


def test_a_rank_without_owned_rows():
    """Ghost rows alone: nothing to sum up, no launch without rows."""
    from mace_ictc.engine import ForceEngine
    model = _model()
    pos = torch.rand(5, 3, device="cuda")
    empty = torch.zeros(0, dtype=torch.int64, device="cuda")
    energy, grad, atomic = ForceEngine(model).energy_and_gradient(pos, empty.new_zeros(5), empty, empty, None, [9.0, 9.0, 9.0], 0,
                                                                  empty.new_zeros(1))
    assert float(energy) == 0.0 and atomic.numel() == 0 and bool((grad == 0).all())


@pytest.mark.parametrize("side,chunk_rows", [(6, None), (22, None), (22, 4000)])
def test_energies_repeat_bit_by_bit(side, chunk_rows):
    """Below and above the sizes where a warp of the readout takes several atoms; an order of additions that changed from run to
    run would show in the last bit of some of these sums."""
    from mace_ictc import synthetic as S
    from mace_ictc.hp import energy_and_forces
    from mace_ictc.md import MolecularDynamics
    model = _model()
    with torch.no_grad():
        model.layer_energy_readouts[0].readout.weight.mul_(1e3)         # large terms of both signs
    pos, box, species = S.jittered_lattice(side, side, side, 2.15, 0.1, 5)
    z = np.array(ELEMENTS)[species]
    md = MolecularDynamics(model, pos, z, box, seed=2, chunk_rows=chunk_rows)
    md.compute_forces()
    first = md.energy.clone()
    whole = MolecularDynamics(model, pos, z, box, seed=2)
    whole.compute_forces()
    assert torch.equal(first, whole.energy)
    exact = float(whole.engine.energy_and_gradient(whole.pos, whole.species, *_edges(whole))[2].double().sum())
    assert abs(float(first) - exact) <= 1e-7 * abs(exact)              # the blocks' sums are in double precision
    for _ in range(5):
        md.compute_forces()
        assert torch.equal(md.energy, first)
    src, dst, shifts = whole._eager_list.src, whole._eager_list.dst, whole._eager_list.shifts
    graph = [whole.pos, whole.z, torch.zeros_like(whole.z), src[:whole.num_edges], dst[:whole.num_edges], shifts[:whole.num_edges],
             torch.diag(whole.box_f).unsqueeze(0)]
    energies = {float(energy_and_forces(model, *graph)["energy"]) for _ in range(5)}
    assert len(energies) == 1


def _edges(md):
    nl, e = md._eager_list, md.num_edges
    return nl.src[:e], nl.dst[:e], nl.shifts[:e], md.box.tolist(), md.pos.shape[0], nl.rowptr


def test_a_deleted_model_gives_its_memory_back_at_once():
    import gc
    import weakref
    from mace_ictc.engine import ForceEngine
    from mace_ictc.hp import energy_and_forces
    graph = _graph(np.random.default_rng(1), (20,), False)
    model = _model()
    energy_and_forces(model, *graph)
    before = torch.cuda.memory_allocated()
    gc.disable()
    try:
        model = _model()
        energy_and_forces(model, *graph)
        seen, engine = weakref.ref(model), weakref.ref(model.__dict__["_force_engine"])
        del model
        assert seen() is None and engine() is None
        assert torch.cuda.memory_allocated() <= before
    finally:
        gc.enable()
    engine = ForceEngine(_model())                  # an engine of its own keeps its model
    assert engine.model is not None and engine.stands_for() is not None


@pytest.mark.parametrize("chunk_rows", [None, 3])
def test_a_profile_names_every_heavy_launch(chunk_rows):
    from mace_ictc import synthetic as S
    from mace_ictc.md import MolecularDynamics
    pos, box, species = S.jittered_lattice(9, 9, 9, 2.15, 0.1, 5)
    md = MolecularDynamics(_model(), pos, np.array(ELEMENTS)[species], box, chunk_rows=chunk_rows, stream_gates=True)
    md.engine.profile = profile = []
    md.compute_forces()
    torch.cuda.synchronize()
    names = [name for name, start, end in profile if start.elapsed_time(end) >= 0]
    chunks = 1 if chunk_rows is None else 243
    for layer, gates in ((0, 192), (1, 704)):
        assert names.count(f"graph_forward_l{layer}") == names.count(f"graph_adjoint_l{layer}") == chunks
        assert names.count(f"gate_gemm_backward_{gates}") == chunks
        assert names.count(f"gate_gemm_forward_{gates}") == (1 if chunk_rows is None else 2 * chunks)
        assert names.count(f"radial_mlp_hidden_backward_{gates}") == 1


def test_negative_numbers_index_the_species_table_as_in_the_forward():
    from mace_ictc.hp import energy_and_forces
    model = _model()
    graph = _graph(np.random.default_rng(4), (40,), False)
    graph[1][5], graph[1][6] = -1, -3                         # of a table of nine: 8 and 6
    _close(energy_and_forces(model, *graph), _autograd(model, graph))


@pytest.mark.parametrize("number", [7, 500, -2, -10])
def test_unknown_atoms_raise_without_input_validation(number):
    """The status word is read in any case: an unknown atom never counts as a known one."""
    from mace_ictc.hp import energy_and_forces
    model = _model()
    model.skip_input_validation = True
    graph = _graph(np.random.default_rng(4), (40,), False)
    graph[1][5] = number
    with pytest.raises(ValueError, match="atomic numbers"):
        energy_and_forces(model, *graph)


def test_traced_hooked_and_negated_calls_take_the_autograd_route():
    from mace_ictc.hp import energy_and_forces
    from torch.fx.experimental.proxy_tensor import make_fx
    model = _model()
    graph = _graph(np.random.default_rng(9), (30,), False)
    want = _autograd(model, graph)
    with pytest.raises((ValueError, RuntimeError)):         # tracing is refused, not recorded as a constant
        make_fx(lambda p: energy_and_forces(model, p, *graph[1:])["forces"])(graph[0])
    for k in (0, 5, 6):
        other = list(graph)
        other[k] = torch._neg_view(-graph[k].float())
        _close(energy_and_forces(model, *other), want)
    pinned = list(graph)                                    # an atom held in place by a hook on the positions
    pinned[0] = graph[0].clone().requires_grad_(True)
    pinned[0].register_hook(lambda g: g * (torch.arange(30, device="cuda") != 4).unsqueeze(1))
    got = energy_and_forces(model, *pinned)["forces"]
    assert bool((got[4] == 0).all()) and float((got[5:] - want["forces"][5:]).abs().max()) < TOL * float(want["forces"].abs().max())


@pytest.mark.parametrize("dtype", [torch.bool, torch.int32, torch.float64])
def test_engine_takes_masks_and_species_of_any_type_and_stride(dtype):
    from mace_ictc.engine import ForceEngine
    from ictc_o3.ops.topology import build_csr
    model = _model()
    pos, z, _, src, dst, shifts, cell = _graph(np.random.default_rng(6), (50,), False)
    order = torch.argsort(dst, stable=True)
    src, dst, shifts = src[order], dst[order], shifts[order].float()
    species, engine = model.species_index(z), ForceEngine(model)
    mask = torch.arange(50, device="cuda") % 3 != 1
    args = (src, dst, shifts, cell[0].diag().tolist(), 50, build_csr(dst, 50, True)[0])
    want = engine.energy_and_gradient(pos, species, *args, row_mask=mask.float())
    wide = torch.zeros(50, 2, dtype=dtype, device="cuda")
    wide[:, 0] = mask.to(dtype)
    got = engine.energy_and_gradient(pos, species.to(torch.int32), *args, row_mask=wide[:, 0])
    got2 = engine.energy_and_gradient(pos, species.repeat_interleave(2)[::2], *args, row_mask=mask.to(dtype))
    for other in (got, got2):
        assert torch.equal(other[1], want[1]) and torch.equal(other[2], want[2])
        assert abs(float(other[0] - want[0])) <= 1e-6 * abs(float(want[0]))


@pytest.mark.parametrize("chunk_rows", [None, 300])
def test_stages_around_a_ghost_exchange(chunk_rows):
    """One rank that owns the whole box and sees its periodic images as ghost rows: same forces as the periodic list."""
    from mace_ictc import synthetic as S
    from mace_ictc.md import MolecularDynamics
    model = _model()
    pos, box, species = S.jittered_lattice(8, 9, 7, 2.15, 0.1, 3)
    z = np.array(ELEMENTS)[species]
    whole = MolecularDynamics(model, pos, z, box, seed=2)
    want = whole.gather(whole.compute_forces())
    split = MolecularDynamics(model, pos, z, box, seed=2, skin=1.0, chunk_rows=chunk_rows, stream_gates=True)
    split.engine.chunk_margin = 12.0         # ghost rows have few edges, so a chunk of owned rows is far above the mean
    split._setup_distributed()
    split._forces_distributed()
    got = split.gather(split.forces)
    assert float((got - want).abs().max()) < TOL * float(want.abs().max())
    assert abs(float(split._dist["energy"]) - float(whole.energy)) < 1e-6 * abs(float(whole.energy))
    assert int(split.engine.overflow.item()) == 0
