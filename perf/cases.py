"""What is measured: the work a user has this framework do, through its public entry points.

Five paths, each with a small, an ordinary and (where the path has one) a large size:

* ``edges``    ``EdgeTensorProduct`` on edge rows (either layout), output and first derivatives;
* ``message``  ``PackedGraphMessage`` (gather, tensor product, receiver sum) on a neighbour graph, output alone
               (inference) or with the gradients of features, harmonics and gates;
* ``sc``       ``create_symmetric_contraction``: contraction per species, with the feature gradient and, in training,
               the weight gradients;
* ``model``    ``create_model`` / ``configure_model`` / ``energy_and_forces`` on graphs that the caller has built:
               energy and forces, or the training step (force loss, gradients of all parameters);
* ``md``       ``MolecularDynamics``: velocity-Verlet steps with the neighbour list rebuilt in every step, launched
               eagerly or replayed as a CUDA graph, gates whole or in chunks of rows.

Everything is float32, the only type the kernels have.  Inputs are the systems of ``bench.py``: uniform boxes of
0.1 atoms / A^3 for the message, jittered H/C/O lattices of 2.15 A spacing for the model, both with a 4.5 A cutoff.
"""
import math
import os
import sys

import numpy as np
import torch

_PACKAGES = os.path.join(os.getcwd(), "ictc-o3-hp-k100_b200")      # the packages ictc_o3 and mace_ictc
if _PACKAGES not in sys.path:
    sys.path.insert(1, _PACKAGES)

CUTOFF, DENSITY, SPACING, SIGMA = 4.5, 0.1, 2.15, 0.1
ELEMENTS = (1, 6, 8)
# compiled path sets: (input, edge, output degree) -> (paths, sum over paths of (2 l_in + 1)(2 l_out + 1))
PATHS = {(2, 2, 2): (11, 115), (0, 2, 2): (3, 9), (1, 1, 1): (4, 16), (2, 2, 0): (3, 9)}
SC_FMA = {0: (250, 230), 2: (2100, 1830)}     # multiply-adds per (node, channel): value, feature gradient


def listed():
    return [
        # one small batch of edges with 32 channels: a unit test, a small molecule, latency of a single operator
        {"name": "edges_257", "kind": "edges", "edges": 257, "channels": 32, "degrees": "222", "layout": "ir_mul"},
        # an operator inside a caller's own network that keeps [channel, component] rows; ragged edge count
        {"name": "edges_20011_mul_ir", "kind": "edges", "edges": 20011, "channels": 64, "degrees": "222",
         "layout": "mul_ir"},
        # message of one molecule-sized graph, output only: inference of a caller's own network
        {"name": "message_1501_forward", "kind": "message", "nodes": 1501, "channels": 64, "degrees": "222",
         "gradients": False},
        # message with all first derivatives at the size of a full simulation box (2.3 million edges)
        {"name": "message_65536", "kind": "message", "nodes": 65536, "channels": 64, "degrees": "222",
         "gradients": True},
        # contraction of a large node table, value and feature gradient: the force path
        {"name": "sc_262144", "kind": "sc", "nodes": 262144, "channels": 64, "target": 2, "elements": 4,
         "weights": False},
        # contraction to scalars with the weight gradients: the last layer of a network in training
        {"name": "sc_5003_weights", "kind": "sc", "nodes": 5003, "channels": 64, "target": 0, "elements": 3,
         "weights": True},
        # energy and forces of one small cell: geometry optimisation, a calculator called from a script
        {"name": "model_216", "kind": "model", "nx": 6, "ny": 6, "nz": 6, "graphs": 1, "channels": 64,
         "training": False, "sorted": False},
        # energies and forces of a batch of structures with edges that are already sorted by receiver
        {"name": "model_12x720", "kind": "model", "nx": 8, "ny": 9, "nz": 10, "graphs": 12, "channels": 64,
         "training": False, "sorted": True},
        # the training step on one large structure: force loss, mixed second derivatives, every parameter's gradient
        {"name": "train_32768", "kind": "model", "nx": 32, "ny": 32, "nz": 32, "graphs": 1, "channels": 64,
         "training": True, "sorted": False},
        # molecular dynamics of a small system, recorded: the latency-bound end of MD
        {"name": "md_1000", "kind": "md", "nx": 10, "ny": 10, "nz": 10, "steps": 10, "recorded": True, "chunk": 0},
        # molecular dynamics launched step by step (the default of the driver) on an ordinary, ragged box
        {"name": "md_13430_eager", "kind": "md", "nx": 23, "ny": 24, "nz": 25, "steps": 3, "recorded": False,
         "chunk": 0},
        # molecular dynamics at the size of one GPU's share of a large run, recorded
        {"name": "md_131072", "kind": "md", "nx": 64, "ny": 64, "nz": 32, "steps": 2, "recorded": True, "chunk": 0},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lattice(rng, lo, hi):
    """Sites per axis of a box with about lo..hi sites, axes of different lengths, none under 6 (two cutoffs)."""
    side = _log_uniform(rng, lo, hi) ** (1.0 / 3.0)
    nx = max(6, int(side * rng.uniform(0.8, 1.2)))
    ny = max(6, int(side * rng.uniform(0.8, 1.2)))
    return nx, ny, max(6, min(int(side ** 3 / (nx * ny)), hi // (nx * ny)))


def draw(rng):
    kind = rng.choice(("edges", "message", "sc", "model", "md"))
    if kind == "edges":
        return {"kind": kind, "edges": _log_uniform(rng, 100, 300000), "channels": rng.choice((32, 64, 64, 128)),
                "degrees": rng.choice(("222", "222", "111", "022")), "layout": rng.choice(("ir_mul", "mul_ir"))}
    if kind == "message":
        return {"kind": kind, "nodes": _log_uniform(rng, 1000, 65536), "channels": rng.choice((32, 64, 64)),
                "degrees": rng.choice(("222", "222", "022", "220")), "gradients": rng.random() < 0.6}
    if kind == "sc":
        target, weights = rng.choice((0, 2)), rng.random() < 0.4
        elements = rng.choice((1, 2, 3, 4, 8))
        return {"kind": kind, "nodes": _log_uniform(rng, 200, 65536 if weights else 262144),
                "channels": rng.choice((32, 64, 64)), "target": target, "elements": elements, "weights": weights}
    if kind == "model":
        training = rng.random() < 0.5
        graphs = rng.choice((1, 1, 4, 16))
        nx, ny, nz = _lattice(rng, 216, max(400, 30000 // graphs))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "graphs": graphs, "channels": rng.choice((32, 64, 64)),
                "training": training, "sorted": rng.random() < 0.5}
    recorded = rng.random() < 0.6
    nx, ny, nz = _lattice(rng, 300, 120000 if recorded else 60000)
    atoms = nx * ny * nz
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": rng.randint(5, 12) if atoms < 5000 else 2,
            "recorded": recorded, "chunk": -(-atoms // 5) if atoms > 5000 and rng.random() < 0.4 else 0}


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32)


def _degrees(case):
    return tuple(int(d) for d in case["degrees"])


def _directions(gen, vectors, top):
    from ictc_o3 import direction_harmonics
    unit = vectors / vectors.norm(dim=1, keepdim=True)
    return torch.cat(direction_harmonics(unit.contiguous(), top), -1).contiguous()


def _prepare_edges(case, seed):
    from ictc_o3 import EdgeTensorProduct
    gen = _generator(seed)
    lin, ledge, lout = _degrees(case)
    e, c = case["edges"], case["channels"]
    op = EdgeTensorProduct.create(input_lmax=lin, edge_lmax=ledge, output_lmax=lout, channels=c, layout=case["layout"])
    sh = _directions(gen, _normal(gen, e, 3), ledge)
    leaves = [_normal(gen, e, c * (lin + 1) ** 2), sh, _normal(gen, e, op.gate_width)]
    return {"op": op, "leaves": [t.requires_grad_(True) for t in leaves], "cotangent": _normal(gen, e, op.output_width)}


def _message_edges(nodes):
    return int(0.92 * nodes * DENSITY * 4.0 / 3.0 * math.pi * CUTOFF ** 3)


def _uniform_graph(gen, nodes):
    """Atoms at uniform random places of a periodic cube, sorted by cells of the cutoff's size as an MD code keeps
    them, and their neighbour list (sorted by receiver) with the edge vectors.  The list is thinned at random to a
    number of edges that depends on the number of nodes alone, so that the outputs of all seeds have one shape."""
    from mace_ictc.md import neighbor_list
    box = (nodes / DENSITY) ** (1.0 / 3.0)
    pos = torch.rand(nodes, 3, generator=gen, device="cuda") * box
    cells = max(1, int(box // CUTOFF))
    at = (pos * (cells / box)).long().clamp(max=cells - 1)
    pos = pos[torch.argsort((at[:, 0] * cells + at[:, 1]) * cells + at[:, 2], stable=True)].contiguous()
    src, dst, shifts, _ = neighbor_list(pos, nodes, [0, 0, 0], [box] * 3, [box] * 3, (1, 1, 1), CUTOFF)
    count = src.numel()
    keep = torch.randperm(count, generator=gen, device="cuda")[:_message_edges(nodes)].sort().values
    src, dst, shifts = src[keep], dst[keep], shifts[keep]
    return src, dst, pos[dst] - pos[src] + shifts * box


def _gates(vectors, width, seed):
    from mace_ictc import synthetic
    r = vectors.norm(dim=1)
    weights = synthetic.random_radial_mlp([8, 64, 64, 64, width], seed, "cuda")
    return torch.cat([synthetic.radial_gates(synthetic.bessel_basis(part, CUTOFF), weights)
                      for part in r.split(262144)], 0)


def _prepare_message(case, seed):
    from ictc_o3 import PackedGraphMessage
    gen = _generator(seed)
    lin, ledge, lout = _degrees(case)
    n, c = case["nodes"], case["channels"]
    op = PackedGraphMessage.create(channels=c, input_lmax=lin, edge_lmax=ledge, output_lmax=lout)
    src, dst, vectors = _uniform_graph(gen, n)
    leaves = [_normal(gen, n, c * (lin + 1) ** 2), _directions(gen, vectors, ledge), _gates(vectors, op.gate_width, seed)]
    if not case["gradients"]:
        return {"op": op, "leaves": leaves, "src": src, "dst": dst}
    return {"op": op, "leaves": [t.requires_grad_(True) for t in leaves], "src": src, "dst": dst,
            "cotangent": _normal(gen, n, op.output_width)}


def _prepare_sc(case, seed):
    from ictc_o3 import create_symmetric_contraction
    gen = _generator(seed)
    torch.manual_seed(seed)
    n, c = case["nodes"], case["channels"]
    op = create_symmetric_contraction(num_elements=case["elements"], lmax=2, target_lmax=case["target"], channels=c,
                                      training=case["weights"])
    op.requires_grad_(case["weights"])
    return {"op": op, "x": _normal(gen, n, 9 * c).requires_grad_(True),
            "species": torch.randint(case["elements"], (n,), generator=gen, device="cuda"),
            "cotangent": _normal(gen, n, c * (case["target"] + 1) ** 2),
            "weights": list(op.parameters()) if case["weights"] else []}


def _prepare_model(case, seed):
    from mace_ictc import synthetic
    from mace_ictc.hp import configure_model, create_model
    from mace_ictc.md import neighbor_list
    gen = _generator(seed)
    torch.manual_seed(seed)
    model = create_model(channels=case["channels"], lmax=2, cutoff=CUTOFF, atomic_numbers=ELEMENTS,
                         avg_num_neighbors=32.0)
    configure_model(model, policy="generated", training=case["training"], preserve_edge_order=case["sorted"],
                    skip_input_validation=case["sorted"])
    parts, atoms = [], case["nx"] * case["ny"] * case["nz"]
    for g in range(case["graphs"]):
        pos, box, species = synthetic.jittered_lattice(case["nx"], case["ny"], case["nz"], SPACING, SIGMA,
                                                       1000 * seed + g)
        pos = torch.as_tensor(pos).cuda()
        src, dst, shifts, _ = neighbor_list(pos, atoms, [0, 0, 0], list(box), list(box), (1, 1, 1), CUTOFF)
        parts.append((pos, torch.as_tensor(np.asarray(ELEMENTS)[species]).cuda(), src + g * atoms, dst + g * atoms,
                      shifts, torch.full((atoms,), g, dtype=torch.long, device="cuda"),
                      torch.as_tensor(np.diag(box), dtype=torch.float32).cuda()))
    pos, z, src, dst, shifts, batch = (torch.cat(p, 0) for p in list(zip(*parts))[:6])
    return {"model": model, "training": case["training"], "atoms": atoms,
            "graph": (pos, z, batch, src, dst, shifts, torch.stack([p[6] for p in parts])),
            "target": 0.05 * _normal(gen, pos.shape[0], 3)}


def _prepare_md(case, seed):
    from mace_ictc import synthetic
    from mace_ictc.hp import create_model
    from mace_ictc.md import MolecularDynamics
    torch.manual_seed(seed)
    model = create_model(channels=64, lmax=2, cutoff=CUTOFF, atomic_numbers=ELEMENTS, avg_num_neighbors=32.0)
    pos, box, species = synthetic.jittered_lattice(case["nx"], case["ny"], case["nz"], SPACING, SIGMA, seed)
    options = {"chunk_rows": case["chunk"], "stream_gates": True} if case["chunk"] else {}
    md = MolecularDynamics(model, pos, np.asarray(ELEMENTS)[species], box, dt=1.0, temperature=300.0, seed=seed,
                           **options)
    md.compute_forces()
    if case["recorded"]:
        md.enable_graph()
    return {"md": md, "steps": case["steps"], "start": (md.pos.clone(), md.vel.clone(), md.forces.clone())}


def prepare(case, seed):
    return {"kind": case["kind"], **globals()["_prepare_" + case["kind"]](case, seed)}


# ------------------------------------------------------------------------------------------------ one pass
def _run_edges(s):
    out = s["op"](*s["leaves"])
    return [out.detach(), *torch.autograd.grad(out, s["leaves"], s["cotangent"])]


def _run_message(s):
    if "cotangent" not in s:
        with torch.no_grad():
            return s["op"](*s["leaves"], s["src"], s["dst"])
    out = s["op"](*s["leaves"], s["src"], s["dst"])
    return [out.detach(), *torch.autograd.grad(out, s["leaves"], s["cotangent"])]


def _run_sc(s):
    out = s["op"](s["x"], None, s["species"])
    return [out.detach(), *torch.autograd.grad(out, [s["x"], *s["weights"]], s["cotangent"])]


def _run_model(s):
    from mace_ictc.hp import energy_and_forces
    got = energy_and_forces(s["model"], *s["graph"], training=s["training"])
    if not s["training"]:
        return got
    model = s["model"]
    model.zero_grad(set_to_none=True)
    loss = (got["energy"] / s["atoms"]).square().mean() + (got["forces"] - s["target"]).square().mean()
    loss.backward()
    return {"loss": loss.detach(), "energy": got["energy"].detach(), "forces": got["forces"].detach(),
            "gradients": {name: p.grad for name, p in model.named_parameters() if p.grad is not None}}


def _run_md(s):
    """A short run from the saved start (a restart file, a new replica), read out in the caller's atom order."""
    md = s["md"]
    for now, start in zip((md.pos, md.vel, md.forces), s["start"]):
        now.copy_(start)
    md.run(s["steps"])
    return {"energy": md.energy.detach(), "positions": md.gather(md.pos), "velocities": md.gather(md.vel),
            "forces": md.gather(md.forces)}


def run(state):
    return globals()["_run_" + state["kind"]](state)


# ------------------------------------------------------------------------------------------------ work, tolerance
def _tp_work(rows_in, edges, rows_out, c, degrees, gradients):
    lin, ledge, lout = degrees
    paths, fma = PATHS[degrees]
    slots = {(2, 2, 2): 35, (0, 2, 2): 9, (1, 1, 1): 8, (2, 2, 0): 3}[degrees]
    inputs = rows_in * c * (lin + 1) ** 2 + edges * ((ledge + 1) ** 2 + paths * c)
    output = rows_out * slots * c
    floats = inputs + output + ((output + inputs) if gradients else 0)
    return {"bytes": 4 * floats, "flops": edges * c * 2 * (fma + paths) * (4 if gradients else 1)}


def work(case):
    kind = case["kind"]
    if kind == "edges":
        e = case["edges"]
        return _tp_work(e, e, e, case["channels"], _degrees(case), True)
    if kind == "message":
        n = case["nodes"]
        edges = _message_edges(n)
        got = _tp_work(n, edges, n, case["channels"], _degrees(case), case["gradients"])
        got["bytes"] += 16 * edges
        return got
    if kind == "sc":
        n, c, ny = case["nodes"], case["channels"], (case["target"] + 1) ** 2
        value, gradient = SC_FMA[case["target"]]
        flops = 2 * (value + gradient + (value if case["weights"] else 0))
        return {"bytes": 4 * n * (c * (9 + ny + 9 + ny) + 2), "flops": n * c * flops}
    atoms = case["nx"] * case["ny"] * case["nz"] * case.get("graphs", 1)
    edges, c = 32 * atoms, case.get("channels", 64)
    # per pair of edges: the radial networks of both layers; per atom: channel linears and contractions
    linear = 2 * (edges // 2 * (2 * (8 * 64 + 2 * 64 * 64) + 64 * 14 * c) + atoms * c * c * (10 + 44 + 10 + 2))
    product = edges * c * 2 * (9 + 3 + 115 + 11) + atoms * c * 2 * (SC_FMA[0][0] + SC_FMA[2][0])
    if kind == "model" and case["training"]:
        return {"bytes": 28 * edges + 48 * atoms, "flops": 6 * linear + 12 * product}
    flops = 2 * linear + 4 * product
    if kind == "model":
        return {"bytes": 28 * edges + 36 * atoms, "flops": flops}
    return {"bytes": 72 * atoms * case["steps"], "flops": flops * case["steps"]}


def tolerance(case):
    kind = case["kind"]
    if kind in ("edges", "message", "sc"):
        return {"rel": 1e-5}                      # one operator: 32-bit sums of products
    if kind == "model" and case["training"]:
        return {"rel": 5e-5}                      # derivatives of forces: four sweeps through two layers in 32 bits
    return {"rel": 2e-5}                          # forces: two sweeps through two layers in 32 bits
