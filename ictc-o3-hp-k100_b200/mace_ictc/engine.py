"""Force engine: energy and position gradient of the MACE-ICTC model by an explicit forward and reverse
sweep over the B200 kernels, without the autograd tape.

Same arithmetic as ``MaceIctcModel.forward`` followed by ``autograd.grad(E, pos)``
(reference: mace_ictc/hp/runtime.py:82-111 over mace_ictc/models/mace/backbone.py:860-1246), specialised to
what an MD step and an energy-and-forces call need: frozen weights, gradient with respect to positions only.  The
launch sequence is native (``csrc/sweep.cu``); this module lays the weights out for it, sizes the workspace and
calls it, once, or stage by stage where ghost rows are exchanged in between.  Tests compare it with the autograd path.
Node features live in ir_mul rows ([rows, 9C], degree blocks [2l+1, C]) from end to end, so channel
linears are GEMMs over contiguous rows and no mul_ir <-> ir_mul conversion is made.

Gates are streamed (reference: ictc_o3/ops/streamed_gate_message.py:112-116, 193-221; chunk sizes
mace_ictc/interfaces/lammps_hp.py:163-172).  The per-edge gate table [E, P*C] and its gradient are the largest
tensors of the step, so the sweeps can run over chunks of owner rows (``chunk_rows``): the forward produces the
gates of a chunk's edges from the 64-wide hidden state, consumes them and reuses the buffer; the reverse sweep
recomputes the chunk's gates, lets the tensor-product adjoint write the chunk's gate gradients and contracts
them back to the hidden width at once.  No tensor wider than 64 floats per edge outlives a chunk.  Without
chunking the gate table of the (edge, reverse edge) pairs is kept for both sweeps and only the gate gradient is
per edge.  Both modes run the same arithmetic per edge in the same order, so their results agree bit for bit (the energy of
one graph included; those of a batch are added up with double-precision atomics).
"""
from __future__ import annotations

import ctypes as C
import math
import threading
import weakref

import torch

from ictc_o3 import _lib, tables
from ictc_o3.basis.ictd_irreps import EdgeWeightedPathPreservingTensorProduct
from ictc_o3.operators import EdgeTensorProduct, PackedGraphMessage
from ictc_o3.ops.topology import build_csr
from ictc_o3.symmetric_contraction import ICTDBridgeUSymmetricContractionSO3, _Contraction, _Contractions
from .model import (ElementConditionedLinearSO3, EquivariantChannelLinearSO3, InteractionBlock, MaceIctcModel, MLPReadout,
                    Normalize2MomSiLU, PathPreservingLinearSO3, ProductBlock, ScalarReadout)

_ALL, _STAGES = 31, (1, 2, 4, 8, 16)
_LABELS = ("radial_mlp_hidden_forward_{nout}", "gate_gemm_forward_{nout}", "graph_forward_l{layer}",
           "graph_adjoint_l{layer}", "gate_gemm_backward_{nout}", "radial_mlp_hidden_backward_{nout}",
           "channel_linear_tc", "symmetric_contraction_l{layer}")
_WATCH_WORDS = 2048      # words of a parameter that one block of the sweep compares
_HOOKS = ("_forward_hooks", "_forward_pre_hooks", "_backward_hooks", "_backward_pre_hooks")
_GLOBAL_HOOKS = ("_global_forward_hooks", "_global_forward_pre_hooks", "_global_backward_hooks", "_global_backward_pre_hooks")
_local = threading.local()


def _linear(module, rows, cols, bias=False):
    """A Linear of this shape (rows None: any) and nothing else; without a bias where the bias would count."""
    return (type(module) is torch.nn.Linear and (bias or module.bias is None) and module.weight.shape[1] == cols
            and (rows is None or module.weight.shape[0] == rows))


def _table(params, degrees, shape_of):
    return type(params) is torch.nn.ParameterDict and all(
        str(l) in params and tuple(params[str(l)].shape) == shape_of(l) for l in degrees)


def _has(module, kind, **attributes):
    return type(module) is kind and all(getattr(module, k, None) == v for k, v in attributes.items())


def covers(m):
    """Is every module at its place the one whose forward the sweep reproduces, with the shapes that the layout reads and
    nothing (a bias, another activation, a further output) that it does not read?"""
    c, species = 64, getattr(m, "num_elements", None)
    if not (isinstance(m, MaceIctcModel) and type(m).forward is MaceIctcModel.forward and _has(m, type(m), channels=c, lmax=2, num_interaction=2)
            and _linear(m.node_embedding, c, species, bias=True)
            and all(_has(x, torch.nn.ModuleList) for x in (m.interactions, m.products, m.layer_energy_readouts))
            and len(m.interactions) == len(m.products) == 2 and len(m.layer_energy_readouts) >= 1):
        return False
    first, last = m.layer_energy_readouts[0], m.last_layer_energy_readout
    if not (_has(first, ScalarReadout, channels=c) and _linear(first.readout, 1, c)
            and _has(last, MLPReadout) and _linear(last.linear_1, None, c) and _has(last.activation, Normalize2MomSiLU)
            and _linear(last.linear_2, 1, last.linear_1.weight.shape[0])):
        return False
    for inter, prod, l_in, l_out in zip(m.interactions, m.products, (0, 2), (2, 0)):
        if not (_has(inter, InteractionBlock, channels=c, lmax=2, input_lmax=l_in, sc_lmax=0)
                and _has(inter.tp, EdgeWeightedPathPreservingTensorProduct, channels=c, internal_compute_dtype=torch.float32)
                and [tuple(path) for path in inter.tp.paths] == tables.natural_paths(l_in, 2, 2)
                and tuple(inter.tp.weight.shape) == (len(inter.tp.paths), c)):
            return False
        op = inter._message                    # made by the first forward of the model
        if op is not None and not (type(op) is PackedGraphMessage and type(op.edge) is EdgeTensorProduct and op.tp is inter.tp):
            return False
        if not (_has(inter.fc, torch.nn.Sequential) and len(inter.fc) == 7
                and all(_has(inter.fc[k], Normalize2MomSiLU) for k in (1, 3, 5))
                and all(_linear(inter.fc[k], *shape) for k, shape in
                        ((0, (64, m.number_of_basis)), (2, (64, 64)), (4, (64, 64)), (6, (inter.tp.num_paths * c, 64))))):
            return False
        up, ml, sc = inter.linear_up, inter.message_linear, inter.self_connection
        if not (_has(up, EquivariantChannelLinearSO3, channels=c, lmax=l_in) and _has(up.adapters, torch.nn.ModuleDict)
                and all(str(l) in up.adapters and _linear(up.adapters[str(l)], c, c, bias=True) for l in range(l_in + 1))
                and _has(ml, PathPreservingLinearSO3, out_channels=c, lmax=2)
                and _table(ml.weights, range(3), lambda l: (c, c * inter.tp.path_counts_by_l[l]))
                and _has(sc, ElementConditionedLinearSO3, channels=c, lmax=0, num_elements=species)
                and _table(sc.weights, (0,), lambda l: (species, c, c))):
            return False
        con = prod.symmetric_contractions if _has(prod, ProductBlock, channels=c, lmax=2, target_lmax=l_out) else None
        if not (_has(con, ICTDBridgeUSymmetricContractionSO3, channels=c, lmax=2, target_lmax=l_out, num_elements=species,
                     ir_mul=False)
                and _has(con.symmetric_contractions, _Contractions)
                and all(_has(x, _Contraction) for x in con.symmetric_contractions.contractions)
                and _table(prod.linear, range(l_out + 1), lambda l: (c, c))):
            return False
    return True


class _Weights:
    """The sweep's view of one state of the parameters: packed operands and the struct that points at them."""


class ForceEngine:
    """``chunk_rows``: owner rows per chunk of the streamed gate evaluation (None: one pass over everything).
    ``chunk_margin``: a chunk buffer holds ``chunk_rows x mean degree x chunk_margin`` edges; a chunk with more
    edges than that raises ``overflow`` (device flag) and its surplus edges are dropped, never written out of
    bounds.  ``stream_gates``: see the attribute.  ``owned``: the model keeps this engine, which then holds no reference to it
    (a cycle would keep the laid-out weights of a deleted model until the next garbage collection)."""

    def __init__(self, model: MaceIctcModel, chunk_rows: int | None = None, chunk_margin: float = 1.3,
                 stream_gates: bool | None = None, lay_out: bool = True, owned: bool = False):
        if len(model.interactions) != 2:
            raise ValueError("the force engine covers the two-interaction model")
        if model.channels != 64:
            raise ValueError("the force engine runs on the 64-channel tensor-core kernels; other widths use the "
                             "autograd route (MolecularDynamics(..., use_engine=False))")
        self._model, self._held = weakref.ref(model), None if owned else model
        self.c = model.channels
        self.dev = next(model.parameters()).device
        self.lib = _lib.load()
        self._weights = None
        self._watched = None
        self._fit = None         # (state of the model, do its sizes fit the sweep?)
        self.chunk_rows = None if chunk_rows is None else int(chunk_rows)
        self.chunk_margin = float(chunk_margin)
        # with chunks: True = the gates are streamed too (produced per chunk in the forward sweep, recomputed per chunk
        # in the reverse sweep: nothing of size [E, P*C] exists); False = the gate table of the edge pairs is kept whole
        # and only the gate GRADIENT, the largest tensor, lives per chunk (half the GEMM work of streaming);
        # None = keep the table while both layers' tables take less than 40 % of the device memory
        self.stream_gates = stream_gates
        self.overflow = torch.zeros(1, dtype=torch.int32, device=self.dev)   # sticky: a chunk buffer was too small
        self.profile = None      # list of (kernel name, start event, end event) when enabled by a benchmark
        self._bounds = {}
        if lay_out:
            self.refresh()

    @property
    def model(self) -> MaceIctcModel:
        return self._model()

    # ---------------------------------------------------------------- weights
    def _watch(self):
        """Every module and parameter slot of the model with what it holds now: a replaced one is noticed by identity, a new
        one by the size of its table."""
        slots, sizes, modules = [], [], list(self.model.modules())
        for module in modules:
            for table in (module._modules, module._parameters, module._buffers):
                sizes.append((table, len(table)))
                slots.extend((table, key, value) for key, value in table.items())
        params = list(self.model.parameters())
        inter = list(self.model.interactions)
        hooks = [module.__dict__[name] for module in modules for name in _HOOKS]
        own = [module.__dict__ for module in modules[1:]]           # without the model's own, where this engine may be kept
        return slots, sizes, params, inter, covers(self.model), own, hooks

    def _state(self):
        params, inter = self._watched[2:4]
        m = self.model
        return ([(p._version, p.data_ptr()) for p in params], [i.avg_num_neighbors for i in inter], m.max_radius,
                m.polynomial_cutoff_p, m.number_of_basis)

    def stands_for(self):
        """Does the sweep compute what the model's own ``forward`` would?  Not with hooks, with other modules than those it was
        written for (``covers``), with a replaced ``forward``, with base coefficients that still require grad, or with other
        widths.  Returns the state of the model for ``energy_and_forces``, or None."""
        if self._watched is None or self._replaced():
            self._watched, self._weights, self._fit = self._watch(), None, None
        _, _, _, inter, covered, own, hooks = self._watched
        table = torch.nn.modules.module
        if (not covered or any(getattr(table, name) for name in _GLOBAL_HOOKS) or any(hooks)
                or "forward" in self.model.__dict__ or any("forward" in d for d in own) or any(i.tp.weight.requires_grad for i in inter)):
            return None
        state, fit = self._state(), self._fit
        if fit is None or fit[0] != state:
            fit = self._fit = state, self._sizes_fit()
        return state if fit[1] else None

    def _sizes_fit(self):
        m, index = self.model, self.model.atomic_number_to_index
        return (type(m.number_of_basis) is int and 1 <= m.number_of_basis <= 8 and type(m.polynomial_cutoff_p) is int
                and m.polynomial_cutoff_p >= 2 and m.max_radius > 0 and index.dtype == torch.int64 and index.device == self.dev
                and index.is_contiguous() and all(p.dtype == torch.float32 and p.device == self.dev for p in self._watched[2]))

    def _replaced(self):
        return (any(table.get(key) is not value for table, key, value in self._watched[0])
                or any(len(table) != size for table, size in self._watched[1]))

    def refresh(self, state=None):
        """(Re)build the GEMM-ready weight views when a parameter changed.  ``state``: what ``stands_for`` has just found."""
        if state is None:
            if self._watched is None or self._replaced():
                self._watched, self._weights, self._fit = self._watch(), None, None
            state = self._state()
        w, stream = self._weights, torch.cuda.current_stream(self.dev)
        if w is None or w.state != state:
            with _lib.on_device(self.dev):
                w = self._layout()
                w.event = torch.cuda.Event()
                w.event.record(stream)
            w.state, w.streams = state, {stream.cuda_stream}
            self._weights = w
        elif stream.cuda_stream not in w.streams and not torch.cuda.is_current_stream_capturing():
            # laid out on another stream: wait for that, and keep the memory until this stream is done with it
            stream.wait_event(w.event)
            for t in w.keep:
                t.record_stream(stream)
            w.streams.add(stream.cuda_stream)
        return w

    def _layout(self):
        m, c, w = self.model, self.c, _Weights()
        if any(p.dtype != torch.float32 or p.device != self.dev for p in self._watched[2]):
            raise ValueError("the force engine needs float32 parameters on one CUDA device")
        if not self._watched[4] or not self._sizes_fit():
            raise ValueError("the force engine reproduces the forward of the stock model with a radial MLP num_basis (<= 8) -> 64 "
                             "-> 64 -> 64 -> P*C and readouts without biases; a model with other modules runs on the "
                             "autograd route (MolecularDynamics(..., use_engine=False))")
        w.keep, w.struct = [], _lib.Sweep()

        def hold(t):
            w.keep.append(t)
            return t.data_ptr()

        with torch.no_grad():
            emb = m.node_embedding.weight.t()                                            # [S, C]
            w.nout = []
            for k, (inter, prod) in enumerate(zip(m.interactions, m.products)):
                fc = [mod.weight.contiguous() for mod in inter.fc if isinstance(mod, torch.nn.Linear)]
                L = w.struct.layer[k]
                L.w0 = hold(fc[0])
                L.hid = (hold(self._pack(fc[1], 0)), hold(self._pack(fc[2], 0)))
                L.hid_t = (hold(self._pack(fc[1], 1)), hold(self._pack(fc[2], 1)))
                L.w3, L.w3t = hold(self._pack(fc[3], 0)), hold(self._pack(fc[3], 1))
                L.num_gates = fc[3].shape[0]
                w.nout.append(fc[3].shape[0])
                L.path_weight = None if bool(torch.all(inter.tp.weight == 1)) else hold(inter.tp.weight.contiguous())
                L.slots = tuple(inter.tp.path_counts_by_l[l] for l in range(3))
                L.bank = hold(prod.symmetric_contractions.weight_bank())
                ml = [inter.message_linear.weights[str(l)] / max(inter.avg_num_neighbors, 1e-8) for l in range(3)]
                L.ml = tuple(hold(self._pack_lin(v, v.t())) for v in ml)                 # x @ ml^T
                L.ml_b = tuple(hold(self._pack_lin(v.t(), v)) for v in ml)               # x @ ml
                if k == 0:
                    pl = [prod.linear[str(l)] / math.sqrt(c) for l in range(3)]
                    L.pl = tuple(hold(self._pack_lin(v.t(), v)) for v in pl)             # x @ pl
                    L.pl_b = tuple(hold(self._pack_lin(v, v.t())) for v in pl)           # x @ pl^T
                else:
                    up = [inter.linear_up.adapters[str(l)].weight for l in range(3)]
                    L.up = tuple(hold(self._pack_lin(v, v.t())) for v in up)             # x @ up^T
                    L.up_b = tuple(hold(self._pack_lin(v.t(), v)) for v in up)           # x @ up
            # products of weights alone; in double precision, rounded once
            d = lambda t: t.double()                                                     # noqa: E731
            first, last = m.interactions
            s = w.struct
            s.up0_table = hold((d(emb) @ d(first.linear_up.adapters["0"].weight).t()).float().contiguous())
            s.sc0_table = hold(torch.einsum("si,soi->so", d(emb), d(first.self_connection.weights["0"])).float().contiguous())
            ro = m.last_layer_energy_readout
            w1 = d(ro.linear_1.weight)                                                   # [H, C]
            s.readout_rp = hold((w1 @ d(m.products[1].linear["0"]).t() / math.sqrt(c)).float().contiguous())
            s.readout_rs = hold(torch.einsum("ho,soi->shi", w1, d(last.self_connection.weights["0"])).float().contiguous())
            s.readout_w2 = hold(ro.linear_2.weight.reshape(-1).contiguous())
            # a copy: read two floats at a time, and a parameter may stand at any word of a flattened buffer
            s.readout_ro0 = hold(m.layer_energy_readouts[0].readout.weight.reshape(-1).clone())
            s.hidden, s.num_species = w1.shape[0], m.num_elements
            s.num_basis, s.poly_p, s.r_max = m.number_of_basis, m.polynomial_cutoff_p, m.max_radius
            w.tiles, w.copy = self._snapshot(w.keep)
            s.species_table, s.species_table_size = hold(m.atomic_number_to_index), m.atomic_number_to_index.numel()
        return w

    def _snapshot(self, keep):
        """The parameters' words as they are now, in pieces, and where each piece stands: the sweep of a call with the
        caller's own graph compares them, since a write through ``parameter.data`` changes neither address nor version."""
        table, flat = [], []
        for p in self._watched[2]:
            if not p.is_contiguous():
                return None, None                     # laid out anew on every call
            words = p.detach().reshape(-1)
            pieces = (words.numel() + _WATCH_WORDS - 1) // _WATCH_WORDS
            table += [(p.data_ptr() + 4 * _WATCH_WORDS * k, min(_WATCH_WORDS, words.numel() - _WATCH_WORDS * k))
                      for k in range(pieces)]
            flat.append(torch.nn.functional.pad(words, (0, pieces * _WATCH_WORDS - words.numel())))
        tiles, copy = torch.tensor(table, dtype=torch.int64, device=self.dev), torch.cat(flat)
        keep += [tiles, copy]
        return tiles, copy

    def _pack(self, w, transpose):
        """A [rows, 64] matrix in the shared-memory operand layout of the tcgen05 kernels."""
        out = torch.empty(2 * w.numel(), dtype=torch.float32, device=w.device)
        with _lib.on_device(w.device):
            _lib.check(self.lib.ictc_gate_pack_weights(w.shape[0], w.data_ptr(), transpose, out.data_ptr(),
                                                       _lib.stream(w.device)), "gate_pack_weights")
        return out

    def _pack_lin(self, w_out_major, w_in_major):
        """Operand copy for out = x @ w_in_major, where w_in_major is [K, N] and w_out_major its transpose."""
        k, n = w_in_major.shape
        if k == 64:
            return self._pack(w_out_major.contiguous(), 0)
        if n != 64:
            raise ValueError("tensor-core channel linear needs a 64-wide side")
        return self._pack(w_in_major.contiguous(), 1)

    # ---------------------------------------------------------------- buffers
    @staticmethod
    def bucket(rows):
        """Row count rounded up to 1/16 of its power of two.  Edge and atom counts change a little every MD step;
        allocating the rounded size keeps the sizes repeating, so the caching allocator reuses its blocks
        instead of splitting, freeing and re-allocating multi-GB segments."""
        rows = int(rows)
        if rows <= 4096:
            return 4096
        g = 1 << (rows.bit_length() - 5)
        return (rows + g - 1) // g * g

    def _streaming(self, table_rows):
        """Are the gates streamed per chunk (True) or is the table of ``table_rows`` rows kept for both sweeps?"""
        if self.stream_gates is not None:
            return bool(self.stream_gates)
        total = torch.cuda.get_device_properties(self.dev).total_memory
        return 4 * table_rows * sum(self.refresh().nout) > 0.4 * total

    def _chunk_capacity(self, rows, rowptr, edges):
        """Edge capacity of a chunk buffer of a sweep over ``rows`` owner rows (0: one pass over everything); also raises
        the device-side overflow flag when a chunk holds more edges than the buffer."""
        if self.chunk_rows is None or self.chunk_rows >= rows:
            return 0
        step = self.chunk_rows
        key = (rows, step)
        if key not in self._bounds:        # built outside any stream capture: the first call is a warm-up step
            bounds = list(range(0, rows, step)) + [rows]
            self._bounds[key] = torch.tensor(bounds, dtype=torch.int64, device=self.dev)
        cap = self.bucket(int(step * (edges / max(rows, 1)) * self.chunk_margin) + 1024)
        cuts = rowptr.index_select(0, self._bounds[key])
        self.overflow.logical_or_(((cuts[1:] - cuts[:-1]) > cap).any())
        return cap

    # ---------------------------------------------------------------- the sweep
    def _run(self, s, w, plan):
        """Workspace, then the launch sequence: at once, or stage by stage around the exchanges of ``plan``."""
        need = int(self.lib.ictc_sweep_workspace(C.byref(s)))
        if need < 0:
            raise RuntimeError(f"ictc_sweep_workspace: {_lib.last_error()}")
        if not torch.cuda.is_current_stream_capturing():
            need = self.bucket(need >> 8) << 8
        work = torch.empty(need, dtype=torch.uint8, device=self.dev)
        s.work, s.work_bytes = work.data_ptr(), need
        counts = (C.c_int64 * 2)()
        s.host_counts = C.addressof(counts)
        if self.profile is not None:
            # room for every timed launch: some 40 of a sweep, per chunk and interaction two receiver and three sender launches
            chunks = 1 if not s.chunk_rows else -(-max(s.n_owned, s.n_local) // s.chunk_rows)
            marks = 64 + 10 * chunks
            events = [torch.cuda.Event(enable_timing=True) for _ in range(2 * marks)]
            for e in events:
                e.record()
            handles = (C.c_void_p * (2 * marks))(*[e.cuda_event for e in events])
            labels = (C.c_int64 * marks)()
            s.host_marks, s.host_marks_capacity, s.host_mark_labels = C.addressof(handles), marks, C.addressof(labels)
        st = _lib.stream(self.dev)

        def stages(mask):
            _lib.check(self.lib.ictc_sweep_run(C.byref(s), mask, st), "ictc_sweep_run")

        if plan is None:
            stages(_ALL)
        else:
            n, feats, grads = s.n_owned, plan.features, plan.feature_grad
            stages(_STAGES[0])
            halo = plan.exchange.forward_async(feats[:n])         # the ghost rows travel while the hidden state is computed
            stages(_STAGES[1])
            feats[n:] = halo()
            stages(_STAGES[2])
            halo = plan.exchange.adjoint_async(grads[n:].contiguous())      # and back while the radial MLP is differentiated
            stages(_STAGES[3])
            grads[:n] += halo()
            stages(_STAGES[4])
        _lib.CALLS += int(counts[0])
        if self.profile is not None:
            for k in range(int(counts[1])):
                kind, layer = divmod(int(labels[k]), 2)
                self.profile.append((_LABELS[kind].format(layer=layer, nout=w.nout[layer]), events[2 * k], events[2 * k + 1]))

    @torch.no_grad()
    def energy_and_gradient(self, pos, species, src, dst, shifts, box, n_owned, dst_rowptr, plan=None, n_rows=None,
                            pairs=None, row_mask=None, src_csr=None, out=None, sign=1.0):
        """pos [N_local,3] (owned rows first), species [N_local] (index), edges sorted by receiver with all
        receivers < n_owned, dst_rowptr [n_owned+1].  Returns (energy of owned atoms, dE/dpos [N_local,3],
        per-atom energies [n_owned]).  ``n_rows`` < N_local marks trailing rows of ``pos`` as padding: they may
        be named by inert edges (whose sender index is then outside the sender CSR) but carry no features.
        ``pairs`` = (gate_row [E], rep_edge [U], other_edge [U]) evaluates the radial MLP once per edge pair; an
        optional fourth element is a device int64 scalar with the number of pair rows in use when U is a capacity.
        ``plan`` (an exchange plan of ``mace_ictc.domain``) refreshes the ghost rows between the interactions.
        ``row_mask`` [n_owned] (0 / 1) leaves padding rows among the owned rows out of the energy (and hence of
        the gradient: a padding row has no edges).  ``src_csr`` = (row offsets, edge ids) of the senders where the caller
        has them.  ``out`` = (energy [1], gradient [N_local,3]) receives the results, the gradient times ``sign``."""
        w, dev = self.refresh(), self.dev
        # read as plain words by the sweep: other types and strides are converted (these are no-ops for the MD drivers)
        species = species.to(torch.int64).contiguous()
        row_mask = None if row_mask is None else row_mask.to(torch.float32).contiguous()
        n_local, e = (pos.shape[0] if n_rows is None else int(n_rows)), int(src.numel())
        with _lib.on_device(dev):
            if src_csr is None:
                src_csr = build_csr(src, n_local, assume_sorted=False)
            energy, grad = out if out is not None else (torch.empty(1, dtype=torch.float32, device=dev),
                                                        torch.empty(n_local, 3, dtype=torch.float32, device=dev))
            atomic = torch.empty(n_owned, dtype=torch.float32, device=dev)
            status = torch.empty(3, dtype=torch.int32, device=dev)
            s = _lib.Sweep.from_buffer_copy(w.struct)
            s.n_local, s.n_owned, s.edges, s.graphs, s.mask_atomic, s.gradient_sign = n_local, n_owned, e, 1, 1, sign
            s.box = tuple(float(b) for b in box)
            s.pos, s.src, s.dst, s.shifts = pos.data_ptr(), src.data_ptr(), dst.data_ptr(), _lib.ptr(shifts)
            s.species, s.status = species.data_ptr(), status.data_ptr()
            s.dst_rowptr, s.src_rowptr, s.src_order = dst_rowptr.data_ptr(), src_csr[0].data_ptr(), _lib.ptr(src_csr[1])
            rows = e
            if pairs is not None:
                s.gate_row, s.rep, s.other = (t.data_ptr() for t in pairs[:3])
                s.live = pairs[3].data_ptr() if len(pairs) > 3 else None
                rows = int(pairs[1].numel())
            s.pair_rows = rows
            s.row_mask = _lib.ptr(row_mask)
            if self.chunk_rows is not None and self.chunk_rows < max(n_owned, n_local):
                s.chunk_rows, s.stream_gates = self.chunk_rows, int(self._streaming(rows))
                s.chunk_capacity_dst = self._chunk_capacity(n_owned, dst_rowptr, e) or self.bucket(max(e, 1))
                s.chunk_capacity_src = self._chunk_capacity(n_local, src_csr[0], e) or self.bucket(max(e, 1))
            s.energy, s.atomic, s.gradient = energy.data_ptr(), atomic.data_ptr(), grad.data_ptr()
            halo = None
            if plan is not None:
                halo = _Halo(plan, n_local, 9 * self.c, dev)
                s.features, s.feature_grad = halo.features.data_ptr(), halo.feature_grad.data_ptr()
            self._run(s, w, halo)
        return energy[0], grad, atomic

    @torch.no_grad()
    def energy_and_forces(self, pos, numbers, batch, src, dst, shifts, cell, row_mask, state=None):
        """(energy per graph, forces, per-atom energies) of a graph whose edges the caller has built, in any order.
        An atomic number that the model does not know and a graph or edge index outside its range raise ValueError."""
        if self._weights is not None and self._weights.tiles is None:
            self._weights = None
        w, dev = self.refresh(state), self.dev
        n, graphs = pos.shape[0], cell.shape[0]
        with _lib.on_device(dev):
            energy = torch.empty(graphs, dtype=torch.float32, device=dev)
            forces = torch.empty(n, 3, dtype=torch.float32, device=dev)
            atomic = torch.empty(n, dtype=torch.float32, device=dev)
            species = torch.empty(n, dtype=torch.int64, device=dev)
            status = torch.zeros(3, dtype=torch.int32, device=dev)
            s = _lib.Sweep.from_buffer_copy(w.struct)
            s.n_local = s.n_owned = n
            s.edges = s.pair_rows = src.numel()
            s.graphs, s.gradient_sign = graphs, -1.0
            s.pos, s.src, s.dst, s.shifts = pos.data_ptr(), src.data_ptr(), dst.data_ptr(), shifts.data_ptr()
            s.cells, s.batch, s.numbers = cell.data_ptr(), batch.data_ptr(), numbers.data_ptr()
            s.species, s.status, s.row_mask = species.data_ptr(), status.data_ptr(), _lib.ptr(row_mask)
            s.energy, s.atomic, s.gradient = energy.data_ptr(), atomic.data_ptr(), forces.data_ptr()
            if w.tiles is not None:
                s.watch_tiles, s.watch_copy, s.watch_count = w.tiles.data_ptr(), w.copy.data_ptr(), w.tiles.shape[0]
            flags, event = _status_mailbox(dev)
            s.host_status, s.host_status_event = flags.data_ptr(), event.cuda_event
            self._run(s, w, None)
            event.synchronize()
            bits, by_dst, by_src = flags.tolist()
        if bits & 4:                     # a parameter was written behind its version counter
            self._weights = None
            return self.energy_and_forces(pos, numbers, batch, src, dst, shifts, cell, row_mask)
        if bits & 1:
            raise ValueError(f"Encountered atomic numbers outside {self.model.atomic_numbers}")
        if bits & 2:
            raise ValueError(f"batch: graph index outside [0, {graphs})")
        if by_dst < 0 or by_src < 0:
            raise ValueError("edge index outside [0, num_nodes)")
        return energy, forces, atomic


class _Halo:
    """Exchange plan and the two feature buffers whose ghost rows it fills."""

    def __init__(self, exchange, rows, width, device):
        self.exchange = exchange
        self.features = torch.empty(rows, width, dtype=torch.float32, device=device)
        self.feature_grad = torch.empty(rows, width, dtype=torch.float32, device=device)


def _status_mailbox(device):
    """Pinned words and an event of this thread and device: a sweep's status is copied early and read when the sweep has
    been queued, so that the host does not wait for the sweep itself."""
    boxes = _local.__dict__.setdefault("boxes", {})
    if device not in boxes:
        event = torch.cuda.Event()
        event.record()
        boxes[device] = (torch.zeros(3, dtype=torch.int32, pin_memory=True), event)
    return boxes[device]
