"""Which models the native force sweep may answer for (host logic, no GPU): the stock model, and none whose own forward computes
something that the sweep does not read."""
import copy
import ctypes

import pytest
import torch
from torch import nn


def _model():
    from mace_ictc.model import MaceIctcModel
    torch.manual_seed(0)
    return MaceIctcModel(channels=64, cutoff=4.5)


def _stands_for(model):
    from mace_ictc.engine import ForceEngine
    try:
        return ForceEngine(model, lay_out=False).stands_for() is not None
    except ValueError:                                    # another width or depth: no engine at all
        return False


def _biased(rows, cols):
    return nn.Linear(cols, rows, bias=True)


def _set(path, make):
    def change(model):
        *parents, last = path.split(".")
        owner = model
        for name in parents:
            owner = owner[int(name)] if name.isdigit() else getattr(owner, name)
        if last.isdigit():
            owner[int(last)] = make()
        else:
            setattr(owner, last, make())
    return change


def _mlp_readout():
    from mace_ictc.model import MLPReadout
    return MLPReadout(9 * 64)


OTHER_MODELS = {
    "bias of the last linear": _set("last_layer_energy_readout.linear_2", lambda: _biased(1, 16)),
    "bias set on the hidden linear": _set("last_layer_energy_readout.linear_1.bias", lambda: nn.Parameter(torch.randn(16))),
    "bias of the first readout": _set("layer_energy_readouts.0.readout", lambda: _biased(1, 64)),
    "three outputs": _set("last_layer_energy_readout.linear_2", lambda: nn.Linear(16, 3, bias=False)),
    "identity for the readout's activation": _set("last_layer_energy_readout.activation", nn.Sequential),
    "another activation": _set("interactions.0.fc.3", nn.Tanh),
    "identity for a radial activation": _set("interactions.1.fc.1", nn.Sequential),
    "bias in the radial network": _set("interactions.0.fc.2", lambda: _biased(64, 64)),
    "another first readout": _set("layer_energy_readouts.0", _mlp_readout),
    "a further radial layer": lambda m: m.interactions[0].fc.append(nn.Linear(704, 704, bias=False)),
    "a further interaction": lambda m: (m.interactions.append(m.interactions[1]), m.products.append(m.products[1])),
    "contraction of the other layout": lambda m: setattr(m.products[0].symmetric_contractions, "ir_mul", True),
    "a fractional cutoff order": lambda m: setattr(m, "polynomial_cutoff_p", 5.5),
    "double precision": lambda m: m.double(),
    "a forward of its own on the model": lambda m: setattr(m, "forward", lambda *a, **k: None),
    "a forward of its own on a block": lambda m: setattr(m.products[1], "forward", lambda *a, **k: None),
    "a hook": lambda m: m.interactions[0].linear_up.register_forward_hook(lambda *_: None),
    "a hook on the model": lambda m: m.register_forward_pre_hook(lambda *_: None),
    "trainable base coefficients": lambda m: m.interactions[0].tp.weight.requires_grad_(True),
}


@pytest.mark.parametrize("name", OTHER_MODELS)
@pytest.mark.parametrize("seen_before", [False, True])
def test_other_models_go_to_the_autograd_route(name, seen_before):
    """Changed before the engine first looks at the model, and behind its back afterwards."""
    from mace_ictc.engine import ForceEngine
    model = _model()
    if seen_before:
        engine = ForceEngine(model, lay_out=False)
        if not name.startswith("contraction"):          # a plain attribute: read when the structure is walked
            assert engine.stands_for() is not None
        OTHER_MODELS[name](model)
        assert engine.stands_for() is None
    else:
        OTHER_MODELS[name](model)
        assert not _stands_for(model)


def test_the_stock_model_is_covered():
    from mace_ictc.model import MaceIctcModel
    assert _stands_for(_model()) and _stands_for(copy.deepcopy(_model()))
    assert _stands_for(MaceIctcModel(correlation=2, number_of_basis=6, readout_hidden_channels=20, atomic_numbers=(1, 6, 7, 8)))
    assert _stands_for(MaceIctcModel(correlation=1, atomic_numbers=(14,)))
    assert not _stands_for(MaceIctcModel(radial_mlp_hidden=(64, 64)))
    biased = _model()                                     # these two read the weight alone in the forward, too
    biased.node_embedding = _biased(64, 3)
    biased.interactions[1].linear_up.adapters["1"] = _biased(64, 64)
    assert _stands_for(biased)


def test_subclasses_with_the_stock_forward_keep_the_engine():
    from mace_ictc.engine import covers
    from mace_ictc.model import MaceIctcModel

    class Named(MaceIctcModel):
        name = "mine"

    class Other(MaceIctcModel):
        def forward(self, *args, **kwargs):
            return 2 * super().forward(*args, **kwargs)

    assert covers(Named()) and not covers(Other()) and not covers(torch.nn.Linear(2, 2))


def test_misaligned_weights_and_buffers_are_refused_before_any_launch():
    """Made-up addresses, none of which is touched: the check comes before the first launch."""
    from ictc_o3 import _lib
    lib = _lib.load()

    def sweep():
        s = _lib.Sweep(n_local=4, n_owned=4, edges=8, pair_rows=8, num_species=3, graphs=1, num_basis=8, poly_p=5, hidden=16,
                       r_max=4.5, work_bytes=0)
        for name in ("pos", "src", "dst", "species", "energy", "atomic", "gradient", "status", "work", "up0_table", "sc0_table",
                     "readout_rp", "readout_rs", "readout_w2", "readout_ro0"):
            setattr(s, name, 4096)
        for k in range(2):
            for name in ("w0", "w3", "w3t", "bank"):
                setattr(s.layer[k], name, 4096)
            for name, count in (("hid", 2), ("hid_t", 2), ("up", 3), ("up_b", 3), ("ml", 3), ("ml_b", 3), ("pl", 3), ("pl_b", 3)):
                setattr(s.layer[k], name, (4096,) * count)
            s.layer[k].num_gates = 64 * (3, 11)[k]
            s.layer[k].slots = ((1, 1, 1), (3, 4, 4))[k]
        return s

    def refused(s, text):
        assert lib.ictc_sweep_run(ctypes.byref(s), 31, None) == -2 and text in _lib.last_error()

    refused(sweep(), "too small")                         # everything in order, but the workspace has no room
    for name, off in (("work", 16), ("features", 16), ("feature_grad", 4), ("up0_table", 8), ("readout_rp", 4), ("readout_rs", 4),
                      ("readout_ro0", 4)):
        s = sweep()
        setattr(s, name, 4096 + off)
        refused(s, "aligned")
    for k, name in ((0, "w3"), (1, "w3t")):
        s = sweep()
        setattr(s.layer[k], name, 4096 + 8)
        refused(s, "aligned")
    s = sweep()
    s.layer[1].up = (4096, 0, 4096)
    refused(s, "NULL")
