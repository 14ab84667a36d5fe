"""Who calls a network's layers: their own forward() while nothing hangs on the call of a module, the module otherwise."""
import functools
import subprocess
import sys

import pytest
import torch

from simnets_tf_b200.simnet import _caller


@pytest.mark.parametrize("name", ["__call__", "_call_impl"])
def test_a_replaced_call_of_all_modules_sees_every_layer(monkeypatch, name):
    layer, seen = torch.nn.Linear(2, 3), []
    assert _caller()(layer) == layer.forward
    own = getattr(torch.nn.Module, name)

    @functools.wraps(own)
    def watched(self, *args, **kwargs):
        seen.append(self)
        return own(self, *args, **kwargs)
    monkeypatch.setattr(torch.nn.Module, name, watched)
    _caller()(layer)(torch.zeros(1, 2))
    assert seen == [layer]
    monkeypatch.undo()
    assert _caller()(layer) == layer.forward


def test_a_symbolic_tracer_sees_the_layers_as_modules():
    class Leaves(torch.fx.Tracer):
        def is_leaf_module(self, m, name):
            return True

    class Net(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.layer = torch.nn.Linear(2, 3)

        def forward(self, x):
            return _caller()(self.layer)(x)
    assert [n.target for n in Leaves().trace(Net()).nodes if n.op == "call_module"] == ["layer"]


def test_a_call_that_was_replaced_before_the_import_is_left_in_place():
    code = """
import torch
seen = []
own = torch.nn.Module.__call__
torch.nn.Module.__call__ = lambda self, *a, **k: (seen.append(self), own(self, *a, **k))[1]
from simnets_tf_b200.simnet import _caller
layer = torch.nn.Linear(2, 3)
_caller()(layer)(torch.zeros(1, 2))
assert seen == [layer]
"""
    assert subprocess.run([sys.executable, "-c", code], timeout=300).returncode == 0


def test_what_hangs_on_one_layer():
    layer, other = torch.nn.Linear(2, 3), torch.nn.Linear(3, 2)
    handle = layer.register_forward_hook(lambda m, i, o: None)
    call = _caller()
    assert call(layer) is layer and call(other) == other.forward
    handle.remove()

    class Counted(torch.nn.Linear):
        def __call__(self, *args, **kwargs):
            return super().__call__(*args, **kwargs)
    counted = Counted(2, 3)
    assert _caller()(counted) is counted and _caller()(layer) == layer.forward
