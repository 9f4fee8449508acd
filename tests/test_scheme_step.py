"""What a scheme keeps of an allocation that starts before a layer's backward."""
import copy
import threading
from types import SimpleNamespace

import pytest
import torch

import actnn_b200 as actnn
from actnn_b200 import ops


@pytest.fixture
def closing_scheme(monkeypatch):
    """The scheme of the only layer, whose backward ends the step; nothing here needs a device."""
    actnn.set_optimization_level("L3")
    monkeypatch.setattr(actnn.QScheme, "update_scale", False)
    # as an event and a pinned copy, what start_perlayer returns cannot be copied
    monkeypatch.setattr(actnn.QScheme, "start_perlayer", staticmethod(lambda: [threading.Lock()]))
    scheme = actnn.QScheme(torch.nn.Linear(3, 2))
    scheme.C, scheme.dim = torch.ones(4), 3
    return scheme


def failing_backward(kind, scheme, monkeypatch):
    def no_memory(*args):
        assert scheme._started is not None
        raise torch.OutOfMemoryError("no memory")
    monkeypatch.setattr(ops, "dequantize_activation", no_memory)
    ctx = SimpleNamespace(scheme=scheme, saved=((), None, None), needs_input_grad=[True] * 3)
    grad = torch.ones(4, 2, 1, 1)
    if kind == "linear":
        ctx.other_args = ((4, 3), torch.float32)
        ops.linear.backward(ctx, grad.view(4, 2))
    elif kind == "conv2d":
        ctx.other_args = ((4, 3, 1, 1), 1, 0, 1, 1, torch.float32)
        ops.conv2d.backward(ctx, grad)
    else:
        ctx.other_args = ((4, 3, 1, 1), 1, 0, 0, 1, 1, torch.float32)
        ops.conv_transpose2d.backward(ctx, grad)


@pytest.mark.parametrize("kind", ["linear", "conv2d", "conv_transpose2d"])
def test_a_failed_backward_keeps_nothing_of_it(kind, closing_scheme, monkeypatch):
    widths = closing_scheme.bits
    with pytest.raises(torch.OutOfMemoryError):
        failing_backward(kind, closing_scheme, monkeypatch)
    assert closing_scheme._started is None and closing_scheme.bits is widths
    assert copy.deepcopy(closing_scheme).bits == widths


def test_a_program_can_put_its_own_allocation_in_place(closing_scheme, monkeypatch):
    calls = []
    monkeypatch.setattr(actnn.QScheme, "allocate_perlayer", staticmethod(lambda: calls.append("own")))
    closing_scheme.start_allocation()
    assert closing_scheme._started is None and not calls
    closing_scheme.if_allocate_perlayer()
    assert calls == ["own"]
