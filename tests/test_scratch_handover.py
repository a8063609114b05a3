"""The scratch that the operators hand to the library for its next call: never left behind when a call is not made.  On the CPU, with a
stand-in for the library."""
import pytest
import torch

from helpers import cabi, quant_ops, synth


class _Library:
    """Keeps the pending scratch as the library does: set by scratch_next, taken by the next call."""

    def __init__(self, result=0, error=None):
        self.pending, self.seen, self.result, self.error = None, [], result, error

    def b200q_scratch_bytes(self, rows, k, dtype):
        return rows * k * 2 if dtype == cabi.BF16 and rows >= 5 else 0

    def b200q_scratch_next(self, ptr, size):
        self.pending = ptr
        return 0

    def _call(self, *args):
        if self.error is not None:
            raise self.error
        self.seen.append(self.pending)
        self.pending = None
        return self.result

    b200q_qmatvec = b200q_gate_up_swiglu = b200q_norm_qmatvec = _call

    def b200q_strerror(self, code):
        return b"stand-in"


@pytest.fixture
def library(monkeypatch):
    lib = _Library()
    monkeypatch.setattr(cabi, "load", lambda: lib)
    monkeypatch.setattr(cabi, "require_cuda", lambda *tensors: None)
    monkeypatch.setattr(cabi, "stream", lambda: 0)
    return lib


def _gate_up(norm_weight, dtype=torch.bfloat16):
    w, s, z = synth.quantized_weight(32, 64, 4, 32, seed=1)
    x = synth.activations((5, 64), 2, "cpu", dtype)
    return quant_ops.gate_up_rows(4, x, w, w, s, s, z, z, 32, want_act=True, norm_weight=norm_weight)


def test_a_call_gets_the_scratch_and_leaves_none(library):
    _gate_up(torch.ones(64))
    assert library.seen[0] is not None and library.pending is None


def test_an_argument_that_is_refused_leaves_none(library):
    with pytest.raises(TypeError, match="unsupported dtype"):
        _gate_up(torch.ones(64, dtype=torch.float64))
    assert library.seen == [] and library.pending is None


@pytest.mark.parametrize("error", [None, RuntimeError("conversion failed")])
def test_a_call_that_fails_leaves_none(library, error):
    library.error, library.result = error, -2
    with pytest.raises(RuntimeError):
        _gate_up(torch.ones(64))
    assert library.pending is None


def test_a_call_without_scratch_clears_what_was_left(library):
    library.pending = 4096
    _gate_up(torch.ones(64), torch.float16)
    assert library.seen == [None]
