"""A trace records torch's operations, and of a launch only the empty tensors around it: kernels are refused while one is recorded,
by the Python binding and in front of the C++ nodes."""
import pytest
import torch

from primus_b200.ops import _lib


def test_launches_are_not_traced(monkeypatch):
    launched = []
    monkeypatch.setattr(_lib, "_BOUND", {("k", True): (lambda args, stream: launched.append(args) or 0, 1)})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 0)

    def op(x):
        out = torch.empty_like(x)
        _lib.call("k", x, out)
        return out

    with pytest.raises(_lib.NativeLibraryError, match="trace"):
        torch.jit.trace(op, (torch.zeros(4),), check_trace=False)
    assert not launched
    op(torch.zeros(4))
    assert len(launched) == 1


def test_nodes_are_not_traced(monkeypatch):
    node = object()
    monkeypatch.setattr(_lib, "_NODES", [node])

    def op(x):
        assert _lib.nodes() is node
        return x * 1

    with pytest.raises(_lib.NativeLibraryError, match="trace"):
        torch.jit.trace(op, (torch.zeros(4),), check_trace=False)
    op(torch.zeros(4))
