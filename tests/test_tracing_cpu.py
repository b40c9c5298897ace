"""While torch.jit.trace records, sizes are tensors: their addresses do not travel as sizes, and the C++ nodes, of which a trace would
keep the empty tensors around the launches, leave the layers to the Python functions."""
import pytest
import torch

from primus_b200.ops import _lib


@pytest.mark.parametrize("known", [False, True])
def test_recorded_sizes_are_refused(monkeypatch, known):
    launched = []

    def launch(args, stream):
        if isinstance(args[1], torch.Tensor):
            return None                         # the kind of argument that a bound launcher refuses
        launched.append(args)
        return 0

    monkeypatch.setattr(_lib, "_BOUND", {("k", True): (launch, 1)} if known else {})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 0)

    def op(x, rows=None):
        out = torch.empty_like(x)
        _lib.call("k", x, x.shape[0] if rows is None else rows, out)
        return out

    x = torch.zeros(4)
    with pytest.raises(_lib.NativeLibraryError, match="trace"):
        torch.jit.trace(op, (x,), check_trace=False)
    assert not launched
    if known:
        op(x)
        torch.jit.trace(lambda x: op(x, 4), (x,), check_trace=False)      # (a size that is a number)
        assert [a[1] for a in launched] == [4, 4]


def test_nodes_are_not_traced(monkeypatch):
    node, seen = object(), []
    monkeypatch.setattr(_lib, "_NODES", [node])

    def op(x):
        seen.append(_lib.nodes())
        return x * 1

    torch.jit.trace(op, (torch.zeros(4),), check_trace=False)
    op(torch.zeros(4))
    assert seen == [None, node]
