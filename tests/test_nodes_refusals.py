"""Calls that the Python functions of the layers refuse are refused by the C++ autograd nodes too, with the same class of error and
before anything is launched, and what the module has from the library is what the library says.  Here the module is called by itself,
on tensors of the host: no case gets as far as a launch."""
import pytest
import torch

from primus_b200.ops import _lib, attention, fused, layers, moe


@pytest.fixture(scope="module")
def nodes():
    with pytest.MonkeyPatch.context() as m:
        m.setattr(torch.cuda, "is_available", lambda: True)
        module = _lib._load_nodes()
    if module is None:
        pytest.skip("the autograd nodes are not built")
    return module


def _zeros(*shape):
    return torch.zeros(*shape, dtype=torch.bfloat16)


ROPE_ARGS = (None, None, None, 1, 4, 2, 64, 64, True, 0.125)      # no rotation, 4 query and 2 key / value heads of 64


@pytest.mark.parametrize("qkv,error", [(lambda: _zeros(128, 520), RuntimeError),                  # 8 heads and 8 columns more
                                       (lambda: _zeros(128, 512)[:, :448], RuntimeError),         # a head less, of a wider buffer
                                       (lambda: _zeros(128, 1024)[:, ::2], AssertionError),       # every other column
                                       (lambda: _zeros(2, 64, 512), RuntimeError)])
def test_rope_attention_of_other_layouts(nodes, monkeypatch, qkv, error):
    with pytest.raises(error, match="heads"):
        nodes.rope_attention(qkv(), *ROPE_ARGS, 0, None, 0.0)
    monkeypatch.setattr(_lib, "call", lambda *a: None)             # (the Python function, whose launches do nothing)
    with pytest.raises(error):
        layers.RopeAttentionFn.apply(qkv(), *ROPE_ARGS)


@pytest.mark.parametrize("labels,weights", [(30, 29), (30, 31), (30, 1), (30, 0), (29, 30), (1, 30), (29, 29), (31, None), (29, None)])
def test_cross_entropy_of_other_lengths(nodes, monkeypatch, labels, weights):
    logits, labels = _zeros(2, 15, 64), torch.zeros(labels, dtype=torch.int64)
    weights = None if weights is None else torch.ones(weights)
    launched = []
    monkeypatch.setattr(_lib, "call", lambda *a: launched.append(a))
    for call in (nodes.cross_entropy, lambda x, l, w, unit: fused.CrossEntropyFn.apply(x, l, 0, None, w, unit)):
        with pytest.raises(RuntimeError, match="30 rows"):
            call(logits, labels, weights, False)
    assert not launched
    with pytest.raises(RuntimeError):                              # the reference of the host's tensors
        fused.cross_entropy(logits, labels, weights=weights)


def test_attention_of_no_sequences(nodes, monkeypatch):
    q, qkv = _zeros(128, 2, 64), _zeros(128, 512)
    rope = (*ROPE_ARGS[:3], 0, *ROPE_ARGS[4:])
    monkeypatch.setattr(_lib, "call", lambda *a: None)
    for call in (lambda: nodes.flash_attention(q, q, q, 0, True, 0.125, 0, 0, None, 0.0),
                 lambda: attention.FlashAttnFn.apply(q, q, q, 0, True, 0.125),
                 lambda: nodes.rope_attention(qkv, *rope, 0, None, 0.0), lambda: layers.RopeAttentionFn.apply(qkv, *rope)):
        with pytest.raises(ZeroDivisionError):                     # (an integer division ended the process)
            call()


@pytest.mark.parametrize("rows", [0, 1, 295, 296, 297, 100000])
def test_partial_sums_have_the_librarys_size(nodes, rows):
    assert nodes.partial_rows(rows) == _lib.call_ret("rmsnorm_bwd_num_partials", rows)


@pytest.mark.parametrize("layer", ["swiglu", "swiglu_linear"])
@pytest.mark.parametrize("rows", [64, 16])
def test_gated_rows_of_odd_width(nodes, monkeypatch, layer, rows):
    x, w = _zeros(rows, 17), _zeros(24, 8)
    monkeypatch.setattr(_lib, "call", lambda *a, **k: None)
    monkeypatch.setattr(layers.gemm, "gemm", lambda a, b, **k: _zeros(rows, 24))
    calls = [lambda: nodes.swiglu(x, None, 0.0, 0), lambda: fused.SwiGLUFn.apply(x, None, 0.0)]
    if layer == "swiglu_linear":
        calls = [lambda: nodes.swiglu_linear(x, w, 0.0, 0), lambda: layers.SwiGLULinearFn.apply(x, w, None, 0.0, None, False)]
    for call in calls:
        with pytest.raises(RuntimeError, match="shape|halves"):
            call()


@pytest.mark.parametrize("which", range(3))
@pytest.mark.parametrize("shape", [(128, 64), (1, 128, 2, 64)])
def test_attention_of_other_dimensions(nodes, monkeypatch, which, shape):
    monkeypatch.setattr(_lib, "call", lambda *a, **k: None)
    qkv = [_zeros(128, 2, 64) for _ in range(3)]
    qkv[which] = _zeros(*shape)
    errors = []
    for call in (lambda: nodes.flash_attention(*qkv, 1, True, 0.125, 0, 0, None, 0.0), lambda: attention.FlashAttnFn.apply(*qkv, 1, True, 0.125)):
        with pytest.raises((ValueError, IndexError, AssertionError)) as e:
            call()
        errors.append(e.type)
    assert errors[0] is errors[1]


@pytest.mark.parametrize("which", ["router", "router 1", "pos", "pos 1", "weight", "weight 2"])
def test_moe_tensors_of_other_dimensions(nodes, monkeypatch, which):
    """Logits [T, E], positions [T, k], weights [E, N, K]: the Python functions unpack these shapes."""
    monkeypatch.setattr(_lib, "call", lambda *a, **k: None)
    ints = torch.zeros(2, 3, 4, dtype=torch.int32)
    sched = moe.Schedule(*[ints] * 5, rows_cap=8)
    x = _zeros(8, 16)
    calls = {
        "router": [(f, _zeros(2, 3, 8)) for f in (nodes.router, moe.RouterFn.apply)],
        "router 1": [(f, _zeros(8)) for f in (nodes.router, moe.RouterFn.apply)],
        "pos": [(lambda p, f=f: f(x, p, ints), ints) for f in (nodes.combine_rows, moe.CombineRowsFn.apply)],
        "pos 1": [(lambda p, f=f: f(x, p, ints), ints[0, 0]) for f in (nodes.combine_rows, moe.CombineRowsFn.apply)],
        "weight": [(lambda w: nodes.grouped_linear(x, w, ints, ints, ints), _zeros(1, 2, 16, 16)),
                   (lambda w: moe.GroupedLinearFn.apply(x, w, sched), _zeros(1, 2, 16, 16))],
        "weight 2": [(lambda w: nodes.grouped_linear(x, w, ints, ints, ints), _zeros(16, 16)),
                     (lambda w: moe.GroupedLinearFn.apply(x, w, sched), _zeros(16, 16))],
    }[which]
    for call, t in calls:
        with pytest.raises(ValueError):
            call(t, None, 2, False, False, 0, 0, 1.0, None) if which.startswith("router") else call(t)
