"""The C++ autograd nodes against the Python functions that they stand in for: same bits, and the same answers to what surrounds a
node (gradient buffers and their callbacks, deferred weight gradients, hooks on saved tensors, recipes, transforms, errors)."""
import pytest
import torch

from primus_b200.ops import _lib, attention, fused, gemm, layers

pytestmark = pytest.mark.gpu


def _gen(seed=0):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, device="cuda", generator=g).bfloat16()


def _param(g, *shape, main):
    p = torch.nn.Parameter(_randn(g, *shape) * 0.1 + (1.0 if len(shape) == 1 else 0.0))
    if main:
        p.main_grad = torch.ones(*shape, device="cuda")
        p.calls = []
        p._grad_ready_cb = lambda w: w.calls.append(w is p)
    return p


def _both(monkeypatch, build, n_params, callbacks=True, skip=()):
    """Runs ``build(native)`` -> (outputs, leaves, params) with and without the nodes and compares everything."""
    runs = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(_lib, "_NODES", [None])
        outs, leaves, params, dys = build()
        before = _lib.launch_count()
        torch.autograd.backward(outs, dys)
        assert callbacks is False or skip or (type(outs[0].grad_fn).__name__.startswith("CppFunction") or "Cpp" in outs[0].grad_fn.name()) == native
        runs.append([o.detach() for o in outs] + [t.grad for t in leaves] + [getattr(p, "main_grad", p.grad) for p in params])
        runs[-1].append(_lib.launch_count() - before)
        for p in params:
            if hasattr(p, "main_grad") and callbacks:
                assert p.grad is None and (p.dim() == 1 or (p.calls == [True] and p.grad_added_to_main_grad))
    monkeypatch.undo()
    for i, (a, b) in enumerate(zip(*runs)):
        assert i in skip or (a is None and b is None) or (a == b if isinstance(a, int) else torch.equal(a, b)), i


@pytest.mark.parametrize("shape", [(37, 512), (3, 5, 64), (200, 2048), (1, 16384)])
@pytest.mark.parametrize("residual", ["none", "leaves", "inner"])
@pytest.mark.parametrize("main", [False, True])
@pytest.mark.parametrize("what", ["norm", "norm_linear"])
def test_norms(monkeypatch, shape, residual, main, what):
    def build():
        g = _gen(1)
        x, r = _randn(g, *shape).requires_grad_(), _randn(g, *shape).requires_grad_()
        w, p = _param(g, shape[-1], main=main), _param(g, 136, shape[-1], main=main)
        a, b = (x, r) if residual == "leaves" else (x * 1, r * 1)
        b = None if residual == "none" else b
        leaves = [x] if b is None else [x, r]
        if what == "norm":
            outs = fused.rmsnorm(a, w, 1e-5, b)
            outs = [outs] if b is None else list(outs)
            return outs, leaves, [w], [_randn(g, *o.shape) for o in outs]
        outs = list(layers.norm_linear(a, b, w, p, 1e-5))
        if b is None:
            outs = outs[:1]
        return outs, leaves, [w, p], [_randn(g, *o.shape) for o in outs]

    _both(monkeypatch, build, 2)


@pytest.mark.parametrize("used", [0, 1])
def test_norm_with_one_output_used(monkeypatch, used):
    def build():
        g = _gen(2)
        x, r = _randn(g, 20, 256).requires_grad_(), _randn(g, 20, 256).requires_grad_()
        w, p = _param(g, 256, main=False), _param(g, 128, 256, main=False)
        o = layers.norm_linear(x, r, w, p, 1e-5)[used]
        return [o], [x, r], [w, p], [_randn(g, *o.shape)]

    _both(monkeypatch, build, 2)


@pytest.mark.parametrize("T,K,N", [(1, 64, 64), (300, 256, 688), (1024, 1024, 1024), (130, 4096, 128)])
@pytest.mark.parametrize("main", [False, True])
def test_linear_and_swiglu(monkeypatch, T, K, N, main):
    def lin():
        g = _gen(3)
        x, w = _randn(g, T, K).requires_grad_(), _param(g, N, K, main=main)
        o = gemm.linear(x.view(1, T, K), w)
        return [o], [x], [w], [_randn(g, *o.shape)]

    def glu(clamp, act):
        def build():
            g = _gen(4)
            x, w = _randn(g, T, 2 * K).requires_grad_(), _param(g, N, K, main=main)
            o = layers.swiglu_linear(x, w, clamp=clamp, act=act)
            return [o], [x], [w], [_randn(g, *o.shape)]
        return build

    _both(monkeypatch, lin, 1)
    _both(monkeypatch, glu(0.0, "silu"), 1)
    _both(monkeypatch, glu(0.7, "gelu"), 1)


@pytest.mark.parametrize("frozen", ["x", "w"])
def test_linear_with_one_gradient(monkeypatch, frozen):
    def build():
        g = _gen(5)
        x, w = _randn(g, 64, 128), _param(g, 256, 128, main=False)
        x.requires_grad_(frozen != "x")
        w.requires_grad_(frozen != "w")
        o = gemm.linear(x, w)
        return [o], [x], [w], [_randn(g, *o.shape)]

    _both(monkeypatch, build, 1)


@pytest.mark.parametrize("d,dv", [(64, 64), (128, 128), (192, 128)])
@pytest.mark.parametrize("window,sinks", [(0, False), (100, True)])
def test_attention(monkeypatch, d, dv, window, sinks):
    if d != dv and (window or sinks):
        pytest.skip("plain attention only")

    def build():
        g = _gen(6)
        hq, hkv = (4, 2) if d == dv else (2, 2)
        qkv = _randn(g, 256, (hq + hkv) * d + hkv * dv)
        q, k, v = (t.reshape(256, n, e) if d != dv else t.view(256, n, e) for t, n, e in (
            (qkv[:, :hq * d], hq, d), (qkv[:, hq * d:(hq + hkv) * d], hkv, d), (qkv[:, (hq + hkv) * d:], hkv, dv)))
        leaves = [t.requires_grad_() for t in (q, k, v)]
        s = torch.randn(hq, device="cuda", generator=g).requires_grad_() if sinks else None
        o = attention.flash_attention(*leaves, 2, True, window=window, sinks=s)
        return [o], leaves + ([s] if sinks else []), [], [_randn(g, *o.shape)]

    _both(monkeypatch, build, 0)


@pytest.mark.parametrize("rope", [False, True])
@pytest.mark.parametrize("sinks", [False, True])
@pytest.mark.parametrize("qknorm", [False, True])
def test_rope_attention(monkeypatch, rope, sinks, qknorm):
    def build():
        g = _gen(7)
        T, hq, hkv, d = 256, 4, 2, 64
        x = _randn(g, T, (hq + 2 * hkv) * d).requires_grad_()
        cos, sin = fused.rope_tables(T, d, 1e4, "cuda") if rope else (None, None)
        pos = torch.arange(T, device="cuda", dtype=torch.int32) % 128 if rope else None
        ws = [_param(g, d, main=False) for _ in range(2)] if qknorm else []
        y = x * 1
        if qknorm:
            t = fused.qk_norm_rope(y, *ws, hq, hkv, d, 1e-5, cos, sin, pos, d) if rope else fused.qk_norm(y, *ws, hq, hkv, d)
            y, cos, sin, pos = t, None, None, None
        s = torch.randn(hq, device="cuda", generator=g).requires_grad_() if sinks else None
        o = layers.rope_attention(y, cos, sin, pos, 2, hq, hkv, d, window=0, sinks=s)
        return [o], [x] + ([s] if sinks else []), ws, [_randn(g, *o.shape)]

    _both(monkeypatch, build, 0)


@pytest.mark.parametrize("weighted,unit", [(False, False), (True, False), (True, True)])
def test_cross_entropy(monkeypatch, weighted, unit):
    def build():
        g = _gen(12)
        x = _randn(g, 2, 150, 1032).requires_grad_()
        labels = torch.randint(0, 1032, (2, 150), device="cuda", generator=g)
        weights = torch.rand(2, 150, device="cuda", generator=g) if weighted else None
        o = fused.cross_entropy(x * 1, labels, weights=weights, unit_upstream=unit)
        exact = torch.nn.functional.cross_entropy(x.detach().double().view(300, -1), labels.view(-1), reduction="none").view(2, 150)
        exact = (exact * weights.double()).sum() if weighted else exact
        assert torch.allclose(o.double(), exact, rtol=2.0 ** -18, atol=2.0 ** -18)
        # (the weighted sum in another order than torch's: its bits are compared with the formula above)
        return [o * 1 if not unit else o], [x], [], [torch.ones_like(o) if unit else torch.full_like(o, 0.7)]

    _both(monkeypatch, build, 0, callbacks=False, skip=(0,) if weighted else ())


@pytest.mark.parametrize("main", [False, True])
def test_embedding(monkeypatch, main):
    def build():
        g = _gen(13)
        w = _param(g, 300, 64, main=False)
        if main:
            w.main_grad = torch.ones(300, 64, device="cuda")
        t = torch.randperm(300, device="cuda", generator=g)[:128].view(2, 64)
        o = fused.embedding(t, w)
        return [o], [], [w], [_randn(g, *o.shape)]

    _both(monkeypatch, build, 1, callbacks=False)


@pytest.mark.parametrize("main", [False, True])
@pytest.mark.parametrize("kw", [dict(), dict(moe_router_score_function="sigmoid", moe_router_enable_expert_bias=True),
                                dict(moe_router_pre_softmax=True, moe_aux_loss_coeff=0.0)])
def test_moe_layer(monkeypatch, main, kw):
    from primus_b200.models.config import TransformerConfig
    from primus_b200.models.moe import MoELayer
    from primus_b200.parallel.distributed import ParamGradBuffer

    def build():
        torch.manual_seed(0)
        cfg = TransformerConfig(**{**dict(num_layers=2, hidden_size=256, num_experts=8, moe_router_topk=2, moe_ffn_hidden_size=192,
                                          moe_aux_loss_coeff=1e-2), **kw})
        m = MoELayer(cfg, 0, "cuda", 1)
        if main:
            m.buffer = ParamGradBuffer(list(m.parameters()), None, 1, 0)
        g = _gen(14)
        x = _randn(g, 200, 256).requires_grad_()
        o = m(x)
        m.keep = o
        return [o], [x], list(m.parameters()), [_randn(g, *o.shape)]

    _both(monkeypatch, build, 3, callbacks=False)


def test_hooks_on_saved_tensors_see_them_all():
    g = _gen(8)
    x, r, w, p = _randn(g, 64, 256).requires_grad_(), _randn(g, 64, 256).requires_grad_(), _param(g, 256, main=False), _param(g, 128, 256, main=False)

    def grads(hooked):
        for t in (x, r, w, p):
            t.grad = None
        packed = []
        hooks = torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.cpu(), lambda t: t.cuda())
        if hooked:
            with hooks:
                o, s = layers.norm_linear(x, r, w, p, 1e-5)
        else:
            o, s = layers.norm_linear(x, r, w, p, 1e-5)
        torch.autograd.backward([o, s], [torch.ones_like(o), torch.ones_like(s)])
        return packed, [t.grad.clone() for t in (x, r, w, p)]

    packed, a = grads(True)
    _, b = grads(False)
    assert len(packed) == 4 and all(torch.equal(u, v) for u, v in zip(a, b))


def test_changed_input_is_noticed():
    g = _gen(9)
    w = _param(g, 128, 64, main=False)
    x = _randn(g, 64, 64).requires_grad_() * 1
    o = gemm.linear(x, w)
    x.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        o.sum().backward()


def test_deferred_weight_gradients():
    g = _gen(10)
    x, w = _randn(g, 64, 128).requires_grad_(), _param(g, 256, 128, main=True)
    o = gemm.linear(x, w)
    gemm.WGRAD_STORE.begin("k")
    try:
        o.backward(torch.ones_like(o))
    finally:
        gemm.WGRAD_STORE.end()
    assert (w.main_grad == 1).all() and not w.calls
    gemm.WGRAD_STORE.flush("k")
    want = torch.ones_like(w.main_grad) + torch.ones(256, 64, device="cuda") @ x.detach().float()
    assert torch.allclose(w.main_grad, want, rtol=1e-4, atol=1e-4) and w.calls == [True]


def test_recipe_set_between_forward_and_backward():
    g = _gen(11)
    x, w = _randn(g, 128, 256).requires_grad_(), _param(g, 128, 256, main=False)
    grads = []
    for change in (False, True):
        x.grad = w.grad = None
        o = gemm.linear(x, w) if change else gemm.LinearFn.apply(x, w)
        gemm.set_fp8_recipe("mxfp8")
        try:
            o.backward(torch.ones_like(o) * 0.3)
        finally:
            gemm.set_fp8_recipe(None)
        grads.append((x.grad.clone(), w.grad.clone()))
    assert all(torch.equal(a, b) for a, b in zip(*grads))


def test_transforms_are_refused_as_before():
    w = torch.ones(64, device="cuda").bfloat16()
    x = torch.randn(4, 64, device="cuda").bfloat16()
    for call in (lambda: torch.func.grad(lambda t: fused.rmsnorm(t, w).float().sum())(x), lambda: torch.vmap(lambda t: fused.rmsnorm(t, w))(x[None])):
        with pytest.raises(RuntimeError):
            call()
    with torch.autograd.forward_ad.dual_level(), pytest.raises(RuntimeError):
        fused.rmsnorm(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)), w)


def test_errors_keep_their_class():
    q = torch.zeros(128, 2, 128, device="cuda", dtype=torch.bfloat16)[:, :, :64]
    with pytest.raises(AssertionError):
        attention.flash_attention(q, q, q, 1)     # heads with a gap between them
    x, w = torch.randn(4, 12, device="cuda").bfloat16().requires_grad_(), torch.ones(12, device="cuda").bfloat16()
    with pytest.raises(_lib.NativeLibraryError):
        fused.rmsnorm(x, w)                       # rows of 12 channels: no 16-byte vectors
    p = _param(_gen(), 128, 64, main=True)
    p._grad_ready_cb = lambda w: (_ for _ in ()).throw(KeyError("from the callback"))
    o = gemm.linear(torch.randn(8, 64, device="cuda").bfloat16().requires_grad_(), p)
    with pytest.raises(KeyError, match="from the callback"):
        o.backward(torch.ones_like(o))


@pytest.mark.parametrize("coeff", [None, 0.1])
def test_router_launches_are_counted_alike(monkeypatch, coeff):
    from primus_b200.ops import moe

    logits, counts = _randn(_gen(15), 64, 8), []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(_lib, "_NODES", [None])
        before = _lib.launch_count()
        moe.router_scores(logits, 2, aux_coeff=coeff)
        counts.append(_lib.launch_count() - before)
    assert counts == [1 if coeff is None else 2] * 2
