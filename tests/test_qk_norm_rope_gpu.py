"""Per-head norms with the rotary embedding in the same pass against the two passes, at the sizes where lanes, head rows or tokens
leave a group part empty.  Bit for bit where the whole head rotates; otherwise lanes own other channels, and a row's sum in another
order can move a result by one rounding."""
import pytest
import torch

from primus_b200.ops import fused

from .test_kernel_edges_gpu import _close_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,hq,hkv,d,rot", [(1, 1, 1, 64, 64), (37, 3, 1, 64, 32), (130, 4, 2, 128, 128), (5, 1, 2, 128, 16),
                                            (33, 2, 2, 192, 192), (65, 5, 1, 96, 48), (700, 32, 4, 128, 128), (9, 2, 1, 256, 256)])
@pytest.mark.parametrize("positions", [False, True])
@pytest.mark.parametrize("main_grad", [False, True])
def test_one_pass_equals_two(T, hq, hkv, d, rot, positions, main_grad):
    g = torch.Generator(device="cuda").manual_seed(T + d)
    W = (hq + 2 * hkv) * d
    x = torch.randn(T, W, device="cuda", generator=g).bfloat16()
    dy = torch.randn(T, W, device="cuda", generator=g).bfloat16()
    gains = [(1 + 0.1 * torch.randn(d, device="cuda", generator=g)).bfloat16() for _ in range(2)]
    cos, sin = fused.rope_tables(2 * T, rot, 1e4, "cuda")
    pos = torch.randint(0, 2 * T, (T,), device="cuda", generator=g, dtype=torch.int32) if positions else None

    def leaves():
        ps = [torch.nn.Parameter(w.clone()) for w in gains]
        if main_grad:
            for p in ps:
                p.main_grad = torch.ones(d, device="cuda")
        return x.clone().requires_grad_(), ps

    def turn(t, back):
        t = t.clone()
        fused.rope_inplace_(t[:, :(hq + hkv) * d].view(T, hq + hkv, d), cos, sin, pos, rot, backward=back)
        return t

    a, pa = leaves()
    got = fused.qk_norm_rope(a, *pa, hq, hkv, d, 1e-5, cos, sin, pos, rot)
    got.backward(dy)
    b, pb = leaves()
    want = fused.qk_norm(b, *pb, hq, hkv, d, 1e-5)
    want.backward(turn(dy, True))
    pairs = [(got.detach(), turn(want.detach(), False)), (a.grad, b.grad)]
    pairs += [(p.main_grad, q.main_grad) if main_grad else (p.grad, q.grad) for p, q in zip(pa, pb)]
    for i, (u, v) in enumerate(pairs):
        if rot == d:
            assert torch.equal(u, v), i
        else:
            _close_bf16(u, v, i)


def test_tables_the_kernel_cannot_read_are_left_to_the_two_passes():
    x = torch.randn(4, 4 * 64, device="cuda").bfloat16()
    w = torch.ones(64, device="cuda").bfloat16()
    cos, sin = fused.rope_tables(8, 64, 1e4, "cuda")

    def call(**kw):
        a = dict(cos=cos, sin=sin, pos=None, rot_dim=64, **kw) if "rot_dim" not in kw else dict(cos=cos, sin=sin, pos=None, **kw)
        return fused.qk_norm_rope(x, w, w, 2, 1, 64, 1e-5, **a)

    assert call() is not None
    assert call(rot_dim=72) is None and call(rot_dim=24) is None and call(rot_dim=0) is None
    for bad in (dict(cos=None), dict(cos=cos.double()), dict(sin=sin.t().contiguous().t()), dict(pos=torch.arange(4, device="cuda"))):
        a = dict(cos=cos, sin=sin, pos=None, rot_dim=64)
        a.update(bad)
        assert fused.qk_norm_rope(x, w, w, 2, 1, 64, 1e-5, **a) is None


@pytest.mark.parametrize("columns", [3 * 64, 64])
def test_rows_of_fewer_heads_are_not_read_past_their_end(columns):
    x = torch.zeros(4, 8 * 64, device="cuda").bfloat16()[:, :columns]        # (of 2 query and 2 + 2 key / value heads)
    w = torch.ones(64, device="cuda").bfloat16()
    with pytest.raises(RuntimeError):
        fused.qk_norm(x, w, w, 2, 2, 64)
    cos, sin = fused.rope_tables(8, 64, 1e4, "cuda")
    assert fused.qk_norm_rope(x, w, w, 2, 2, 64, 1e-5, cos, sin, None, 64) is None
