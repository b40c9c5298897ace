"""RMSNorm around the row counts at which its backward changes kernel or number of CTAs."""
import pytest
import torch

from primus_b200.ops import _lib, fused, layers

from .test_kernel_edges_gpu import _close_bf16, _gen, _rms64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [7, 149, 296, 592, 593, 1184, 2367, 2368])
@pytest.mark.parametrize("H", [64, 256, 512, 520, 1024, 1032, 4096, 8200])
def test_norm_and_gradients(rows, H):
    g = _gen(rows + H)
    x, r, dy, ds = (torch.randn(rows, H, device="cuda", generator=g).bfloat16() for _ in range(4))
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).bfloat16()
    leaves = [x.clone().requires_grad_(), w.clone().requires_grad_(), r.clone().requires_grad_()]
    y, s = fused.rmsnorm(leaves[0], leaves[1], 1e-5, leaves[2])
    torch.autograd.backward([y, s], [dy, ds])
    s64, w64 = (x + r).double().requires_grad_(), w.double().requires_grad_()
    y64 = _rms64(s64, w64)
    torch.autograd.backward([y64, s64 * 1.0], [dy.double(), ds.double()])
    _close_bf16(y.detach(), y64.detach(), "y")
    _close_bf16(leaves[0].grad, s64.grad, "dx")
    _close_bf16(leaves[1].grad, w64.grad, "dw")


@pytest.mark.parametrize("rows, H", [(1, 8), (37, 64), (700, 520), (129, 1024), (200, 2048), (33, 4104), (40, 8192), (5, 16384)])
@pytest.mark.parametrize("layer", [False, True])
def test_gradients_of_two_leaves_are_two_tensors(rows, H, layer):
    """The shared input gradient is written twice where both inputs are leaves, and equals the one that producers share."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    x, r, dy, ds = (torch.randn(rows, H, device="cuda", generator=g).bfloat16() for _ in range(4))
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).bfloat16()
    proj = (torch.randn(128, H, device="cuda", generator=g) * 0.02).bfloat16()

    def grads(leaves):
        a, b, p = x.clone().requires_grad_(), r.clone().requires_grad_(), torch.nn.Parameter(w.clone())
        ia, ib = (a, b) if leaves else (a * 1, b * 1)
        if layer:
            y, s = layers.norm_linear(ia, ib, p, torch.nn.Parameter(proj.clone()), 1e-5)
            torch.autograd.backward([y, s], [dy[:, :1].expand(rows, 128).contiguous(), ds])
        else:
            y, s = fused.rmsnorm(ia, p, 1e-5, ib)
            torch.autograd.backward([y, s], [dy, ds])
        return a.grad, b.grad, p.grad

    two, shared = grads(True), grads(False)
    assert two[0].data_ptr() != two[1].data_ptr()
    for t, u in zip(two, shared):
        assert torch.equal(t, u)
    assert torch.equal(two[0], two[1])


@pytest.mark.parametrize("rows, H", [(3, 64), (129, 1024), (40, 4104)])
@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("layer", [False, True])
def test_gradients_of_a_column_slice(rows, H, residual, layer):
    """Rows with a pitch: outputs and gradients are those of a dense copy."""
    g = torch.Generator(device="cuda").manual_seed(H)
    wide, other = (torch.randn(rows, H + 24, device="cuda", generator=g).bfloat16() for _ in range(2))
    dy, ds = (torch.randn(rows, H, device="cuda", generator=g).bfloat16() for _ in range(2))
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).bfloat16()
    proj = (torch.randn(128, H, device="cuda", generator=g) * 0.02).bfloat16()

    def run(copy):
        a, b = (t[:, 8:8 + H] for t in (wide, other))
        a, b = (t.clone() if copy else t.detach() for t in (a, b))
        leaves = [a.requires_grad_()] + ([b.requires_grad_()] if residual else []) + [torch.nn.Parameter(w.clone())]
        if layer:
            y, s = layers.norm_linear(a, b if residual else None, leaves[-1], torch.nn.Parameter(proj.clone()), 1e-5)
            torch.autograd.backward([y, s], [dy[:, :1].expand(rows, 128).contiguous(), ds])
        elif residual:
            y, s = fused.rmsnorm(a, leaves[-1], 1e-5, b)
            torch.autograd.backward([y, s], [dy, ds])
        else:
            y = fused.rmsnorm(a, leaves[-1], 1e-5)
            y.backward(dy)
        return [y.detach()] + [t.grad for t in leaves]

    for t, u in zip(run(False), run(True)):
        assert torch.equal(t, u)


@pytest.mark.parametrize("H", [64, 4096])
def test_gain_gradient_of_no_rows_is_zero(H):
    for _ in range(4):
        junk = [torch.full((H,), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(8)]
        del junk                                # what the gradient's memory held before
        x, r = (torch.empty(0, H, device="cuda", dtype=torch.bfloat16).requires_grad_() for _ in range(2))
        p = torch.nn.Parameter(torch.ones(H, device="cuda", dtype=torch.bfloat16))
        y, s = fused.rmsnorm(x, p, 1e-5, r)
        torch.autograd.backward([y, s], [torch.ones_like(y), torch.ones_like(s)])
        assert p.grad.shape == (H,) and not p.grad.any() and x.grad.shape == (0, H)


@pytest.mark.parametrize("rows, H", [(1, 72), (37, 128), (700, 520), (129, 1024), (3000, 1024), (200, 2048), (33, 4104), (40, 8192),
                                     (5, 16384)])
@pytest.mark.parametrize("residual, two", [(False, False), (True, False), (True, True)])
def test_backward_gives_the_normalised_rows_again(rows, H, residual, two):
    """With ``y`` the backward writes what the forward wrote, and its gradients stay the same to the last bit."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    x, dy, ds = (torch.randn(rows, H, device="cuda", generator=g).bfloat16() for _ in range(3))
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).bfloat16()
    y, rstd = torch.empty_like(x), torch.empty(rows, device="cuda")
    _lib.call("rmsnorm_fwd", x, None, w, y, None, rstd, rows, H, H, H, 1e-5)
    again = torch.full_like(x, float("nan"))
    dres = ds if residual else None
    got = fused.norm_backward(dy, x, w, rstd, dres, None, two, x.shape, again)
    want = fused.norm_backward(dy, x, w, rstd, dres, None, two, x.shape)
    assert torch.equal(again, y)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    assert (got[0].data_ptr() != got[1].data_ptr()) == two


@pytest.mark.parametrize("rows", [1183, 1184, 1185, 2367, 2368, 2400])
@pytest.mark.parametrize("H", [1024, 1032, 1544, 2048, 2056, 4096, 4104, 8192, 8200, 16384])
@pytest.mark.parametrize("residual", [False, True])
def test_forward_around_the_rows_that_ctas_stay_for(rows, H, residual):
    """The kernel of many rows gives the bits of the one for few (the same rows in two halves)."""
    g = _gen(rows + H)
    x, r = (torch.randn(rows, H, device="cuda", generator=g).bfloat16() for _ in range(2))
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).bfloat16()

    def run(a, b):
        y, s, rstd = torch.empty_like(a), torch.empty_like(a), torch.empty(a.shape[0], device="cuda")
        _lib.call("rmsnorm_fwd", a, b if residual else None, w, y, s if residual else None, rstd, a.shape[0], H, H, H, 1e-5)
        return (y, s, rstd) if residual else (y, rstd)

    whole = run(x, r)
    halves = [run(x[i:i + 600].contiguous(), r[i:i + 600].contiguous()) for i in range(0, rows, 600)]
    for i, t in enumerate(whole):
        assert torch.equal(t, torch.cat([h[i] for h in halves])), i
    s64 = (x + r if residual else x).double()
    _close_bf16(whole[0], _rms64(s64, w.double()), "y")
