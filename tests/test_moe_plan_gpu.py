"""Routing and layout of a MoE layer in their fused forms against the separate ones, around the sizes of a warp, a CTA
and a step of the kernels."""
import pytest
import torch

from primus_b200.ops import moe as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,k", [(1, 8, 1), (7, 8, 2), (64, 33, 4), (513, 64, 8), (1000, 256, 8), (40, 1024, 32)])
@pytest.mark.parametrize("score,pre", [("softmax", False), ("softmax", True), ("sigmoid", False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_load_balancing_loss_of_the_router(T, E, k, score, pre, dtype):
    g = torch.Generator(device="cuda").manual_seed(T + E)
    logits = torch.randn(T, E, device="cuda", generator=g).to(dtype)
    dp, coeff = torch.randn(T, k, device="cuda", generator=g), 0.37
    a = logits.clone().requires_grad_()
    probs, idx, full, counts, aux = M.router_scores(a, k, score, pre, return_counts=True, aux_coeff=coeff)
    assert torch.equal(counts, torch.bincount(idx.reshape(-1), minlength=E).int()) and counts.dtype == torch.int32
    torch.autograd.backward([probs, aux], [dp, torch.full_like(aux, 3.0)])
    b = logits.clone().requires_grad_()
    probs2, idx2, full2, counts2 = M.router_scores(b, k, score, pre, return_counts=True)
    assert torch.equal(probs, probs2) and torch.equal(idx, idx2) and torch.equal(full, full2) and torch.equal(counts, counts2)
    want = M.load_balancing_loss(full2.double(), idx2, E, k, coeff)
    torch.autograd.backward([probs2, want.float()], [dp, torch.full_like(aux, 3.0)])
    assert abs(aux.item() - want.item()) <= 2.0 ** -20 * abs(want.item())       # fp32 sums of positive terms in a tree
    # one rounding to the logits' type, and fp32 roundings of terms that may cancel
    tol = (2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -18) * (b.grad.abs() + 2.0 ** -8 * b.grad.abs().max())
    assert ((a.grad.double() - b.grad.double()).abs() <= tol).all()


@pytest.mark.parametrize("T,E,k", [(1, 8, 1), (64, 8, 2), (2048, 8, 8), (2049, 64, 8), (37, 1024, 3), (5000, 16, 7)])
@pytest.mark.parametrize("skew", [False, True])
def test_local_plan(T, E, k, skew):
    g = torch.Generator(device="cuda").manual_seed(T)
    idx = torch.randint(0, 1 if skew else E, (T, k), device="cuda", generator=g)
    probs = torch.rand(T, k, device="cuda", generator=g)
    counts = torch.bincount(idx.reshape(-1), minlength=E).int()
    dout = torch.randn(M.rows_capacity(T * k, E), device="cuda", generator=g)
    a, b = probs.clone().requires_grad_(), probs.clone().requires_grad_()
    sched, pos, src_token, perm = M.local_plan(a, idx, counts, k)
    perm.backward(dout)
    want = M.build_schedule(counts, M.rows_capacity(T * k, E))
    src, pos2, src_token2 = M.token_maps(idx.reshape(-1), want, k)
    perm2 = M.permute_probs(b, src, pos2)
    perm2.backward(dout)
    for n in ("padded", "row_start", "mblock_expert", "total_rows", "rows_cap"):
        u, v = getattr(sched, n), getattr(want, n)
        assert u == v if isinstance(u, int) else torch.equal(u, v), n
    assert torch.equal(pos.reshape(-1), pos2) and torch.equal(src_token, src_token2)
    assert torch.equal(perm, perm2) and torch.equal(a.grad, b.grad)
