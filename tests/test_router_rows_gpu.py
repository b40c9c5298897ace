"""Routing of tokens whose scores are no numbers, or that have fewer eligible experts than selections: their experts are distinct
and exist, the counts add up, and no other token notices."""
import pytest
import torch

from primus_b200.ops import moe

pytestmark = pytest.mark.gpu
NAN, INF = float("nan"), float("inf")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("E,k,groups,group_topk", [(8, 2, 0, 0), (8, 8, 0, 0), (33, 32, 0, 0), (64, 8, 8, 1), (64, 8, 4, 2), (1024, 32, 0, 0)])
@pytest.mark.parametrize("score,pre,bias", [("softmax", False, False), ("softmax", True, False), ("sigmoid", False, False),
                                            ("sigmoid", False, True)])
def test_rows_without_scores(dtype, E, k, groups, group_topk, score, pre, bias):
    g = torch.Generator(device="cuda").manual_seed(E + k)
    T = 41                                                     # a CTA takes eight rows: every row of one, and a remainder
    clean = torch.randn(T, E, device="cuda", generator=g).to(dtype)
    b = torch.randn(E, device="cuda", generator=g) if bias else None
    bad = clean.clone()
    bad[0] = NAN
    bad[9, E // 2] = NAN                                       # (the softmax makes the whole row one)
    bad[18] = -INF
    bad[27, 1:] = -INF                                         # one expert left
    bad[28, ::2] = NAN
    bad[40, :-1] = NAN
    rows = torch.tensor([0, 9, 18, 27, 28, 40], device="cuda")
    others = torch.ones(T, dtype=torch.bool, device="cuda").index_fill(0, rows, False)

    def route(x):
        x = x.clone().requires_grad_()
        out = moe.router_scores(x, k, score, pre, b, 1.5, groups, group_topk, return_counts=True)
        out[0].backward(torch.ones_like(out[0]) * torch.arange(k, device="cuda"))
        return [t.detach() for t in out] + [x.grad]

    p, idx, full, counts, dx = route(bad)
    p0, idx0, full0, _, dx0 = route(clean)
    assert idx.min() >= 0 and idx.max() < E
    assert (idx.sort(1).values.diff(dim=1) > 0).all()
    assert torch.equal(counts, torch.bincount(idx.reshape(-1), minlength=E).int()) and counts.sum() == T * k
    for a, c in ((p, p0), (idx, idx0), (full, full0), (dx, dx0)):
        assert torch.equal(a[others], c[others])
    assert p[0].isnan().all()                                  # what is no number goes on
    if not groups:                                             # (with groups, an expert of another group comes before one of no number)
        assert p[40].isnan().any()
    if score == "softmax" and not pre:
        assert idx[27, 0] == 0 and p[27, 0] == 1.5 and (p[27, 1:] == 0).all()
