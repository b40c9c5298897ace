"""Row gather and combine around the lines of their dispatch (row width, copies per token, tokens), bit for bit."""
import pytest
import torch

from primus_b200.ops import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [8, 248, 256, 264, 520, 1032])
@pytest.mark.parametrize("R,limit,scaled", [(1, None, False), (7, None, True), (1000, 517, False), (20001, 20001, True), (64, 0, False)])
def test_gather_rows(H, R, limit, scaled):
    g = torch.Generator(device="cuda").manual_seed(H + R)
    x = torch.randn(300, H, device="cuda", generator=g).bfloat16()
    src = torch.randint(-1, 300, (R,), device="cuda", generator=g, dtype=torch.int32)
    scale = torch.rand(R, device="cuda", generator=g) if scaled else None
    lim = None if limit is None else torch.tensor([limit], device="cuda", dtype=torch.int32)
    out = torch.full((R, H), 7.0, device="cuda").bfloat16()
    _lib.call("moe_gather_rows", x, src, scale, out, R, H, lim)
    want = x[src.clamp_min(0).long()].float()
    if scaled:
        want = want * scale[:, None]
    want = torch.where((src >= 0)[:, None], want, torch.zeros((), device="cuda")).bfloat16()
    if limit is not None:
        want[limit:] = 7.0
    assert torch.equal(out, want)


@pytest.mark.parametrize("H", [8, 248, 256, 264, 512, 520, 1032])
@pytest.mark.parametrize("topk", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("T", [1, 130, 2367, 2368, 16383, 16385])
def test_combine_rows(H, topk, T):
    g = torch.Generator(device="cuda").manual_seed(H + topk + T)
    y = torch.randn(500, H, device="cuda", generator=g).bfloat16()
    pos = torch.randint(-1, 500, (T, topk), device="cuda", generator=g, dtype=torch.int32)
    out = torch.full((T, H), 7.0, device="cuda").bfloat16()
    _lib.call("moe_combine_rows", y, pos, out, T, topk, H)
    acc = torch.zeros(T, H, device="cuda")
    for k in range(topk):
        p = pos[:, k]
        acc = torch.where((p >= 0)[:, None], acc + y[p.clamp_min(0).long()].float(), acc)
    assert torch.equal(out, acc.bfloat16())
