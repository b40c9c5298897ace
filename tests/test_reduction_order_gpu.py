"""The squared sum behind the gradient norm adds in one fixed order: a change of that order moves the norm by a last bit,
the clip coefficient with it, and through it every moment and weight of the optimizer."""
import pytest
import torch

from primus_b200.ops import optim

pytestmark = pytest.mark.gpu

BLOCKS, WIDTH = 1184, 512


def _tree(s):
    """Sum over the last dimension (a power of two) by halves: s[i] + s[i + n / 2]."""
    while s.shape[-1] > 1:
        h = s.shape[-1] // 2
        s = s[..., :h] + s[..., h:]
    return s[..., 0]


def _block(s):
    return _tree(_tree(s.unflatten(-1, (16, 32))))


def _ordered(x):
    """Chain j adds the squares of the elements j, j + BLOCKS * WIDTH, ... in turn; blocks of WIDTH chains fold into
    partial sums, and those fold the same way.  Squares of bf16 values are exact in fp32, so a fused and a separate
    multiplication agree bit for bit."""
    chains = BLOCKS * WIDTH
    sq = torch.zeros(-(-x.numel() // chains) * chains)
    sq[:x.numel()] = x.float() ** 2
    s = torch.zeros(chains)
    for row in sq.view(-1, chains):
        s = s + row
    partial = torch.zeros(3 * WIDTH)
    partial[:BLOCKS] = _block(s.view(BLOCKS, WIDTH))
    t = torch.zeros(WIDTH)
    for row in partial.view(3, WIDTH):
        t = t + row
    return _block(t)


@pytest.mark.parametrize("n", [1, 7, 511, 4096, BLOCKS * WIDTH - 3, BLOCKS * WIDTH + 5, 9 * BLOCKS * WIDTH + 1234567])
@pytest.mark.parametrize("off", [0, 1, 2, 4, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_squared_sum_order(n, off, dtype):
    x = torch.randn(n, generator=torch.Generator().manual_seed(n)).bfloat16()
    d = torch.zeros(n + off, dtype=dtype, device="cuda")[off:]
    d.copy_(x)
    out = torch.full((1,), 0.25, device="cuda")
    optim.sumsq_(d, out)
    want = _ordered(x)
    assert out.item() == want.item()
    optim.sumsq_(d, out, accumulate=True)
    assert out.item() == (want + want).item()
