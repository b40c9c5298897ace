"""Gradients that arrive as contiguous views off a 16-byte boundary."""
import pytest
import torch

from primus_b200.ops import fused

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,hq,hkv,d,off", [(1, 1, 1, 64, 1), (5, 4, 2, 128, 3), (130, 2, 1, 72, 4), (33, 2, 1, 256, 8)])
def test_qk_norm_backward_of_a_misaligned_gradient(T, hq, hkv, d, off):
    g = torch.Generator(device="cuda").manual_seed(d)
    W = (hq + 2 * hkv) * d
    qkv = torch.randn(T, W, device="cuda", generator=g).bfloat16()
    dy = torch.randn(T * W + off, device="cuda", generator=g).bfloat16()[off:].view(T, W)
    wq, wk = ((1 + 0.1 * torch.randn(d, device="cuda", generator=g)).bfloat16() for _ in range(2))
    grads = []
    for grad in (dy, dy.clone()):
        leaves = [t.clone().requires_grad_() for t in (qkv, wq, wk)]
        fused.qk_norm(*leaves, hq, hkv, d).backward(grad)
        grads.append([t.grad for t in leaves])
    for a, b in zip(*grads):
        assert torch.equal(a, b)
