"""RMSNorm around the row counts at which its backward changes kernel or number of CTAs."""
import pytest
import torch

from primus_b200.ops import fused

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
