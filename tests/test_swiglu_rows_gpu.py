"""SwiGLU and its backward at the sizes where the kernels' walk over rows and vectors can go wrong: one row, one vector per row,
rows longer than a warp's round, remainders, and more vectors than threads."""
import pytest
import torch

from primus_b200.ops import _lib, fused

from .test_kernel_edges_gpu import _close_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,I", [(1, 8), (1, 14336), (700, 8), (37, 776), (768, 688), (130, 2056), (5000, 1032)])
@pytest.mark.parametrize("probs", [False, True])
@pytest.mark.parametrize("clamp", [0.0, 1.5])
@pytest.mark.parametrize("act", ["silu", "gelu"])
def test_swiglu_and_gradients(T, I, probs, clamp, act):
    g = torch.Generator(device="cuda").manual_seed(T + I)
    h1 = torch.randn(T, 2 * I, device="cuda", generator=g).bfloat16()
    dy = torch.randn(T, I, device="cuda", generator=g).bfloat16()
    p = torch.rand(T, device="cuda", generator=g) if probs else None
    kind = fused.GATE_KINDS[act]
    y, again = torch.empty_like(dy), dy.clone()
    din, din2 = torch.empty_like(h1), torch.empty_like(h1)
    dp, dp2 = (torch.empty(T, device="cuda") if probs else None for _ in range(2))
    _lib.call("swiglu_fwd", h1, p, y, T, I, clamp, kind)
    _lib.call("swiglu_bwd", dy, h1, p, din, dp, T, I, clamp, kind)
    _lib.call("swiglu_bwd_act", again, h1, p, din2, dp2, again, T, I, clamp, kind)      # over its own gradient
    assert torch.equal(again, y) and torch.equal(din, din2) and (not probs or torch.equal(dp, dp2))
    h64 = h1.double().requires_grad_()
    gate, up = h64.chunk(2, -1)
    if clamp:
        gate, up = gate.clamp(max=clamp), up.clamp(-clamp, clamp)
    a = torch.nn.functional.silu(gate) if act == "silu" else torch.nn.functional.gelu(gate, approximate="tanh")
    p64 = p.double().requires_grad_() if probs else None
    y64 = a * up * (p64[:, None] if probs else 1.0)
    y64.backward(dy.double())
    _close_bf16(y, y64.detach(), "y")
    _close_bf16(din, h64.grad, "din")
    if probs:       # fp32 sums of I products whose factors carry the exponential's 2^-21
        scale = (dy.double() * (y64 / p64[:, None]).detach()).abs().sum(1)
        assert ((dp - p64.grad).abs() <= 2.0 ** -18 * scale + 1e-6).all()
