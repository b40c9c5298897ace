"""SwiGLU fused with quantisation against quantising the un-fused kernel's output, byte for byte, below and above the tile count
at which a CTA takes several warps per strip."""
import pytest
import torch

from primus_b200.ops import fp8, fused

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,I", [(128, 128), (512, 37 * 128), (384, 50 * 128)])          # 1, 148, 150 tiles
@pytest.mark.parametrize("clamp", [0.0, 1.5])
def test_fused_quantisation_is_that_of_the_activation(T, I, clamp):
    g = torch.Generator(device="cuda").manual_seed(T + I)
    h1 = torch.randn(T, 2 * I, device="cuda", generator=g).bfloat16()
    dact = torch.randn(T, I, device="cuda", generator=g).bfloat16()
    leaf = h1.clone().requires_grad_()
    act = fused.swiglu(leaf, None, clamp)
    act.backward(dact)
    for got, x in ((fp8.swiglu_quantize_mxfp8(h1, clamp, True, True), act.detach()),
                   (fp8.swiglu_bwd_quantize_mxfp8(h1, dact, clamp), leaf.grad)):
        want = fp8.quantize_mxfp8(x, scaling="mxfp8")
        for name in ("q_row", "sf_row", "q_col", "sf_col"):
            assert torch.equal(getattr(got, name), getattr(want, name)), name


@pytest.mark.parametrize("T,I", [(128, 128), (512, 37 * 128), (384, 50 * 128)])
@pytest.mark.parametrize("clamp", [0.0, 1.5])
def test_backward_gives_the_activation_too(T, I, clamp):
    g = torch.Generator(device="cuda").manual_seed(T + I)
    h1 = torch.randn(T, 2 * I, device="cuda", generator=g).bfloat16()
    dact = torch.randn(T, I, device="cuda", generator=g).bfloat16()
    got, act = fp8.swiglu_bwd_quantize_mxfp8(h1, dact, clamp, act=True)
    for a, b in ((got, fp8.swiglu_bwd_quantize_mxfp8(h1, dact, clamp)), (act, fp8.swiglu_quantize_mxfp8(h1, clamp, False, True))):
        for name in ("q_row", "sf_row", "q_col", "sf_col"):
            x, y = getattr(a, name), getattr(b, name)
            assert (x is None and y is None) or torch.equal(x, y), name
