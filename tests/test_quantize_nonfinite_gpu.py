"""Non-finite values in the block quantisers: a maximum ignores NaN, so a block of nothing but NaN is scaled like a block of
zeros, in both directions and by every kernel that quantises 32-blocks."""
import pytest
import torch

from primus_b200.ops import fp8

pytestmark = pytest.mark.gpu


def _scales(sf, rows, cols):
    """UE8M0 bytes [rows, cols / 32] of the operand layout with `rows` along its first dimension."""
    mn = torch.arange(rows, device="cuda")[:, None].expand(rows, cols // 32)
    kb = torch.arange(cols // 32, device="cuda")[None, :].expand(rows, cols // 32)
    return sf[fp8.sf_offsets(mn, kb, cols // 128).reshape(-1)].view(rows, cols // 32)


def _check(q, x):
    R, C = x.shape
    nan_rows = x.isnan().view(R, C // 32, 32).all(-1)
    nan_cols = x.isnan().view(R // 32, 32, C).all(1).t()
    assert nan_rows.any() and nan_cols.any()
    assert (_scales(q.sf_row, R, C)[nan_rows] == 0).all(), "row direction"
    assert (_scales(q.sf_col, C, R)[nan_cols] == 0).all(), "column direction"


@pytest.mark.parametrize("R,C", [(128, 128), (256, 384)])
@pytest.mark.parametrize("scaling", ["mxfp8", "mxfp4"])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_nan_blocks_have_the_smallest_scale(R, C, scaling, sign):
    x = torch.randn(R, C, device="cuda", generator=torch.Generator(device="cuda").manual_seed(R)).bfloat16()
    x[3, 32:64] = x[R - 1, C - 32:] = x[32:64, 5] = x[64:96, 64:96] = torch.copysign(torch.tensor(float("nan")), torch.tensor(sign))
    x[7, :31] = float("nan")                 # a NaN beside a number does not count
    x[8, 2] = float("inf")
    q = fp8.quantize_mxfp8(x, scaling=scaling)
    _check(q, x)
    assert _scales(q.sf_row, R, C)[7, 0] != 0
    finite = x.isfinite().view(R, C // 32, 32).all(-1)
    assert torch.equal(_scales(q.sf_row, R, C)[finite],
                       _scales(fp8.quantize_mxfp8_ref(x, scaling=scaling).sf_row, R, C)[finite])


def test_nan_blocks_of_the_fused_activations():
    T, I = 128, 256
    h1 = torch.randn(T, 2 * I, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).bfloat16()
    dact = torch.randn(T, I, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)).bfloat16()
    h1[2, :64] = h1[96:, 40] = float("nan")                     # gate: the activation and both gradients of it
    gate, up = h1.float().chunk(2, -1)
    act = torch.nn.functional.silu(gate) * up
    _check(fp8.swiglu_quantize_mxfp8(h1, rowwise=True, colwise=True), act)
    _check(fp8.swiglu_bwd_quantize_mxfp8(h1, dact), torch.cat([act, act], -1))


@pytest.mark.parametrize("scaling", ["mxfp8", "mxfp4"])
def test_scale_of_every_maximum(scaling):
    """Block maxima of all bf16 magnitudes from zero over the subnormals to infinity, against the scale and bytes of the plain
    formula, in both directions."""
    g = torch.Generator().manual_seed(3)
    bits = torch.arange(32768).clamp(max=0x7f80)
    part = (bits[:, None] * torch.rand(32768, 32, generator=g)).long().clamp(max=0x7f7f)     # smaller in the order of the bits
    part[:, 5] = bits
    part |= torch.randint(0, 2, part.shape, generator=g) << 15
    rows = torch.where(part > 32767, part - 65536, part).to(torch.int16).view(torch.bfloat16).view(1024, 1024)
    for x, names in ((rows, ("q_row", "sf_row")), (rows.t().contiguous(), ("q_col", "sf_col"))):
        got, want = fp8.quantize_mxfp8(x.cuda(), scaling=scaling), fp8.quantize_mxfp8_ref(x, scaling=scaling)
        for n in names:
            assert torch.equal(getattr(got, n).cpu(), getattr(want, n)), n
