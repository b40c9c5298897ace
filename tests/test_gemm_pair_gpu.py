"""The CTA-pair bf16 GEMM and its split reduction at sizes that the choice by size gives to the one-CTA kernel.  Tolerance: fp32
sums of K products in any order, 2^-24 K of the sum of their magnitudes."""
import pytest
import torch

from primus_b200.ops import _lib, gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (256, 264, 72), (264, 256, 200), (520, 1000, 64), (1000, 520, 328),
                                   (136, 264, 2056), (8, 136, 1024)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("parts", [1, 2, 5])
def test_pair_kernel_and_split_reduction(M, N, K, a_mn, b_mn, parts):
    if parts > -(-K // 64):
        pytest.skip("a part needs a K step")
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(*((K, M) if a_mn else (M, K)), device="cuda", generator=g).bfloat16()
    b = torch.randn(*((K, N) if b_mn else (N, K)), device="cuda", generator=g).bfloat16()
    A, B = (a.t() if a_mn else a).double(), (b if b_mn else b.t()).double()
    ref = A @ B
    lim = 2.0 ** -24 * K * (A.abs() @ B.abs()).max()
    ws = torch.empty(parts * -(-M // 256) * 256 * N, device="cuda")
    for mode, out, base, rounding in ((0, torch.empty(M, N, device="cuda", dtype=torch.bfloat16), 0, 2.0 ** -8),
                                      (1, torch.empty(M, N, device="cuda"), 0, 0), (2, torch.ones(M, N, device="cuda"), 1, 2.0 ** -22)):
        if parts == 1:
            gemm.launch_bf16(a, b, out, M, N, K, a_mn, b_mn, mode, 256, two_cta=True)
        else:
            _lib.call("gemm_bf16_splitk", a, b, out, ws, M, N, K, a.stride(0), b.stride(0), N, int(a_mn), int(b_mn), mode, parts,
                      _lib.status_word(a.device))
        torch.cuda.synchronize()
        _lib.check_status()
        err = (out.double() - ref - base).abs()
        assert (err <= lim + rounding * ref.abs().clamp_min(1)).all(), (mode, err.max().item())
