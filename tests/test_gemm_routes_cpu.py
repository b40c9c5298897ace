"""Which of its kernels a bf16 GEMM takes."""
import pytest

from primus_b200.ops import gemm

ONE, PAIR = gemm._ONE_CTA, gemm._CTA_PAIR


@pytest.mark.parametrize("M,N,K,route", [
    (256, 256, 256, ONE), (512, 512, 512, ONE), (2048, 2048, 1024, ONE),          # one wave: a launch of clusters costs more
    (304, 10648, 7360, ONE), (528, 6776, 9440, ONE),       # 256-row tiles would need a second wave for a few rows
    (4096, 4096, 128, ONE), (768, 32000, 256, ONE),        # a few K steps
    (2048, 1024, 2048, ONE), (1536, 1536, 2048, ONE),      # half the pairs idle, but the parts' sums would cost more
    (4096, 4096, 4096, PAIR), (8192, 14336, 4096, PAIR), (4096, 128256, 2048, PAIR),
    (128, 256, 512, ONE), (100, 100, 100, ONE),
    (8192, 4096, 128256, ONE), (8192, 4096, 28672, PAIR), (4096, 2048, 128256, PAIR),      # pairs drift apart over long K
])
def test_route_of_a_size(M, N, K, route):
    assert gemm._bf16_route(M, N, K, False, K, 2, 0) == route


def test_route_splits_long_reductions_of_few_tiles():
    for M, N, K in ((768, 256, 32000), (100, 2048, 8192), (16, 4096, 4096), (1536, 1536, 8192)):
        parts = gemm._bf16_route(M, N, K, False, K, 2, 0)
        assert 1 < parts <= -(-K // 64)
        assert parts * -(-M // 256) * -(-N // 256) <= 74
        assert gemm._bf16_route(M, N - 2, K, False, K, 2, 0) < 2          # the sums are added four columns at a time
        assert gemm._bf16_route(M, N, K, False, K, 2, 64) < 2             # SMs left to other work


def test_route_leaves_the_pair_kernel_to_calls_with_two_ctas():
    assert gemm._bf16_route(8192, 8192, 8192, False, 8192, 2, 1) == ONE
    assert gemm._bf16_route(8192, 8192, 8192, False, 8192, 2, 32) == PAIR


def test_route_of_a_gemm_that_its_output_bounds():
    assert gemm._bf16_route(768, 32000, 256, True, 32000, 8, 0) == ONE
    assert gemm._bf16_route(8192, 4096, 1024, True, 4096, 8, 0) == PAIR
