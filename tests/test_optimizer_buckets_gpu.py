"""Several tensors or buckets in one launch against one call each, bit for bit: below, at and above the number a launch takes."""
import pytest
import torch

from primus_b200.ops import optim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 3, 4, 5, 32, 33])
@pytest.mark.parametrize("dtype,off", [(torch.float32, 0), (torch.float32, 1), (torch.bfloat16, 0)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_gradient_norm_of_several_tensors(count, dtype, off, accumulate):
    g = torch.Generator(device="cuda").manual_seed(count)
    xs = [torch.randn(1 + 977 * i * i + off, device="cuda", generator=g).to(dtype)[off:] for i in range(count)]
    xs[count // 2] = xs[count // 2][:0]
    want, got = torch.full((1,), 0.5, device="cuda"), torch.full((1,), 0.5, device="cuda")
    coef, norm, skip = (torch.zeros(1, device="cuda", dtype=d) for d in (torch.float32, torch.float32, torch.int32))
    for i, x in enumerate(xs):
        optim.sumsq_(x, want, accumulate=accumulate or i > 0)
    optim.grad_norm_(xs, got, accumulate, clip=dict(max_norm=1.0, coef=coef, norm_out=norm, skip=skip, check_finite=True, spike=0.25))
    assert torch.equal(got, want)
    c, n, s = torch.zeros_like(coef), torch.zeros_like(norm), torch.zeros_like(skip)
    optim.clip_coef_(want, 1.0, c, n, skip=s, check_finite=True, spike=0.25)
    assert torch.equal(coef, c) and torch.equal(norm, n) and torch.equal(skip, s)
    optim.grad_norm_(xs, got, accumulate)
    assert torch.equal(coef, c)


@pytest.mark.parametrize("count", [1, 2, 32, 34])
@pytest.mark.parametrize("grad_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("state", [torch.float32, torch.bfloat16])
def test_adamw_of_several_buckets(count, grad_dtype, state):
    g = torch.Generator(device="cuda").manual_seed(count)
    hyper = dict(lrs=[1e-3, 2e-3, 3e-3, 4e-3], beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=3)

    def bucket(i):
        n = (1, 4099, 8192, 8193, 30000)[i % 5]
        cut = n // 8 * 4
        ranges = [(0, cut, 1.0, i % 4), (cut, n, 0.0, 0)] if cut else [(0, n, 1.0, i % 4)]
        return (torch.randn(n, device="cuda", generator=g), torch.randn(n, device="cuda", generator=g).to(state),
                torch.rand(n, device="cuda", generator=g).to(state), torch.randn(n, device="cuda", generator=g).to(grad_dtype),
                torch.zeros(n, device="cuda", dtype=torch.bfloat16), optim.range_table(ranges, 0, n, "cuda"))

    one = [bucket(i) for i in range(count)]
    many = [tuple(t.clone() for t in b[:5]) + (b[5],) for b in one]
    for b in one:
        optim.adamw_ranges_(*b, **hyper)
    optim.adamw_buckets_(many, **hyper)
    for a, b in zip(one, many):
        for x, y in zip(a[:5], b[:5]):
            assert torch.equal(x, y)
