"""Kernels that may start before the one in front of them has ended: a chain of launches gives the same bits as the same chain with
the device idle between any two of them, in a stream and as a captured graph."""
import pytest
import torch

from primus_b200.ops import attention, fp8, fused, gemm, moe

pytestmark = pytest.mark.gpu


def _chain(T, H, step):
    """A dozen dependent launches, each of which overwrites or frees what the one before has read; `step` runs between them."""
    g = torch.Generator(device="cuda").manual_seed(T + H)

    def rnd(*shape):
        return torch.randn(*shape, device="cuda", generator=g).bfloat16()

    x, w1, w2, wn = rnd(T, H), rnd(2 * H, H) / H ** 0.5, rnd(H, H) / H ** 0.5, 1 + 0.1 * rnd(H)
    heads = H // 64
    cos, sin = fused.rope_tables(T, 64, 1e4, "cuda")
    wr = rnd(8, H) / H ** 0.5

    def run():
        y, outs = x.clone(), []
        for _ in range(4):
            n = fused.rmsnorm(y, wn)
            step()
            q = n.view(T, heads, 64).clone()
            step()
            fused.rope_inplace_(q, cos, sin)
            step()
            o, lse = attention.flash_attn_fwd(q, q, q, 1, True, 0.125)[:2]
            step()
            dq, dk, dv = attention.flash_attn_bwd(n.view(T, heads, 64), q, q, q, o, lse, 1, True, 0.125)
            step()
            h = gemm.gemm(o.view(T, H), w1)
            step()
            a = fused.swiglu(h)
            step()
            qa, qw = fp8.quantize_mxfp8(a), fp8.quantize_mxfp8(w2)
            step()
            z = fp8.gemm_mxfp8(qa.q_row, qa.sf_row, qw.q_row, qw.sf_row, T, H, H)
            step()
            logits = gemm.gemm(z, wr)
            step()
            probs, idx, counts = moe.router_scores(logits.float(), 2)[:3]
            step()
            outs += [dq, dk, dv, probs]
            y = z
            y.add_(dv.view(T, H))
            step()
        return outs + [y]

    return run


@pytest.mark.parametrize("T,H", [(128, 256), (1024, 512), (4096, 2048)])
def test_chain_in_stream_order(T, H):
    with torch.no_grad():
        want = _chain(T, H, torch.cuda.synchronize)()
        run = _chain(T, H, lambda: None)
        for _ in range(3):
            for a, b in zip(run(), want):
                assert torch.equal(a, b)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = run()
        for _ in range(3):
            for t in got:
                t.zero_()
            graph.replay()
            for a, b in zip(got, want):
                assert torch.equal(a, b)
