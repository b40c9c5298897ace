"""Kernels that may start before the one in front of them has ended: a chain of launches gives the same bits as the same chain with
the device idle between any two of them, in a stream, as a captured graph, and in several streams at once."""
import threading

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
    wr, we = rnd(8, H) / H ** 0.5, rnd(8, H, H) / H ** 0.5

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
            # (counts that are added to memory set to zero just before, and everything that follows from them)
            probs, idx, full, counts, aux = moe.router_scores(logits, 2, return_counts=True, aux_coeff=0.1)
            step()
            sched, pos, src_token, perm = moe.local_plan(probs, idx, counts, 2)
            step()
            rows = moe.gather_rows(z, src_token, pos)
            step()
            e = moe.grouped_linear(rows, we, sched)
            step()
            m = moe.combine_rows(e, pos, src_token)
            step()
            outs += [dq, dk, dv, probs, idx, full, counts, aux, pos, src_token, perm, m]
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


def test_chains_on_several_streams():
    """Each thread's chain runs on a stream of its own, beside the others'."""
    shapes = [(1024, 512), (2048, 256), (128, 2048)]
    with torch.no_grad():
        runs = [_chain(T, H, lambda: None) for T, H in shapes]
        wants = [_chain(T, H, torch.cuda.synchronize)() for T, H in shapes]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in shapes], [None] * len(shapes)
    start = threading.Barrier(len(shapes))

    def work(i):
        with torch.no_grad(), torch.cuda.stream(streams[i]):
            start.wait(60)
            for _ in range(4):
                got[i] = runs[i]()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(shapes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for outs, want in zip(got, wants):
        assert len(outs) == len(want) and all(torch.equal(a, b) for a, b in zip(outs, want))


def test_chains_that_fork_and_join():
    """Two chains between an event that both wait for and a kernel that waits for both, in streams and as a graph."""
    runs = [_chain(256, 512, lambda: None), _chain(512, 512, lambda: None)]
    w = torch.ones(512, device="cuda").bfloat16()
    x = torch.randn(256, 512, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).bfloat16()
    side = torch.cuda.Stream()

    def work(step):
        with torch.no_grad():
            first = fused.rmsnorm(x, w)
            step()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                b = runs[1]()
                second = fused.rmsnorm(first, w)
            step()
            a = runs[0]()
            step()
            torch.cuda.current_stream().wait_stream(side)
            last = fused.rmsnorm(a[-1], w, residual=second)[0]      # (launched dependent, behind two kernels)
            step()
        return a + b + [second, last]

    want = [t.clone() for t in work(torch.cuda.synchronize)]
    torch.cuda.synchronize()
    for a, b in zip(work(lambda: None), want):
        assert torch.equal(a, b)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = work(lambda: None)
    for _ in range(3):
        for t in got:
            t.zero_()
        graph.replay()
        for a, b in zip(got, want):
            assert torch.equal(a, b)
