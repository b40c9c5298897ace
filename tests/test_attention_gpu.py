"""Flash attention kernels vs an fp32 softmax(QK^T)V reference (GQA, MHA, MLA shapes; causal and full)."""
import math

import pytest
import torch

from primus_b200.ops import _lib
from primus_b200.ops import attention as A

pytestmark = pytest.mark.gpu

CASES = [
    # batch, seq, hq, hkv, dqk, dv, causal
    (1, 128, 2, 2, 128, 128, True),
    (1, 512, 4, 2, 128, 128, True),
    (2, 384, 4, 1, 128, 128, True),
    (1, 256, 2, 2, 128, 128, False),
    (1, 512, 4, 2, 64, 64, True),
    (1, 384, 2, 2, 192, 128, True),
]


def _inputs(batch, seq, hq, hkv, dqk, dv, packed=False, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    T = batch * seq
    if packed and dqk == dv:
        qkv = torch.randn(T, (hq + 2 * hkv) * dqk, device="cuda", generator=g).bfloat16()
        q = qkv[:, : hq * dqk].view(T, hq, dqk)
        k = qkv[:, hq * dqk: (hq + hkv) * dqk].view(T, hkv, dqk)
        v = qkv[:, (hq + hkv) * dqk:].view(T, hkv, dv)
        return q, k, v
    q = torch.randn(T, hq, dqk, device="cuda", generator=g).bfloat16()
    k = torch.randn(T, hkv, dqk, device="cuda", generator=g).bfloat16()
    v = torch.randn(T, hkv, dv, device="cuda", generator=g).bfloat16()
    return q, k, v


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("packed", [False, True])
def test_flash_attn_forward(case, packed):
    batch, seq, hq, hkv, dqk, dv, causal = case
    q, k, v = _inputs(batch, seq, hq, hkv, dqk, dv, packed)
    scale = 1.0 / math.sqrt(dqk)
    o, lse = A.flash_attn_fwd(q, k, v, batch, causal, scale)
    torch.cuda.synchronize()
    _lib.check_status()
    o_ref, lse_ref = A.attention_ref(q, k, v, batch, causal, scale)
    assert (o.float() - o_ref.float()).abs().max().item() <= 2e-2
    assert (lse - lse_ref).abs().max().item() <= 2e-2


@pytest.mark.parametrize("case", CASES)
def test_flash_attn_backward(case):
    batch, seq, hq, hkv, dqk, dv, causal = case
    q, k, v = _inputs(batch, seq, hq, hkv, dqk, dv, seed=1)
    q.requires_grad_(), k.requires_grad_(), v.requires_grad_()
    o = A.flash_attention(q, k, v, batch, causal)
    do = torch.randn_like(o)
    o.backward(do)
    torch.cuda.synchronize()
    _lib.check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    o_ref, _ = A.attention_ref(qr, kr, vr, batch, causal)
    o_ref.backward(do.float())
    for name, a, b in (("dq", q.grad, qr.grad), ("dk", k.grad, kr.grad), ("dv", v.grad, vr.grad)):
        err = (a.float() - b).abs().max().item()
        tol = 3e-2 * b.abs().max().item() + 2e-2
        assert err <= tol, f"{name}: err {err} tol {tol}"


def test_flash_attn_fwd_bwd_at_the_benchmark_length():
    """seq 8192 (64 key blocks, many waves of streamed tiles per CTA), one GQA group of the Llama-3.1-8B shape
    (4 query heads on 1 KV head, d 128), forward and backward against the fp32 reference."""
    batch, seq, hq, hkv, d = 1, 8192, 4, 1, 128
    q, k, v = _inputs(batch, seq, hq, hkv, d, d, seed=7)
    q.requires_grad_(), k.requires_grad_(), v.requires_grad_()
    o = A.flash_attention(q, k, v, batch, True)
    do = torch.randn_like(o)
    o.backward(do)
    torch.cuda.synchronize()
    _lib.check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    o_ref, _ = A.attention_ref(qr, kr, vr, batch, True)
    o_ref.backward(do.float())
    assert (o.float() - o_ref.float()).abs().max().item() <= 2e-2
    for name, a, b in (("dq", q.grad, qr.grad), ("dk", k.grad, kr.grad), ("dv", v.grad, vr.grad)):
        err = (a.float() - b).abs().max().item()
        tol = 3e-2 * b.abs().max().item() + 2e-2
        assert err <= tol, f"{name}: err {err} tol {tol}"
        rel = (a.float() - b).norm().item() / b.norm().item()
        assert rel <= 1e-2, f"{name}: relative error {rel}"


def test_flash_attn_deterministic():
    q, k, v = _inputs(1, 1024, 8, 2, 128, 128, seed=3)
    o1, l1 = A.flash_attn_fwd(q, k, v, 1, True, 0.088)
    o2, l2 = A.flash_attn_fwd(q, k, v, 1, True, 0.088)
    assert torch.equal(o1, o2) and torch.equal(l1, l2)


CHUNK_CASES = [
    # batch, seq_q, q_off, hq, hkv, dqk, dv, causal
    (1, 128, 128, 2, 2, 128, 128, True),
    (1, 256, 384, 4, 2, 128, 128, True),
    (2, 128, 256, 4, 1, 128, 128, True),
    (1, 384, 0, 2, 2, 128, 128, True),
    (1, 256, 256, 2, 2, 192, 128, True),
    (1, 128, 0, 2, 2, 128, 128, False),     # cross attention: 128 queries over 384 keys
]


@pytest.mark.parametrize("case", CHUNK_CASES)
def test_flash_attn_chunk_against_longer_keys(case):
    """Queries of a sequence chunk at key position q_off attending to keys [0, q_off + seq_q) (forward and backward)."""
    batch, sq, q_off, hq, hkv, dqk, dv, causal = case
    sk = q_off + sq if causal else 384
    g = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn(batch * sq, hq, dqk, device="cuda", generator=g).bfloat16().requires_grad_()
    k = torch.randn(batch * sk, hkv, dqk, device="cuda", generator=g).bfloat16().requires_grad_()
    v = torch.randn(batch * sk, hkv, dv, device="cuda", generator=g).bfloat16().requires_grad_()
    o = A.flash_attention(q, k, v, batch, causal, None, q_off if causal else 0)
    do = torch.randn_like(o)
    o.backward(do)
    torch.cuda.synchronize()
    _lib.check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    o_ref, _ = A.attention_ref(qr, kr, vr, batch, causal, None, q_off if causal else 0)
    o_ref.backward(do.float())
    assert (o.float() - o_ref.float()).abs().max().item() <= 2e-2
    for name, a, b in (("dq", q.grad, qr.grad), ("dk", k.grad, kr.grad), ("dv", v.grad, vr.grad)):
        err = (a.float() - b).abs().max().item()
        tol = 3e-2 * b.abs().max().item() + 2e-2
        assert err <= tol, f"{name}: err {err} tol {tol}"


WINDOW_CASES = [
    # batch, seq, hq, hkv, d, window, sinks
    (1, 512, 4, 2, 128, 128, False),
    (1, 640, 2, 2, 128, 200, True),
    (2, 384, 4, 1, 64, 128, True),
    (1, 1024, 2, 1, 128, 300, False),
    (1, 256, 2, 2, 128, 1000, True),     # window longer than the sequence
    (1, 384, 4, 4, 128, 0, True),        # sinks only
]


@pytest.mark.parametrize("case", WINDOW_CASES)
def test_flash_attn_sliding_window_and_sinks(case):
    batch, seq, hq, hkv, d, window, with_sinks = case
    q, k, v = _inputs(batch, seq, hq, hkv, d, d, seed=5)
    q.requires_grad_(), k.requires_grad_(), v.requires_grad_()
    sinks = (torch.randn(hq, device="cuda") * 2).requires_grad_() if with_sinks else None
    o = A.flash_attention(q, k, v, batch, True, None, 0, window, sinks)
    do = torch.randn_like(o)
    o.backward(do)
    torch.cuda.synchronize()
    _lib.check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    sr = sinks.detach().clone().requires_grad_() if with_sinks else None
    o_ref, _ = A.attention_ref(qr, kr, vr, batch, True, None, 0, window, sr)
    o_ref.backward(do.float())
    assert (o.float() - o_ref.float()).abs().max().item() <= 2e-2
    for name, a, b in (("dq", q.grad, qr.grad), ("dk", k.grad, kr.grad), ("dv", v.grad, vr.grad)):
        err = (a.float() - b).abs().max().item()
        tol = 3e-2 * b.abs().max().item() + 2e-2
        assert err <= tol, f"{name}: err {err} tol {tol}"
    if with_sinks:
        err = (sinks.grad - sr.grad).abs().max().item()
        assert err <= 3e-2 * sr.grad.abs().max().item() + 2e-2, (sinks.grad, sr.grad)


def test_packed_document_attention_forward_backward():
    """rope_attention with document segments (packed sequences) vs the fp32 reference run per document."""
    from primus_b200.ops import layers as L

    hq, hkv, d = 4, 2, 128
    T = 1024
    segs = [(0, 256), (256, 384), (384, 896), (896, 1024)]
    g = torch.Generator(device="cuda").manual_seed(9)
    qkv = torch.randn(T, (hq + 2 * hkv) * d, device="cuda", generator=g).bfloat16().requires_grad_()
    out = L.rope_attention(qkv, None, None, None, 1, hq, hkv, d, segments=segs)
    do = torch.randn_like(out)
    out.backward(do)
    torch.cuda.synchronize()
    _lib.check_status()
    ref_in = qkv.detach().float().cpu().requires_grad_()
    ref = L.rope_attention(ref_in, None, None, None, 1, hq, hkv, d, segments=segs)
    ref.backward(do.float().cpu())
    assert (out.float().cpu() - ref).abs().max().item() <= 2e-2
    err = (qkv.grad.float().cpu() - ref_in.grad).abs().max().item()
    assert err <= 3e-2 * ref_in.grad.abs().max().item() + 2e-2, err


@pytest.mark.parametrize("case", [(1, 384, 4, 2, 128, 0, 30.0), (1, 512, 2, 2, 128, 200, 20.0), (2, 256, 4, 1, 64, 0, 50.0)])
def test_flash_attn_softcapped_scores(case):
    batch, seq, hq, hkv, d, window, cap = case
    q, k, v = _inputs(batch, seq, hq, hkv, d, d, seed=11)
    q, k = (q * 3).detach(), (k * 3).detach()                 # large scores, so that the cap bites
    q.requires_grad_(), k.requires_grad_(), v.requires_grad_()
    o = A.flash_attention(q, k, v, batch, True, None, 0, window, None, cap)
    do = torch.randn_like(o)
    o.backward(do)
    torch.cuda.synchronize()
    _lib.check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    o_ref, _ = A.attention_ref(qr, kr, vr, batch, True, None, 0, window, None, cap)
    o_ref.backward(do.float())
    assert (o.float() - o_ref.float()).abs().max().item() <= 3e-2
    for name, a, b in (("dq", q.grad, qr.grad), ("dk", k.grad, kr.grad), ("dv", v.grad, vr.grad)):
        err = (a.float() - b).abs().max().item()
        tol = 4e-2 * b.abs().max().item() + 3e-2
        assert err <= tol, f"{name}: err {err} tol {tol}"


def _clusters(batch, seq, hq, hkv, dqk, dv, causal, window, q_off=0):
    """CTAs per block of the dK / dV and of the dQ pass."""
    lib = _lib.require()
    seq_k = seq + q_off
    return [lib.pb_flash_attn_bwd_cluster(p, batch, seq, seq_k, q_off, hq, hkv, dqk, dv, int(causal), window) for p in (0, 1)]


def _grads_and_reference(q, k, v, batch, causal, q_off=0, window=0, softcap=0.0, sinks=None):
    """Outputs and gradients of the kernels (twice, equal) against the fp32 reference, in the 2-norm: P, dS and the results are
    bf16, 2^-9 each; 3e-3 measured.  A log-sum-exp is fp32: 1e-3, and the 2^-11 that tanh.approx has of a capped score."""
    scale = 1.0 / math.sqrt(q.shape[2])
    o, lse = A.flash_attn_fwd(q, k, v, batch, causal, scale, q_off, window, sinks, softcap)
    do = torch.randn_like(o)
    grads = A.flash_attn_bwd(do, q, k, v, o, lse, batch, causal, scale, q_off=q_off, window=window, softcap=softcap, sinks=sinks)
    o2, lse2 = A.flash_attn_fwd(q, k, v, batch, causal, scale, q_off, window, sinks, softcap)
    again = A.flash_attn_bwd(do, q, k, v, o, lse, batch, causal, scale, q_off=q_off, window=window, softcap=softcap, sinks=sinks)
    torch.cuda.synchronize()
    _lib.check_status()
    leaves = [t.detach().float().requires_grad_() for t in (q, k, v)]
    sinks_ref = None if sinks is None else sinks.clone().requires_grad_()
    o_ref, lse_ref = A.attention_ref(*leaves, batch, causal, None, q_off, window, sinks_ref, softcap)
    o_ref.backward(do.float())
    assert torch.equal(o, o2) and torch.equal(lse, lse2)
    assert (lse - lse_ref).abs().max().item() <= 1e-3 + softcap * 2.0 ** -11
    refs = [o_ref.detach()] + [t.grad for t in leaves] + ([] if sinks is None else [sinks_ref.grad])
    for name, a, b, r in zip(("o", "dq", "dk", "dv", "dsinks")[:len(refs)], (o, *grads), (o, *again), refs, strict=True):
        assert torch.equal(a, b), name
        rel = (a.float() - r).norm().item() / r.norm().item()
        assert rel <= 1e-2, f"{name}: relative error {rel}"


@pytest.mark.parametrize("window, softcap, sinks, causal, q_off", [
    (0, 0.0, False, True, 0), (0, 0.0, False, False, 0), (0, 0.0, True, True, 384), (200, 0.0, True, True, 0),
    (128, 0.0, False, True, 0), (0, 2.0, False, True, 0), (200, 2.0, True, True, 0), (0, 2.0, False, False, 0),
])
@pytest.mark.parametrize("batch, hq, hkv, dqk, dv", [(8, 32, 16, 64, 64), (8, 32, 16, 128, 128), (16, 16, 16, 192, 128)])
def test_flash_attn_of_more_blocks_than_sms(batch, hq, hkv, dqk, dv, window, softcap, sinks, causal, q_off):
    """Every CTA takes several blocks, one after the other: five row blocks of 128 per head (in the forward two pairs and one tile
    alone), blocks of one to eight steps."""
    seq = 640
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert batch * hq * 3 >= 4 * sms and batch * hkv * 5 >= 4 * sms
    assert _clusters(batch, seq, hq, hkv, dqk, dv, causal, window, q_off) == [1, 1]
    q, _, _ = _inputs(batch, seq, hq, hkv, dqk, dv, seed=21)
    _, k, v = _inputs(batch, seq + q_off, hq, hkv, dqk, dv, seed=22)
    logits = torch.linspace(-2, 2, hq, device="cuda") if sinks else None
    _grads_and_reference(q, k, v, batch, causal, q_off, window, softcap, logits)


@pytest.mark.parametrize("batch, seq, hq, hkv, dqk, dv, causal, window, q_off, softcap", [
    (1, 1024, 8, 1, 128, 128, True, 0, 3072, 0.0),          # a chunk of a longer sequence
    (1, 1024, 8, 1, 64, 64, True, 0, 3072, 2.0),
    (1, 512, 2, 2, 192, 128, True, 0, 3584, 0.0),
    (1, 2048, 8, 1, 128, 128, True, 0, 0, 2.0),
    (1, 4096, 2, 1, 64, 64, False, 0, 0, 2.0),
    (1, 2048, 1, 1, 192, 128, True, 0, 0, 2.0),
    (1, 2048, 4, 1, 128, 128, True, 1000, 0, 2.0),
])
def test_flash_attn_shared_blocks_of_chunks_and_capped_scores(batch, seq, hq, hkv, dqk, dv, causal, window, q_off, softcap):
    assert max(_clusters(batch, seq, hq, hkv, dqk, dv, causal, window, q_off)) > 1
    q, _, _ = _inputs(batch, seq, hq, hkv, dqk, dv, seed=23)
    _, k, v = _inputs(batch, seq + q_off, hq, hkv, dqk, dv, seed=24)
    _grads_and_reference(q, k, v, batch, causal, q_off, window, softcap)


@pytest.mark.parametrize("case, shared", [
    # batch, seq, hq, hkv, dqk, dv, causal, window; whether CTAs share the blocks of the dK / dV and of the dQ pass
    ((1, 128, 1, 1, 128, 128, True, 0), (False, False)),    # one step: nothing to share
    ((1, 640, 3, 1, 64, 64, True, 0), (True, False)),       # step counts that the ranks cannot share evenly
    ((1, 2048, 8, 1, 128, 128, True, 0), (True, False)),
    ((1, 4096, 2, 1, 128, 128, False, 0), (True, True)),
    ((2, 1152, 2, 2, 192, 128, True, 0), (True, True)),
    ((1, 2048, 1, 1, 192, 128, True, 0), (True, True)),
    ((1, 2048, 4, 1, 64, 64, True, 1000), (True, False)),
])
def test_flash_attn_backward_of_shared_blocks(case, shared):
    """Blocks whose steps several CTAs share: gradients against the fp32 reference, equal from call to call, and into strided
    views of a packed gradient."""
    batch, seq, hq, hkv, dqk, dv, causal, window = case
    assert tuple(c > 1 for c in _clusters(*case)) == shared
    q, k, v = _inputs(batch, seq, hq, hkv, dqk, dv, seed=5)
    scale = 1.0 / math.sqrt(dqk)
    o, lse = A.flash_attn_fwd(q, k, v, batch, causal, scale, window=window)
    do = torch.randn_like(o)
    grads = A.flash_attn_bwd(do, q, k, v, o, lse, batch, causal, scale, window=window)
    if dqk == dv:
        packed = torch.full((batch * seq, (hq + 2 * hkv) * dqk), 7.0, device="cuda", dtype=torch.bfloat16)
        views = [t.unflatten(1, (-1, dqk)) for t in packed.split([hq * dqk, hkv * dqk, hkv * dqk], 1)]
        again = A.flash_attn_bwd(do, q, k, v, o, lse, batch, causal, scale, *views, window=window)
    else:
        again = A.flash_attn_bwd(do, q, k, v, o, lse, batch, causal, scale, window=window)
    torch.cuda.synchronize()
    _lib.check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    o_ref, _ = A.attention_ref(qr, kr, vr, batch, causal, window=window)
    o_ref.backward(do.float())
    for name, a, b, r in zip(("dq", "dk", "dv"), grads, again, (qr, kr, vr)):
        assert torch.equal(a, b), name
        rel = (a.float() - r.grad).norm().item() / r.grad.norm().item()
        assert rel <= 1e-2, f"{name}: relative error {rel}"     # P, dS and the results in bf16: 2^-9 each, 3e-3 measured


def test_flash_attn_more_sequences_than_a_grid_dimension():
    """65537 sequences of 128 tokens: the first, those around the limit and the last, forward and backward."""
    batch, seq, d = 65537, 128, 64
    q, k, v = _inputs(batch, seq, 1, 1, d, d, seed=9)
    do = torch.randn_like(q)
    scale = 1.0 / math.sqrt(d)
    o, lse = A.flash_attn_fwd(q, k, v, batch, True, scale)
    grads = A.flash_attn_bwd(do, q, k, v, o, lse, batch, True, scale)
    torch.cuda.synchronize()
    _lib.check_status()
    for b in (0, 65534, 65535, 65536):
        r = slice(b * seq, (b + 1) * seq)
        one_o, one_lse = A.flash_attn_fwd(q[r], k[r], v[r], 1, True, scale)
        ones = A.flash_attn_bwd(do[r], q[r], k[r], v[r], one_o, one_lse, 1, True, scale)
        assert torch.equal(o[r], one_o) and torch.equal(lse[b], one_lse[0])
        for a, c in zip(grads, ones):
            assert torch.equal(a[r], c)
