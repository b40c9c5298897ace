"""Kernels at the edges of their tiles and dispatch rules: row widths around every lane-group size of the norms, GEMM
shapes around the 256 x 256 CTA-pair tile, permutation maps around the scan step, ragged vocabularies and masked logits.

Tolerances: a bf16 result rounds once (2^-8 relative at most, 2^-9 on average), so elementwise results are compared
within 2^-7 of their own size plus 2^-9 of the tensor's maximum; fp32 sums of n products of O(1) values within
n * 2^-24 * sqrt(n) of their size, generously 1e-4."""
import pytest
import torch

from primus_b200.ops import _lib, attention, fused, gemm, optim
from primus_b200.ops import moe as M

pytestmark = pytest.mark.gpu


def _gen(seed=0):
    return torch.Generator(device="cuda").manual_seed(seed)


def _close_bf16(got, ref, what):
    ref = ref.double()
    err = (got.double() - ref).abs()
    lim = ref.abs() * 2.0 ** -7 + ref.abs().max() * 2.0 ** -9
    assert (err <= lim).all(), f"{what}: error {err.max().item()} at value {ref.flatten()[err.argmax()].item()}"


def _rms64(x, w, eps=1e-5):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


@pytest.mark.parametrize("H", [8, 64, 72, 128, 136, 256, 264, 512, 520, 1024, 1032, 2048, 2056, 4096, 4104, 8192, 8200, 16384])
@pytest.mark.parametrize("rows,with_res", [(1, True), (13, False), (700, True)])
def test_rmsnorm_widths(H, rows, with_res):
    g = _gen(H + rows)
    x, r, dy, ds = (torch.randn(rows, H, device="cuda", generator=g).bfloat16() for _ in range(4))
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).bfloat16()
    xl, wl = x.clone().requires_grad_(), w.clone().requires_grad_()
    s64 = ((x + r) if with_res else x).double().requires_grad_()
    w64 = w.double().requires_grad_()
    y64 = _rms64(s64, w64)
    if with_res:
        rl = r.clone().requires_grad_()
        y, s = fused.rmsnorm(xl, wl, 1e-5, rl)
        torch.autograd.backward([y, s], [dy, ds])
        torch.autograd.backward([y64, s64 * 1.0], [dy.double(), ds.double()])
        assert torch.equal(s.detach(), x + r) and torch.equal(rl.grad, xl.grad)
    else:
        y = fused.rmsnorm(xl, wl)
        y.backward(dy)
        y64.backward(dy.double())
    _close_bf16(y.detach(), y64.detach(), "y")
    _close_bf16(xl.grad, s64.grad, "dx")
    _close_bf16(wl.grad, w64.grad, "dw")


@pytest.mark.parametrize("R,E,topk", [(1, 1, 1), (31, 5, 1), (4095, 8, 3), (4096, 300, 4), (4100, 7, 2), (12289, 64, 1)])
def test_permutation_maps_match_stable_sort(R, E, topk):
    e = torch.randint(0, E, (R,), generator=torch.Generator().manual_seed(R))
    e[e == E // 2] = 0                                     # an expert without copies (except when it is the only one)
    counts = torch.bincount(e, minlength=E).to(torch.int32)
    cap = M.rows_capacity(R, E)
    cpu = M.token_maps(e, M.build_schedule(counts, cap), topk)
    gpu = M.token_maps(e.cuda(), M.build_schedule(counts.cuda(), cap), topk)
    for c, g, name in zip(cpu, gpu, ("src", "pos", "src_token")):
        assert torch.equal(c, g.cpu()), name
    src, pos = M.permutation_maps(e.cuda(), M.build_schedule(counts.cuda(), cap))
    assert torch.equal(src.cpu(), cpu[0]) and torch.equal(pos.cpu(), cpu[1])
    p = torch.rand(R, device="cuda", requires_grad=True)
    out = M.permute_probs(p, src, pos)
    ref = torch.where(src >= 0, p.detach()[src.clamp_min(0).long()], torch.zeros((), device="cuda"))
    assert torch.equal(out.detach(), ref)
    d = torch.rand(cap, device="cuda")
    out.backward(d)
    assert torch.equal(p.grad, d[pos.long()])


@pytest.mark.parametrize("M_,N_,K_", [(256, 256, 64), (256, 264, 72), (264, 256, 200), (520, 1000, 64), (1000, 520, 328),
                                      (4096, 2048, 136), (8, 136, 2048), (136, 264, 4104), (768, 256, 3208), (256, 512, 2056)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_cta_pair_bf16_gemm(M_, N_, K_, a_mn, b_mn):
    g = _gen(M_ + N_ + K_)
    a = torch.randn(*((K_, M_) if a_mn else (M_, K_)), device="cuda", generator=g).bfloat16()
    b = torch.randn(*((K_, N_) if b_mn else (N_, K_)), device="cuda", generator=g).bfloat16()
    A, B = (a.t() if a_mn else a).double(), (b if b_mn else b.t()).double()
    ref = A @ B
    lim = 2.0 ** -24 * K_ * (A.abs() @ B.abs()).max()     # fp32 accumulation in any order
    for mode, out in (("bf16", None), ("f32", torch.empty(M_, N_, device="cuda")), ("add", torch.ones(M_, N_, device="cuda"))):
        got = gemm.gemm(a, b, a_mn, b_mn, out=out, accumulate=mode == "add").double()
        torch.cuda.synchronize()
        _lib.check_status()
        if mode == "bf16":
            _close_bf16(got, ref, mode)
        else:
            err = (got - ref - (1 if mode == "add" else 0)).abs().max()
            assert err <= lim + 2.0 ** -22 * ref.abs().max(), f"{mode}: {err}"
        again = gemm.gemm(a, b, a_mn, b_mn, out=torch.empty_like(got, dtype=torch.float32) if mode != "bf16" else None)
        if mode != "add":
            assert torch.equal(again.double(), got), "not reproducible"


@pytest.mark.parametrize("T,hq,hkv,d,pad", [(1, 1, 1, 64, 0), (130, 4, 2, 128, 0), (77, 6, 3, 72, 16), (33, 2, 1, 256, 0),
                                            (2000, 8, 1, 128, 8)])
def test_qk_norm_matches_separate_norms(T, hq, hkv, d, pad):
    g = _gen(d)
    W = (hq + 2 * hkv) * d
    buf = torch.randn(T, W + pad, device="cuda", generator=g).bfloat16()
    dy = torch.randn(T, W, device="cuda", generator=g).bfloat16()
    wq, wk = ((1 + 0.1 * torch.randn(d, device="cuda", generator=g)).bfloat16().requires_grad_() for _ in range(2))
    wk.main_grad = torch.ones(d, device="cuda")
    qkv = buf.requires_grad_()
    out = fused.qk_norm(qkv[:, :W], wq, wk, hq, hkv, d)
    out.backward(dy)
    x64 = buf.detach()[:, :W].double().requires_grad_()
    q64, k64 = wq.detach().double().requires_grad_(), wk.detach().double().requires_grad_()
    h = x64.view(T, hq + 2 * hkv, d)
    ref = torch.cat([_rms64(h[:, :hq], q64), _rms64(h[:, hq:hq + hkv], k64), h[:, hq + hkv:]], 1).reshape(T, W)
    ref.backward(dy.double())
    _close_bf16(out.detach(), ref.detach(), "out")
    assert torch.equal(out.detach()[:, (hq + hkv) * d:], buf.detach()[:, (hq + hkv) * d:W])
    _close_bf16(qkv.grad[:, :W], x64.grad, "dqkv")
    _close_bf16(wq.grad, q64.grad, "dwq")
    assert wk.grad is None
    err = (wk.main_grad.double() - 1 - k64.grad).abs().max()
    assert err <= 1e-4 * (1 + k64.grad.abs().max()), f"dwk {err}"


@pytest.mark.parametrize("heads,d,rot,T", [(1, 64, 64, 5), (3, 128, 128, 130), (6, 64, 32, 77), (9, 192, 64, 64)])
def test_rope_head_groups(heads, d, rot, T):
    g = _gen(heads)
    x = torch.randn(T, heads * d + 8, device="cuda", generator=g).bfloat16()
    before = x.clone()
    cos, sin = fused.rope_tables(T + 3, rot, 1e4, "cuda")
    pos = torch.randint(0, T + 3, (T,), device="cuda", generator=g, dtype=torch.int32)
    view = x[:, :heads * d].view(T, heads, d)
    fused.rope_inplace_(view, cos, sin, pos, rot)
    _close_bf16(view, fused.rope_ref(before[:, :heads * d].view(T, heads, d).double(), cos, sin, pos, rot), "rope")
    assert torch.equal(x[:, heads * d:], before[:, heads * d:])
    fused.rope_inplace_(view, cos, sin, pos, rot, backward=True)
    _close_bf16(view, before[:, :heads * d].view(T, heads, d), "inverse")


@pytest.mark.parametrize("batch,S,hq,hkv", [(1, 128, 3, 1), (2, 256, 16, 2)])
def test_sink_gradient_matches_oracle(batch, S, hq, hkv):
    g = _gen(hq)
    q, do = (torch.randn(batch * S, hq, 64, device="cuda", generator=g).bfloat16() for _ in range(2))
    k, v = (torch.randn(batch * S, hkv, 64, device="cuda", generator=g).bfloat16() for _ in range(2))
    sinks = torch.randn(hq, device="cuda", generator=g)
    o, lse = attention.flash_attn_fwd(q, k, v, batch, True, 0.125, sinks=sinks)
    ds = attention.flash_attn_bwd(do, q, k, v, o, lse, batch, True, 0.125, sinks=sinks)[3]
    ref = attention.sink_grad(do, o, lse, sinks, batch)
    assert (ds - ref).abs().max() <= 1e-4 * (1 + ref.abs().max())


@pytest.mark.parametrize("n,off", [(1, 0), (3, 1), (4099, 3), (2 ** 20 + 5, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sumsq_ragged_and_misaligned(n, off, dtype):
    x = torch.randn(n + off, device="cuda", generator=_gen(n)).to(dtype)[off:]
    out = torch.zeros(1, device="cuda")
    optim.sumsq_(x, out)
    ref = x.double().pow(2).sum().item()
    assert abs(out.item() - ref) <= 1e-5 * ref


@pytest.mark.parametrize("cuts", [[0], [0, 4, 8, 8192, 8196, 20000], [0, 8188, 16384]])
@pytest.mark.parametrize("state", [torch.float32, torch.bfloat16])
def test_adamw_ranges_match_one_launch_per_range(cuts, state):
    n, g = 24604, _gen(len(cuts))
    ranges = [(100 + a, 100 + b, float(i % 2), i % 4) for i, (a, b) in enumerate(zip(cuts, cuts[1:] + [n]))]
    lrs = [1e-2, 2e-3, 5e-3, 1e-3]
    hyper = dict(beta1=0.9, beta2=0.95, eps=1e-8, step=3, grad_scale=torch.full((1,), 0.7, device="cuda"))

    def fresh():
        g.manual_seed(1)
        t = [torch.randn(n, device="cuda", generator=g) for _ in range(3)]
        v = torch.rand(n, device="cuda", generator=g)
        return t[0], t[1].to(state), v.to(state), t[2], torch.zeros(n, device="cuda", dtype=torch.bfloat16)

    p, m, v, grad, out = fresh()
    p64, m64, v64, g64 = p.double(), m.double(), v.double(), grad.double() * 0.7
    optim.adamw_ranges_(p, m, v, grad, out, optim.range_table(ranges, 100, n, "cuda"), lrs=lrs, weight_decay=0.1, **hyper)
    p2, m2, v2, grad, out2 = fresh()
    upd = torch.zeros_like(p64)
    for lo, hi, mult, grp in ranges:
        sl = slice(lo - 100, hi - 100)
        optim.adamw_step_(p2[sl], m2[sl], v2[sl], grad[sl], out2[sl], lr=lrs[grp], weight_decay=0.1 * mult, **hyper)
        mm, vv = 0.9 * m64[sl] + 0.1 * g64[sl], 0.95 * v64[sl] + 0.05 * g64[sl] ** 2
        upd[sl] = lrs[grp] * (mm / (1 - 0.9 ** 3)) / ((vv / (1 - 0.95 ** 3)).sqrt() + 1e-8)
        p64[sl] = p64[sl] * (1 - lrs[grp] * 0.1 * mult) - upd[sl]
    for a, b in ((p, p2), (m, m2), (v, v2), (out, out2)):
        assert torch.equal(a, b)
    # fp32 rounding of p and of the update: a few ulp of either; m is a sum that may cancel (0.1 |m| + 0.1 |g| in fp32)
    scale = upd.abs() + max(lrs) * (m64.abs() + g64.abs()) / v64.sqrt().clamp_min(1e-3)
    assert ((p.double() - p64).abs() <= 2.0 ** -22 * (p64.abs() + scale)).all()


@pytest.mark.parametrize("V", [8, 4088, 16384, 16392, 53248, 53256, 106504, 128256])
def test_cross_entropy_masked_and_ragged(V):
    """Rows with -inf and lowest-value masks (a row of nothing but the lowest value has no fp32 log-sum-exp)."""
    g = _gen(V)
    T = 9
    x = (torch.randn(T, V, device="cuda", generator=g) * 4).bfloat16()
    low = torch.finfo(torch.bfloat16).min
    x[1, 1:] = float("-inf")
    x[2, : V - 1] = low
    x[4, V // 2:] = low
    lab = torch.randint(0, V, (T,), device="cuda", generator=g)
    lab[1], lab[2], lab[4] = 0, V - 1, 0
    ref = x.double().requires_grad_()
    loss64 = torch.nn.functional.cross_entropy(ref, lab, reduction="none")
    loss64.sum().backward()
    xl = x.clone().requires_grad_()
    loss = fused.cross_entropy(xl * 1.0, lab)
    loss.sum().backward()
    assert (loss.double() - loss64).abs().max() <= 1e-5 * (1 + loss64.abs().max())
    _close_bf16(xl.grad, ref.grad, "dlogits")


@pytest.mark.parametrize("V", [8, 4096, 57344, 57352, 131072])
@pytest.mark.parametrize("pad", [0, 24])
def test_cross_entropy_rows_with_pitch_spread_and_start_masks(V, pad):
    """The edges between the variants; rows with a pitch, a mask in front, probabilities that are no normal numbers, labels out of
    range (no target: loss 0, gradient the softmax)."""
    g = _gen(V + pad)
    T = 6
    x = (torch.randn(T, V + pad, device="cuda", generator=g) * 4).bfloat16()
    x[1, : V - 3] = float("-inf")
    x[2, ::3] -= 95.0
    x[3, 1:V] -= 300.0
    lab = torch.randint(0, V, (T,), device="cuda", generator=g)
    lab[0], lab[1], lab[4], lab[5] = 0, V - 1, -100, V
    scale = torch.rand(T, device="cuda", generator=g) + 0.5
    want = x.clone()
    lse = torch.logsumexp(x[:, :V].double(), 1)
    p = (x[:, :V].double() - lse[:, None]).exp()
    rows = torch.arange(4, device="cuda")
    loss64 = torch.zeros(T, device="cuda", dtype=torch.float64)
    loss64[:4] = lse[:4] - x[rows, lab[:4]].double()
    p[rows, lab[:4]] -= 1
    want[:, :V] = (p * scale.double()[:, None]).bfloat16()
    loss = torch.empty(T, device="cuda")
    _lib.call("ce_fused", x, lab, scale, loss, T, V, x.stride(0))
    assert torch.equal(x[:, V:], want[:, V:])
    # fp32 sums of 8 to 131072 terms in pairs of chains and trees: a few 2^-24 of the sum, and of the log-sum-exp itself
    assert (loss.double() - loss64).abs().max() <= 1e-5 * (1 + lse.abs().max())
    # exponents of up to 2^-16 absolute at |f - lse| of 300, one rounding to bf16; below 2^-126 an exponential has 2^-149 at best
    err = (x[:, :V].double() - want[:, :V].double()).abs()
    assert (err <= 2.0 ** -7 * want[:, :V].double().abs() + 2.0 ** -22 * (lab < V)[:, None] + 2.0 ** -133).all()
