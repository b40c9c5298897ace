"""Performance cases: the work a training run of this framework has the GPU do, through its public entry points.

Every case is one forward and backward pass of a layer, a block or a small model (or one quantisation, or one optimizer
step), in the layout the model code uses.  Parameters that a training run keeps in a gradient buffer own a fp32
``main_grad`` here too, into which a pass accumulates as one micro-batch of a step does.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from primus_b200.models.config import TransformerConfig
from primus_b200.models.gpt import SelfAttention, build_model
from primus_b200.models.moe import MoELayer
from primus_b200.ops import attention, fp8, fused, gemm, layers
from primus_b200.parallel.distributed import DistributedOptimizer, ParamGradBuffer

DEV = "cuda"
BF16 = torch.bfloat16
EPS = 1e-5


# ----------------------------------------------------------------------------------------------
# the cases
def listed():
    return [
        # the smallest call of a step: a residual norm over a short packed batch, where launches and latency count
        dict(name="norm_small", kind="norm", rows=200, H=2048, residual=True),
        # the residual norm of a Llama-3.1-70B layer, two sequences of 8192 tokens
        dict(name="norm_large", kind="norm", rows=16384, H=8192, residual=True),
        # activation / gradient quantisation for the MXFP8 GEMMs of a Llama-3.1-8B layer, both directions
        dict(name="quantize", kind="quantize", R=8192, C=4096, scaling="mxfp8", weight=False),
        # core attention of Llama-3.1-8B at its training length (8 key / value heads, packed QKV views)
        dict(name="attn_gqa", kind="attn", batch=1, seq=8192, hq=32, hkv=8, dqk=128, dv=128, window=0, sinks=False),
        # core attention of DeepSeek-V2-Lite (multi-latent head shape)
        dict(name="attn_mla", kind="attn", batch=1, seq=4096, hq=16, hkv=16, dqk=192, dv=128, window=0, sinks=False),
        # a sliding-window layer of GPT-OSS (64-wide heads, learned sinks)
        dict(name="attn_window", kind="attn", batch=2, seq=2048, hq=64, hkv=8, dqk=64, dv=64, window=128, sinks=True),
        # attention block of Qwen3-30B-A3B: norm, QKV, per-head norms, rotary embedding, attention, projection
        dict(name="attn_block", kind="block", batch=1, seq=4096, H=2048, hq=32, hkv=4, d=128, qknorm=True, recipe=""),
        # dense MLP block of Llama-3.1-8B under the flagship MXFP8 recipe
        dict(name="mlp_mxfp8", kind="mlp", T=8192, H=4096, I=14336, recipe="mxfp8"),
        # final norm, LM head and loss of Llama-3.2-1B
        dict(name="head_loss", kind="head", T=4096, H=2048, V=128256),
        # mixture-of-experts layer: router, permutation, grouped GEMMs, combine
        dict(name="moe_layer", kind="moe", T=4096, E=64, topk=8, H=2048, I=768),
        # one AdamW step with gradient clipping over flat buffers (about half a Llama-3.1-8B layer)
        dict(name="optimizer", kind="optimizer", width=4096, blocks=6, odd=1029, bf16_state=False),
        # a whole step of the tiny Llama model: many small launches, an FFN width that is no multiple of a tile
        dict(name="tiny_step", kind="model", batch=2, seq=384, layers=2, H=256, I=688, hq=4, hkv=2, d=64, V=32000),
    ]


def _log(rng, lo, hi, step=1):
    return max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step)


def draw(rng):
    kind = rng.choice(["norm", "quantize", "attn", "block", "mlp", "head", "moe", "optimizer", "model"])
    if kind == "norm":
        if rng.random() < 0.3:      # per-head norms: many short rows
            return dict(kind=kind, rows=_log(rng, 500, 262144), H=rng.choice([64, 128, 192]), residual=False)
        H = _log(rng, 256, 8192, 8)
        return dict(kind=kind, rows=_log(rng, 1, min(16384, 2 ** 26 // H)), H=H, residual=rng.random() < 0.6)
    if kind == "quantize":
        C = _log(rng, 128, 14336, 128)
        return dict(kind=kind, R=_log(rng, 128, min(16384, 2 ** 27 // C), 128), C=C,
                    scaling=rng.choice(["mxfp8", "mxfp8", "blockwise", "tensorwise"]), weight=rng.random() < 0.3)
    if kind == "attn":
        dqk, dv = rng.choice(attention.KERNEL_HEAD_DIMS)
        hkv = rng.choice([1, 2, 4, 8])
        hq = hkv * (1 if dqk != dv else rng.choice([1, 2, 4, 8]))
        seq = _log(rng, 128, 8192, 128)
        window = rng.choice([0, 0, 128, 1000]) if dqk == dv else 0
        return dict(kind=kind, batch=rng.choice([1, 1, 2, 3]) if seq <= 4096 else 1, seq=seq, hq=min(hq, 32), hkv=hkv,
                    dqk=dqk, dv=dv, window=window, sinks=dqk == dv and rng.random() < 0.3)
    if kind == "block":
        recipe = rng.choice(["", "mxfp8"])
        d, hkv = rng.choice([64, 128]), rng.choice([2, 4, 8])
        return dict(kind=kind, batch=rng.choice([1, 2]), seq=_log(rng, 128, 3072, 128), H=_log(rng, 256, 4096, 128),
                    hq=hkv * rng.choice([2, 4]), hkv=hkv, d=d, qknorm=rng.random() < 0.5, recipe=recipe)
    if kind == "mlp":
        recipe = rng.choice(["", "mxfp8"])
        step = 128 if recipe else 8
        return dict(kind=kind, T=_log(rng, 128, 8192, 128 if recipe else 1), H=_log(rng, 256, 4096, step),
                    I=_log(rng, 256, 7168, step), recipe=recipe)
    if kind == "head":
        return dict(kind=kind, T=_log(rng, 64, 4096), H=_log(rng, 256, 2048, 64), V=_log(rng, 8192, 128256, 128))
    if kind == "moe":
        return dict(kind=kind, T=_log(rng, 64, 4096), E=rng.choice([8, 16, 32, 64]), topk=rng.choice([2, 4, 6, 8]),
                    H=_log(rng, 256, 2048, 128), I=_log(rng, 128, 768, 64))
    if kind == "optimizer":
        return dict(kind=kind, width=_log(rng, 64, 4096, 8), blocks=rng.randint(1, 6), odd=rng.randint(1, 5000),
                    bf16_state=rng.random() < 0.4)
    hkv = rng.choice([1, 2])
    return dict(kind=kind, batch=rng.choice([1, 2]), seq=_log(rng, 128, 1024, 128), layers=rng.choice([1, 2, 3]),
                H=rng.choice([256, 384, 512]), I=_log(rng, 256, 1400, 8), hq=hkv * rng.choice([2, 4]), hkv=hkv, d=64,
                V=_log(rng, 4096, 32000, 128))


# ----------------------------------------------------------------------------------------------
# inputs
class _State:
    def __init__(self, **kw):
        self.__dict__.update(kw)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, std=1.0):
    return (torch.randn(*shape, generator=g, device=DEV) * std).to(BF16)


def _gain(g, n):
    return (1.0 + 0.1 * torch.randn(n, generator=g, device=DEV)).to(BF16)


def _own_main_grads(params):
    return ParamGradBuffer(list(params), None, 1, 0)


def _attn_inputs(case, g):
    """Query, key and value views into one packed projection output (own tensors for the multi-latent shape)."""
    T, hq, hkv, dqk, dv = case["batch"] * case["seq"], case["hq"], case["hkv"], case["dqk"], case["dv"]
    if dqk != dv:
        return _randn(g, T, hq, dqk), _randn(g, T, hkv, dqk), _randn(g, T, hkv, dv)
    qkv = _randn(g, T, (hq + 2 * hkv) * dqk)
    return (qkv[:, :hq * dqk].view(T, hq, dqk), qkv[:, hq * dqk:(hq + hkv) * dqk].view(T, hkv, dqk),
            qkv[:, (hq + hkv) * dqk:].view(T, hkv, dqk))


def _block_config(case):
    return TransformerConfig(num_layers=4, hidden_size=case["H"], num_attention_heads=case["hq"],
                             num_query_groups=case["hkv"], kv_channels=case["d"], qk_layernorm=case["qknorm"],
                             rotary_base=1e6)


def _moe_config(case):
    return TransformerConfig(num_layers=4, hidden_size=case["H"], num_experts=case["E"], moe_router_topk=case["topk"],
                             moe_ffn_hidden_size=case["I"], moe_aux_loss_coeff=1e-3)


def _model_config(case):
    return TransformerConfig(num_layers=case["layers"], hidden_size=case["H"], ffn_hidden_size=case["I"],
                             num_attention_heads=case["hq"], num_query_groups=case["hkv"], kv_channels=case["d"],
                             vocab_size=case["V"], seq_length=case["seq"])


def _norm_inputs(case, g):
    R, H = case["rows"], case["H"]
    return (_randn(g, R, H), _randn(g, R, H) if case["residual"] else None, _gain(g, H), _randn(g, R, H, std=0.1),
            _randn(g, R, H, std=0.1))


def _mlp_inputs(case, g):
    T, H, I = case["T"], case["H"], case["I"]
    return dict(hidden=_randn(g, T, H), residual=_randn(g, T, H), norm=_gain(g, H), w1=_randn(g, 2 * I, H, std=0.02),
                w2=_randn(g, H, I, std=0.02), dout=_randn(g, T, H, std=0.1), dres=_randn(g, T, H, std=0.1))


def _head_inputs(case, g):
    T, H, V = case["T"], case["H"], case["V"]
    return dict(hidden=_randn(g, T, H), residual=_randn(g, T, H), norm=_gain(g, H), w=_randn(g, V, H, std=0.02),
                labels=torch.randint(0, V, (T,), generator=g, device=DEV),
                weights=torch.full((T,), 1.0 / T, device=DEV))


def _optimizer_inputs(case, g):
    """Parameters of the shapes a layer has (matrices, norm gains, one odd bias) and their gradients."""
    w = case["width"]
    shapes = [(case["odd"],)]
    for _ in range(case["blocks"]):
        shapes += [(w, w), (w,), (w // 4, w), (w,)]
    return [_randn(g, *s, std=0.02) for s in shapes], [torch.randn(*s, generator=g, device=DEV) * 1e-3 for s in shapes]


def _block_module(case, seed):
    torch.manual_seed(seed)
    m = SelfAttention(_block_config(case), 0, DEV, 1)
    g = _gen(seed + 1)
    with torch.no_grad():
        for p in m.parameters():
            if p.dim() == 1:
                p.copy_(_gain(g, p.numel()))
    T = case["batch"] * case["seq"]
    x = [_randn(g, T, case["H"]) for _ in range(2)]
    d = [_randn(g, T, case["H"], std=0.1) for _ in range(2)]
    return m, x, d


def _moe_module(case, seed):
    torch.manual_seed(seed)
    m = MoELayer(_moe_config(case), 0, DEV, 1)
    g = _gen(seed + 1)
    with torch.no_grad():
        m.router.weight.copy_(_randn(g, *m.router.weight.shape, std=0.05))
        for holder in (m.experts.fc1_weight, m.experts.fc2_weight):
            holder.weight.copy_(_randn(g, *holder.weight.shape, std=0.02))
    return m, _randn(g, case["T"], case["H"]), _randn(g, case["T"], case["H"], std=0.1)


def _model_inputs(case, seed):
    model = build_model(_model_config(case), DEV, seed=seed)
    g = _gen(seed + 1)
    shape = (case["batch"], case["seq"])
    tokens = torch.randint(0, case["V"], shape, generator=g, device=DEV)
    labels = torch.randint(0, case["V"], shape, generator=g, device=DEV)
    return model, tokens, labels, torch.full(shape, 1.0 / tokens.numel(), device=DEV)


def prepare(case, seed):
    gemm.set_fp8_recipe(case.get("recipe") or None)     # what a run's configuration selects, once
    kind = case["kind"]
    g = _gen(seed)
    if kind == "norm":
        x, r, w, dy, ds = _norm_inputs(case, g)
        return _State(kind=kind, x=x.requires_grad_(), r=None if r is None else r.requires_grad_(),
                      w=torch.nn.Parameter(w), dy=dy, ds=ds)
    if kind == "quantize":
        # activations with a few large channels
        x = torch.randn(case["R"], case["C"], generator=g, device=DEV)
        x *= torch.exp(torch.randn(1, case["C"], generator=g, device=DEV))
        return _State(kind=kind, x=x.to(BF16), scaling=case["scaling"], weight=case["weight"])
    if kind == "attn":
        q, k, v = _attn_inputs(case, g)
        sinks = torch.randn(case["hq"], generator=g, device=DEV).requires_grad_() if case["sinks"] else None
        return _State(kind=kind, q=q.requires_grad_(), k=k.requires_grad_(), v=v.requires_grad_(), sinks=sinks,
                      do=_randn(g, q.shape[0], case["hq"], case["dv"], std=0.1), batch=case["batch"],
                      window=case["window"])
    if kind == "block":
        m, x, d = _block_module(case, seed)
        rope = (*fused.rope_tables(case["seq"], case["d"], 1e6, DEV),
                None if case["batch"] == 1 else torch.arange(case["seq"], device=DEV, dtype=torch.int32).repeat(case["batch"]))
        return _State(kind=kind, m=m, x=[t.requires_grad_() for t in x], d=d, rope=rope, batch=case["batch"],
                      buffer=_own_main_grads(m.parameters()))
    if kind == "mlp":
        t = _mlp_inputs(case, g)
        p = [torch.nn.Parameter(t[n]) for n in ("norm", "w1", "w2")]
        return _State(kind=kind, hidden=t["hidden"].requires_grad_(), residual=t["residual"].requires_grad_(), p=p,
                      dout=t["dout"], dres=t["dres"], buffer=_own_main_grads(p))
    if kind == "head":
        t = _head_inputs(case, g)
        p = [torch.nn.Parameter(t[n]) for n in ("norm", "w")]
        p[1]._fp8_exempt = True
        return _State(kind=kind, hidden=t["hidden"].requires_grad_(), residual=t["residual"].requires_grad_(), p=p,
                      labels=t["labels"], weights=t["weights"], buffer=_own_main_grads(p))
    if kind == "moe":
        m, x, d = _moe_module(case, seed)
        return _State(kind=kind, m=m, x=x.requires_grad_(), d=d, buffer=_own_main_grads(m.parameters()))
    if kind == "optimizer":
        ps, gs = _optimizer_inputs(case, g)
        ps = [torch.nn.Parameter(p) for p in ps]
        buf = _own_main_grads(ps)
        for p, d in zip(ps, gs):
            p.main_grad.copy_(d)
        opt = DistributedOptimizer([buf], lr=1e-3, state_dtype=BF16 if case["bf16_state"] else torch.float32)
        return _State(kind=kind, opt=opt, buffer=buf, p=ps)
    model, tokens, labels, weights = _model_inputs(case, seed)
    buf = _own_main_grads(model.parameters())
    return _State(kind=kind, model=model, tokens=tokens, labels=labels, weights=weights, buffer=buf,
                  opt=DistributedOptimizer([buf], lr=1e-4))


# ----------------------------------------------------------------------------------------------
# one pass
def run(s):
    if s.kind == "norm":
        s.x.grad = s.w.grad = None
        if s.r is None:
            y = fused.rmsnorm(s.x, s.w, EPS)
            y.backward(s.dy)
            return {"y": y.detach(), "dx": s.x.grad, "dw": s.w.grad}
        s.r.grad = None
        y, xsum = fused.rmsnorm(s.x, s.w, EPS, s.r)
        torch.autograd.backward([y, xsum], [s.dy, s.ds])
        return {"y": y.detach(), "xsum": xsum.detach(), "dx": s.x.grad, "dr": s.r.grad, "dw": s.w.grad}
    if s.kind == "quantize":
        q = fp8.quantize_mxfp8(s.x, scaling=s.scaling, is_weight=s.weight)
        return [q.q_row, q.sf_row, q.q_col, q.sf_col]
    if s.kind == "attn":
        s.q.grad = s.k.grad = s.v.grad = None
        if s.sinks is not None:
            s.sinks.grad = None
        o = attention.flash_attention(s.q, s.k, s.v, s.batch, True, window=s.window, sinks=s.sinks)
        o.backward(s.do)
        out = {"o": o.detach(), "dq": s.q.grad, "dk": s.k.grad, "dv": s.v.grad}
        if s.sinks is not None:
            out["dsinks"] = s.sinks.grad
        return out
    if s.kind == "block":
        for x in s.x:
            x.grad = None
        out, xsum = s.m(s.x[0], s.x[1], s.rope, s.batch)
        torch.autograd.backward([out, xsum], s.d)
        return {"out": out.detach(), "xsum": xsum.detach(), "dx": s.x[0].grad,
                "dw": [p.main_grad for p in s.m.parameters()]}
    if s.kind == "mlp":
        s.hidden.grad = s.residual.grad = None
        h1, xsum = layers.norm_linear(s.hidden, s.residual, s.p[0], s.p[1], EPS)
        out = layers.swiglu_linear(h1, s.p[2])
        torch.autograd.backward([out, xsum], [s.dout, s.dres])
        return {"out": out.detach(), "dx": s.hidden.grad, "dw": [p.main_grad for p in s.p]}
    if s.kind == "head":
        s.hidden.grad = s.residual.grad = None
        logits, _ = layers.norm_linear(s.hidden, s.residual, s.p[0], s.p[1], EPS)
        loss = fused.cross_entropy(logits, s.labels, weights=s.weights, unit_upstream=True)
        loss.backward()
        return {"loss": loss.detach(), "dx": s.hidden.grad, "dw": [p.main_grad for p in s.p]}
    if s.kind == "moe":
        s.x.grad = None
        out = s.m(s.x)
        out.backward(s.d)
        return {"out": out.detach(), "dx": s.x.grad, "dw": [p.main_grad for p in s.m.parameters()]}
    if s.kind == "optimizer":
        norm = s.opt.step()
        return {"norm": norm, "params": s.buffer.param_data, "master": [t["master"] for t in s.opt.state],
                "m": [t["m"] for t in s.opt.state], "v": [t["v"] for t in s.opt.state]}
    s.buffer.zero_grad()
    loss = s.model(s.tokens, s.labels, s.weights, unit_upstream=True)
    loss.backward()
    norm = s.opt.step()
    return {"loss": loss.detach(), "norm": norm, "params": s.buffer.param_data,
            "grads": [p.main_grad for p in s.buffer.params]}


# ----------------------------------------------------------------------------------------------
# what a pass cannot do without
def _attn_flops(batch, seq, hq, dqk, dv, window):
    pairs = seq * (seq + 1) / 2 if not window or window >= seq else window * seq - window * (window - 1) / 2
    # two products forward; five backward (the scores again, and four gradients)
    return batch * hq * pairs * (2 * (dqk + dv) + 2 * (3 * dqk + 2 * dv))


def work(case):
    kind = case["kind"]
    if kind == "norm":
        n = case["rows"] * case["H"]
        # forward reads x (+ r), writes y (+ sum); backward reads dy, x (+ the sum's gradient), writes dx
        return {"bytes": 2 * n * (8 if case["residual"] else 5), "flops": 12 * n}
    if kind == "quantize":
        n = case["R"] * case["C"]
        return {"bytes": 2 * n + 2 * n + 2 * n / 32, "flops": 4 * n}
    if kind == "attn":
        T, hq, hkv, dqk, dv = case["batch"] * case["seq"], case["hq"], case["hkv"], case["dqk"], case["dv"]
        qkv, o = T * (hq * dqk + hkv * (dqk + dv)), T * hq * dv
        return {"bytes": 2 * (2 * qkv + o) + 2 * (qkv + o), "flops": _attn_flops(case["batch"], case["seq"], hq, dqk, dv, case["window"])}
    if kind == "block":
        T, H, d, hq, hkv = case["batch"] * case["seq"], case["H"], case["d"], case["hq"], case["hkv"]
        n = H * (hq + 2 * hkv) * d + H * hq * d
        return {"bytes": 2 * n + 8 * n + 2 * 7 * T * H,
                "flops": 6 * T * n + _attn_flops(case["batch"], case["seq"], hq, d, d, 0)}
    if kind == "mlp":
        T, H, n = case["T"], case["H"], 3 * case["H"] * case["I"]
        return {"bytes": 2 * n + 8 * n + 2 * 7 * T * H, "flops": 6 * T * n}
    if kind == "head":
        T, H, n = case["T"], case["H"], case["H"] * case["V"]
        return {"bytes": 2 * n + 8 * n + 2 * 4 * T * H, "flops": 6 * T * n}
    if kind == "moe":
        T, H, n = case["T"], case["H"], 3 * case["H"] * case["I"]
        active = min(case["E"], T * case["topk"]) * n
        return {"bytes": 10 * active + 2 * 4 * T * H, "flops": 6 * T * (case["topk"] * n + H * case["E"])}
    if kind == "optimizer":
        w = case["width"]
        n = case["odd"] + case["blocks"] * (w * w + w * w // 4 + 2 * w)
        return {"bytes": n * (4 + 8 + (8 if case["bf16_state"] else 16) + 2), "flops": 20 * n}
    T, H, d, hq, hkv = case["batch"] * case["seq"], case["H"], case["d"], case["hq"], case["hkv"]
    layer = H * (2 * hq + 2 * hkv) * d + 3 * H * case["I"]
    mats = case["layers"] * layer + H * case["V"]
    params = mats + H * case["V"]
    # weights, their gradients and the optimizer state, read and written once
    return {"bytes": params * (4 + 8 + 16 + 2),
            "flops": 6 * T * mats + case["layers"] * _attn_flops(case["batch"], case["seq"], hq, d, d, 0)}


# Relative errors (2-norm) that another correct implementation shows: about four times what these paths measure against
# the 64-bit formulas, or, under MXFP8, between two orders of the 32-bit sums that precede a quantisation.
_TOLERANCE = {
    "norm": {"rel": 8e-3},
    "quantize": "exact",            # bytes
    "attn": {"rel": 1e-2},
    "block": {"rel": 1.5e-2},
    "mlp": {"rel": 1.5e-2},
    "head": {"rel": 1e-2},
    "moe": {"rel": 1.5e-2},
    "optimizer": {"rel": 1e-5},
    "model": {"rel": 2e-2},
}


def tolerance(case):
    if case["kind"] == "optimizer" and case["bf16_state"]:
        return {"rel": 4e-3}        # moments rounded to 16 bits: a sum's last bit can move one rounding
    return _TOLERANCE[case["kind"]]


# ----------------------------------------------------------------------------------------------
# the same results in 64 bits
def _d(t):
    return t.detach().double()


def _rms(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w


class _Attention64(torch.autograd.Function):
    """Causal softmax attention, one head at a time, with its derivative written out."""

    @staticmethod
    def _probs(q, k, scale, keep, sink):
        s = (q @ k.t() * scale).masked_fill(~keep, float("-inf"))
        m = s.amax(-1, keepdim=True)
        if sink is not None:
            m = torch.maximum(m, sink)
        e = torch.exp(s - m)
        z = e.sum(-1, keepdim=True)
        if sink is not None:
            z = z + torch.exp(sink - m)
            return e / z, torch.exp(sink - m) / z
        return e / z, None

    @staticmethod
    def _keep(S, window):
        i = torch.arange(S, device=DEV)
        diff = i[:, None] - i[None, :]
        return (diff >= 0) & (diff < window) if window else diff >= 0

    @staticmethod
    def forward(ctx, q, k, v, sinks, batch, window):
        T, hq, d = q.shape
        S, g = T // batch, hq // k.shape[1]
        keep = _Attention64._keep(S, window)
        o = torch.empty(T, hq, v.shape[2], dtype=q.dtype, device=q.device)
        for b in range(batch):
            r = slice(b * S, (b + 1) * S)
            for h in range(hq):
                p, _ = _Attention64._probs(q[r, h], k[r, h // g], d ** -0.5, keep, None if sinks is None else sinks[h])
                o[r, h] = p @ v[r, h // g]
        ctx.save_for_backward(q, k, v, sinks)
        ctx.meta = (batch, window)
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, sinks = ctx.saved_tensors
        batch, window = ctx.meta
        T, hq, d = q.shape
        S, g = T // batch, hq // k.shape[1]
        keep = _Attention64._keep(S, window)
        dq, dk, dv = torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
        ds = None if sinks is None else torch.zeros_like(sinks)
        for b in range(batch):
            r = slice(b * S, (b + 1) * S)
            for h in range(hq):
                p, ps = _Attention64._probs(q[r, h], k[r, h // g], d ** -0.5, keep, None if sinks is None else sinks[h])
                dp = do[r, h] @ v[r, h // g].t()
                delta = (p * dp).sum(-1, keepdim=True)
                dv[r, h // g] += p.t() @ do[r, h]
                dsc = p * (dp - delta) * d ** -0.5
                dq[r, h] = dsc @ k[r, h // g]
                dk[r, h // g] += dsc.t() @ q[r, h]
                if ds is not None:
                    ds[h] = ds[h] - (ps * delta).sum()
        return dq, dk, dv, ds, None, None


def _rotate(x, S, base):
    """Rotate-half rotary embedding of [T, heads, d] with positions 0 .. S - 1 per sequence."""
    T, _, d = x.shape
    inv = 1.0 / (base ** (torch.arange(0, d, 2, dtype=torch.float64, device=DEV) / d))
    a = torch.outer(torch.arange(S, dtype=torch.float64, device=DEV), inv).repeat(T // S, 1)[:, None]
    x1, x2 = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([x1 * a.cos() - x2 * a.sin(), x2 * a.cos() + x1 * a.sin()], -1)


def _self_attention64(x, p, batch, hq, hkv, d, base):
    """Residual stream -> output of the attention block; ``p``: the block's parameters by name, in 64 bits."""
    T = x.shape[0]
    qkv = (_rms(x, p["linear_qkv.layer_norm_weight"]) @ p["linear_qkv.weight"].t()).view(T, hq + 2 * hkv, d)
    q, k, v = qkv[:, :hq], qkv[:, hq:hq + hkv], qkv[:, hq + hkv:]
    if "q_layernorm.weight" in p:
        q, k = _rms(q, p["q_layernorm.weight"]), _rms(k, p["k_layernorm.weight"])
    q, k = _rotate(q, T // batch, base), _rotate(k, T // batch, base)
    return _Attention64.apply(q, k, v, None, batch, 0).reshape(T, hq * d) @ p["linear_proj.weight"].t()


def _leaf64(named):
    return {n: _d(t).requires_grad_() for n, t in named}


def _swiglu64(h):
    a, b = h.chunk(2, -1)
    return F.silu(a) * b


def exact(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    if kind == "norm":
        x, r, w, dy, ds = _norm_inputs(case, g)
        # the sum is defined as rounded to the stream's own type before it is normalised
        s = _d(x if r is None else x + r).requires_grad_()
        w = _d(w).requires_grad_()
        y = _rms(s, w)
        if r is None:
            y.backward(_d(dy))
            return {"y": _d(y), "dx": s.grad, "dw": w.grad}
        torch.autograd.backward([y, s * 1.0], [_d(dy), _d(ds)])
        return {"y": _d(y), "xsum": _d(s), "dx": s.grad, "dr": s.grad, "dw": w.grad}
    if kind == "quantize":
        return None
    if kind == "attn":
        q, k, v = (_d(t).requires_grad_() for t in _attn_inputs(case, g))
        sinks = _d(torch.randn(case["hq"], generator=g, device=DEV)).requires_grad_() if case["sinks"] else None
        do = _randn(g, q.shape[0], case["hq"], case["dv"], std=0.1)
        o = _Attention64.apply(q, k, v, sinks, case["batch"], case["window"])
        o.backward(_d(do))
        out = {"o": _d(o), "dq": q.grad, "dk": k.grad, "dv": v.grad}
        if sinks is not None:
            out["dsinks"] = sinks.grad
        return out
    if kind == "block":
        m, x, d = _block_module(case, seed)
        p = _leaf64(m.named_parameters())
        s = _d(x[0] + x[1]).requires_grad_()
        out = _self_attention64(s, p, case["batch"], case["hq"], case["hkv"], case["d"], 1e6)
        torch.autograd.backward([out, s * 1.0], [_d(t) for t in d])
        return {"out": _d(out), "xsum": _d(s), "dx": s.grad, "dw": [t.grad for t in p.values()]}
    if kind == "mlp":
        t = _mlp_inputs(case, g)
        s = _d(t["hidden"] + t["residual"]).requires_grad_()
        p = _leaf64((n, t[n]) for n in ("norm", "w1", "w2"))
        out = _swiglu64(_rms(s, p["norm"]) @ p["w1"].t()) @ p["w2"].t()
        torch.autograd.backward([out, s * 1.0], [_d(t["dout"]), _d(t["dres"])])
        return {"out": _d(out), "dx": s.grad, "dw": [v.grad for v in p.values()]}
    if kind == "head":
        t = _head_inputs(case, g)
        s = _d(t["hidden"] + t["residual"]).requires_grad_()
        p = _leaf64((n, t[n]) for n in ("norm", "w"))
        loss = (F.cross_entropy(_rms(s, p["norm"]) @ p["w"].t(), t["labels"], reduction="none") * _d(t["weights"])).sum()
        loss.backward()
        return {"loss": _d(loss), "dx": s.grad, "dw": [v.grad for v in p.values()]}
    if kind == "moe":
        m, x, d = _moe_module(case, seed)
        k, E = case["topk"], case["E"]
        x = _d(x).requires_grad_()
        p = _leaf64(m.named_parameters())
        logits = x @ p["router.weight"].t()
        logits = logits + (logits.detach().to(BF16).double() - logits.detach())     # the router reads 16-bit logits
        idx = logits.detach().topk(k, -1).indices
        probs = torch.softmax(logits.gather(1, idx), -1)
        out = torch.zeros_like(x)
        for e in range(E):
            tok, slot = (idx == e).nonzero(as_tuple=True)
            if tok.numel():
                h = _swiglu64(x[tok] @ p["experts.fc1_weight.weight"][e].t()) * probs[tok, slot][:, None]
                out = out.index_add(0, tok, h @ p["experts.fc2_weight.weight"][e].t())
        share = torch.bincount(idx.reshape(-1), minlength=E).double() / idx.numel()
        aux = 1e-3 * E * (share * torch.softmax(logits, -1).mean(0)).sum()
        torch.autograd.backward([out, aux], [_d(d), torch.ones_like(aux)])
        return {"out": _d(out), "dx": x.grad, "dw": [v.grad for v in p.values()]}
    if kind == "optimizer":
        if case["bf16_state"]:
            return None
        gs = _optimizer_inputs(case, g)[1]
        return {"norm": torch.stack([_d(t).pow(2).sum() for t in gs]).sum().sqrt().reshape(1)}
    model, tokens, labels, weights = _model_inputs(case, seed)
    p = _leaf64(model.named_parameters())
    x = p["embedding.word_embeddings.weight"][tokens.reshape(-1)]
    for i in range(case["layers"]):
        pre = "decoder.layers.%d." % i
        attn = {n[len(pre) + 15:]: t for n, t in p.items() if n.startswith(pre + "self_attention.")}
        x = x + _self_attention64(x, attn, case["batch"], case["hq"], case["hkv"], case["d"], 1e4)
        mlp = {n[len(pre) + 4:]: t for n, t in p.items() if n.startswith(pre + "mlp.")}
        x = x + _swiglu64(_rms(x, mlp["linear_fc1.layer_norm_weight"]) @ mlp["linear_fc1.weight"].t()) @ mlp["linear_fc2.weight"].t()
    logits = _rms(x, p["decoder.final_layernorm.weight"]) @ p["output_layer.weight"].t()
    loss = (F.cross_entropy(logits, labels.reshape(-1), reduction="none") * _d(weights).reshape(-1)).sum()
    loss.backward()
    grads = [p[n].grad for n, _ in model.named_parameters()]
    norm = torch.stack([t.pow(2).sum() for t in grads]).sum().sqrt().reshape(1)
    return {"loss": _d(loss), "norm": norm, "params": None, "grads": grads}
