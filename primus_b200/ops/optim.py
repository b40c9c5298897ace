"""Flat-buffer optimizer kernels: fused AdamW (fp32 master/moments, bf16 param write-back, device-side
clip coefficient and skip flag so a step needs no host sync), sum of squares for the gradient norm,
and small cast / scale helpers.  CPU tensors run equivalent PyTorch code.

Parity: FusedAdam swap-in primus/backends/megatron/patches/torch_fused_adam_patches.py:40-88; gradient
clipping / found-inf handling of Megatron's distributed optimizer (primus/configs/modules/megatron/
trainer_base.yaml:72-118).
"""
from __future__ import annotations

import struct

import numpy as np
import torch

from . import _lib
from .fused import scratch


def adamw_step_(master, exp_avg, exp_avg_sq, grad, param_out, *, lr, beta1, beta2, eps, weight_decay,
                step, grad_scale=None, skip=None):
    """In-place AdamW on flat state: fp32 master weights, fp32 or bf16 moments (both the same dtype).  ``grad`` fp32
    or bf16 (flat); ``param_out`` bf16 or None.

    ``grad_scale``: 1-element fp32 tensor multiplied into the gradient (clip coefficient);
    ``skip``: 1-element int32 tensor, non-zero -> the update is skipped (non-finite gradients)."""
    bc1 = 1.0 - beta1 ** step
    bc2 = 1.0 - beta2 ** step
    n = master.numel()
    if not master.is_cuda:
        if skip is not None and int(skip.item()) != 0:
            return
        g = grad.float()
        if grad_scale is not None:
            g = g * grad_scale.float()
        m32 = exp_avg.float().mul_(beta1).add_(g, alpha=1 - beta1)
        v32 = exp_avg_sq.float().mul_(beta2).addcmul_(g, g, value=1 - beta2)
        exp_avg.copy_(m32)
        exp_avg_sq.copy_(v32)
        denom = (v32 / bc2).sqrt_().add_(eps)
        master.mul_(1 - lr * weight_decay).addcdiv_(m32 / bc1, denom, value=-lr)
        if param_out is not None:
            param_out.copy_(master.to(param_out.dtype))
        return
    assert master.dtype == torch.float32 and master.is_contiguous()
    assert grad.numel() == n and grad.is_contiguous()
    if param_out is not None:
        assert param_out.dtype == torch.bfloat16 and param_out.numel() == n
    assert exp_avg.dtype == exp_avg_sq.dtype and exp_avg.dtype in (torch.float32, torch.bfloat16)
    _lib.call("adamw_ex", master, exp_avg, exp_avg_sq, grad, int(grad.dtype == torch.bfloat16),
              int(exp_avg.dtype == torch.bfloat16), param_out, n,
              float(lr), float(beta1), float(beta2), float(eps), float(weight_decay), float(bc1), float(bc2),
              grad_scale, skip)


def range_table(ranges, start: int, n: int, device):
    """Device table of a bucket of ``n`` elements with the ranges ``[(lo, hi, weight-decay multiplier, learning-rate
    group)]`` (consecutive, from ``start``; ``lo`` multiples of 4 relative to it) for :func:`adamw_ranges_`."""
    R, chunk = len(ranges), _lib.call_ret("adamw_ranges_chunk")
    starts = np.array([r[0] - start for r in ranges], dtype=np.int64)
    first = np.searchsorted(starts, np.arange(0, n, chunk), side="right") - 1
    # one buffer, one copy to the device: starts (8 bytes each), multipliers, groups, first ranges (4 bytes each)
    buf = np.concatenate([starts.view(np.int32), np.array([r[2] for r in ranges], dtype=np.float32).view(np.int32),
                          np.array([r[3] for r in ranges], dtype=np.int32), first.astype(np.int32)])
    t = torch.from_numpy(buf).to(device)
    return t[4 * R:], t[:2 * R].view(torch.int64), t[2 * R:3 * R].view(torch.float32), t[3 * R:4 * R]


def adamw_ranges_(master, exp_avg, exp_avg_sq, grad, param_out, table, **hyper):
    """:func:`adamw_step_` of a whole bucket whose ranges differ in weight decay and learning rate (CUDA tensors, bf16
    ``param_out``).  ``table``: see :func:`range_table`; ``lrs``: the rates of groups 0 to 3."""
    adamw_buckets_([(master, exp_avg, exp_avg_sq, grad, param_out, table)], **hyper)


def adamw_buckets_(buckets, *, lrs, beta1, beta2, eps, weight_decay, step, grad_scale=None, skip=None):
    """:func:`adamw_ranges_` of several buckets ``(master, exp_avg, exp_avg_sq, grad, param_out, table)``, gradients of one type
    and moments of one type, in one launch."""
    rows = []
    g0, m0 = buckets[0][3], buckets[0][1]
    for master, m, v, grad, out, (first, starts, mult, group) in buckets:
        n = master.numel()
        assert master.dtype == torch.float32 and master.is_contiguous() and master.data_ptr() % 16 == 0
        assert grad.numel() == n and grad.is_contiguous() and grad.dtype == g0.dtype
        assert m.dtype == v.dtype == m0.dtype and out.dtype == torch.bfloat16 and out.numel() == n
        rows += [master.data_ptr(), m.data_ptr(), v.data_ptr(), grad.data_ptr(), out.data_ptr(), n, first.data_ptr(),
                 starts.data_ptr(), mult.data_ptr(), group.data_ptr(), starts.numel()]
    assert len(lrs) == 4
    hyper = struct.pack("10f", *lrs, beta1, beta2, eps, weight_decay, 1.0 - beta1 ** step, 1.0 - beta2 ** step)
    _lib.call("adamw_ranges", struct.pack(f"{len(rows)}q", *rows), len(buckets), hyper, int(g0.dtype == torch.bfloat16),
              int(m0.dtype == torch.bfloat16), grad_scale, skip)


def sumsq_(x, out, accumulate=False, nonfinite=None):
    """out[0] (+)= sum(x^2) in fp32 (deterministic two-stage reduction)."""
    if not x.is_cuda:
        s = x.float().pow(2).sum()
        out[0] = out[0] + s if accumulate else s
        if nonfinite is not None and not torch.isfinite(out[0]):
            nonfinite.fill_(1)
        return out
    assert x.is_contiguous()
    P = _lib.call_ret("sumsq_num_partials")
    sc = scratch(x.device, "sumsq", P)
    _lib.call("sumsq", x, int(x.dtype == torch.bfloat16), x.numel(), sc, out, int(accumulate), nonfinite)
    return out


def grad_norm_(xs, out, accumulate=False, clip=None):
    """out[0] (+)= the sums of squares of the tensors ``xs``, added in turn; with ``clip``, the arguments of :func:`clip_coef_` after
    the sum, also the clip coefficient of the result.  CUDA tensors of one type take two launches in all."""
    if not xs or not xs[0].is_cuda or any(x.dtype != xs[0].dtype for x in xs):
        if not accumulate:
            out.zero_()
        for x in xs:
            sumsq_(x, out, accumulate=True)
        if clip is not None:
            clip_coef_(out, **clip)
        return out
    assert all(x.is_contiguous() for x in xs)
    sc = scratch(xs[0].device, "sumsq", len(xs) * _lib.call_ret("sumsq_num_partials"))
    c = clip or {}
    table = struct.pack(f"{2 * len(xs)}q", *[v for x in xs for v in (x.data_ptr(), x.numel())])
    _lib.call("grad_norm", table, len(xs), int(xs[0].dtype == torch.bfloat16), sc, out, int(accumulate),
              float(c.get("max_norm", 0.0)), float(c.get("extra", 1.0)), c.get("coef"), c.get("norm_out"), c.get("skip"),
              int(c.get("check_finite", False)), float(c.get("spike", 0.0)))
    return out


def clip_coef_(sumsq, max_norm, coef, norm_out=None, extra=1.0, skip=None, check_finite=False, spike=0.0):
    """coef = min(1, max_norm/(sqrt(sumsq)+1e-6)) * extra, all on device.  ``skip`` (int32): set to whether ``sumsq`` is not
    finite (``check_finite``) or above ``spike`` (if positive)."""
    if not sumsq.is_cuda:
        if skip is not None:
            bad = ~torch.isfinite(sumsq) if check_finite else torch.zeros_like(sumsq, dtype=torch.bool)
            skip.copy_(bad | (sumsq > spike) if spike > 0 else bad)
        nrm = sumsq[0].sqrt()
        if norm_out is not None:
            norm_out[0] = nrm
        c = torch.clamp(max_norm / (nrm + 1e-6), max=1.0) if max_norm > 0 else torch.tensor(1.0)
        coef[0] = c * extra
        return coef
    _lib.call("clip_coef", sumsq, float(max_norm), float(extra), coef, norm_out, skip, int(check_finite), float(spike))
    return coef


def cast_f32_to_bf16_(src, dst):
    if not src.is_cuda:
        dst.copy_(src.to(dst.dtype))
        return dst
    _lib.call("cast_f32_bf16", src, dst, src.numel())
    return dst
