"""The two halves of a light layer as one autograd node and one native call each way (`csrc/block.cpp`).

Same kernels and same arithmetic as the sequence of single ops in `models.blocks.LightBlock.forward`, which serves every
option and shape these do not take.  Two things differ: the gradient that reaches the residual stream past a half is summed
inside the norm's backward pass instead of by autograd, and a weight gradient that autograd will accumulate into an fp32
weight leaves its GEMM in fp32 instead of being rounded to bf16 and cast back.
"""
from __future__ import annotations

import torch
from torch.autograd.forward_ad import unpack_dual

from . import _ext, basic
from .attention import OWN_BWD, own_core, rope_tables


def _trained(w):
    return w.dtype == torch.float32 and w.is_leaf and w.requires_grad and w.is_contiguous()


def _operand(w):
    return basic.shadow_bf16(w) if torch.is_grad_enabled() else basic.dense(basic.weight_bf16(w))


def _common(x, nw, ws):
    if not (_ext.use_cuda(x) and basic.PLAIN_GEMM == "tc" and x.dim() == 3 and x.dtype == torch.float32
            and x.shape[2] % 16 == 0 and x.shape[2] <= 8192 and x.shape[0] * x.shape[1] >= 256):
        return False
    if torch.is_grad_enabled():
        # every weight trained and the stream part of the graph, as in a training step
        return x.requires_grad and nw.requires_grad and all(_trained(w) for w in ws)
    return all(w.dtype in (torch.float32, torch.bfloat16) for w in ws) and _no_tangent(x, nw, *ws)


def _no_tangent(*ts):
    """Without gradients no autograd node stands around the native call: forward-mode derivatives are left to the single ops,
    whose nodes refuse them, instead of being lost."""
    return all(unpack_dual(t).tangent is None for t in ts)


def attn_half_ok(x, pending, nw, wqkv, wo, heads, window):
    """Head dim 64 and lengths that the own attention kernels serve (see `ops.attention.own_core`)."""
    B, T, d = x.shape
    no_grad = not torch.is_grad_enabled()
    return (d == heads * 64 and own_core(B, T, heads, window is not None and window < T, no_grad) and (OWN_BWD or no_grad)
            and wqkv.shape == (3 * d, d) and wo.shape == (d, d) and _common(x, nw, (wqkv, wo))
            and (pending is None or (pending.dtype == torch.bfloat16 and pending.shape == x.shape and (not no_grad or _no_tangent(pending)))))


def ffn_half_ok(h, a, nw, wup, wdown, swiglu):
    N, d = wup.shape
    H = N // 2 if swiglu else N
    return (a.dtype == torch.bfloat16 and a.shape == h.shape and d == h.shape[2] and wdown.shape == (d, H) and N % 16 == 0 and H % 8 == 0
            and (basic.FUSE_DSWIGLU or not swiglu) and _common(h, nw, (wup, wdown)) and (torch.is_grad_enabled() or _no_tangent(a)))


def _taker(ws):
    """(what the native call hands each weight's gradient to as soon as it is enqueued, the gradients it did not keep); without a
    taker of gradients (None, None): the call returns them."""
    if basic.WEIGHT_GRAD_SINK is None:
        return None, None
    left = [None, None]

    def offer(i, g):
        left[i] = basic.offer_grad(ws[i], g)
    return offer, left


class _AttnHalf(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, pending, nw, wqkv, wo, eps, window, half):
        T = x.shape[1]
        cos, sin = rope_tables(T, 64, x.device)
        sq, so = basic.shadow_bf16(wqkv), basic.shadow_bf16(wo)
        h, a, *kept = _ext.C().attn_half_fwd(x, pending, nw, eps, sq, so, cos, sin, half, window)
        _count(x, 4 * x.shape[2], 5)
        ctx.save_for_backward(h, *kept, nw, sq, so)
        ctx.ws, ctx.window, ctx.half, ctx.has_pending, ctx.shape = (wqkv, wo), window, half, pending is not None, x.shape
        ctx.set_materialize_grads(False)
        return (h.view(x.shape) if pending is not None else x), a.view(x.shape)

    @staticmethod
    def backward(ctx, dh, da):
        h, n, rstd, qkv, o, lse, nw, sq, so = ctx.saved_tensors
        if da is None:
            if dh is None:
                return (None,) * 8
            da = torch.zeros(ctx.shape, device=dh.device, dtype=torch.bfloat16)
        cos, sin = rope_tables(ctx.shape[1], 64, h.device)
        offer, left = _taker(ctx.ws)
        dx, lo, dnw, *dws = _ext.C().attn_half_bwd(da, dh, h, n, rstd, qkv, o, lse, nw, sq, so, cos, sin, ctx.half, ctx.window,
                                                   ctx.has_pending, offer is None, offer)
        _count(dx, 8 * dx.shape[1], 9)
        return (dx.view(ctx.shape), lo.view(ctx.shape) if ctx.has_pending else None, dnw.to(nw.dtype),
                *(left or dws), None, None, None)


class _FFNHalf(torch.autograd.Function):
    @staticmethod
    def forward(ctx, h, a, nw, wup, wdown, eps, swiglu, add_out):
        su, sd = basic.shadow_bf16(wup), basic.shadow_bf16(wdown)
        x2, y, *kept = _ext.C().ffn_half_fwd(h, a, nw, eps, su, sd, swiglu, add_out)
        _count(h, wup.shape[0] + wdown.shape[1], 4 if add_out else 3)
        ctx.save_for_backward(x2, *kept, nw, su, sd)
        ctx.ws, ctx.swiglu, ctx.add_out, ctx.shape = (wup, wdown), swiglu, add_out, h.shape
        ctx.set_materialize_grads(False)
        return y.view(h.shape) if add_out else (x2.view(h.shape), y.view(h.shape))

    @staticmethod
    def backward(ctx, *grads):
        x2, n, rstd, pre, hid, nw, su, sd = ctx.saved_tensors
        dx2, dy = (None, grads[0]) if ctx.add_out else grads
        if dy is None:
            if dx2 is None:
                return (None,) * 8
            dy = torch.zeros(ctx.shape, device=x2.device, dtype=torch.bfloat16)
        offer, left = _taker(ctx.ws)
        dh, da, dnw, *dws = _ext.C().ffn_half_bwd(dy, dx2, x2, n, rstd, pre, hid, nw, su, sd, ctx.swiglu, offer is None, offer)
        wup, wdown = ctx.ws
        _count(dh, 2 * (wup.shape[0] + wdown.shape[1]), 6)
        return dh.view(ctx.shape), da.view(ctx.shape), dnw.to(nw.dtype), *(left or dws), None, None, None


def _count(x, width, launches):
    """Launch and FLOP counters: `width` columns of weights of x.shape[-1] rows each."""
    _ext.count(launches)
    _ext.count_flops(2 * x.numel() * width)


def attn_half(x, pending, nw, wqkv, wo, eps, window, half):
    """(x + pending, attention of its norm projected by wo); `window` 0 = plain causal.  Only after `attn_half_ok`."""
    if torch.is_grad_enabled():
        return _AttnHalf.apply(x, pending, nw, wqkv, wo, eps, window, half)
    cos, sin = rope_tables(x.shape[1], 64, x.device)
    h, a = _ext.C().attn_half_fwd(x, pending, nw, eps, _operand(wqkv), _operand(wo), cos, sin, half, window)[:2]
    _count(x, 4 * x.shape[2], 5)
    return h.view(x.shape), a.view(x.shape)


def ffn_half(h, a, nw, wup, wdown, eps, swiglu, add_out):
    """(h + a, feed-forward of its norm), or their sum with `add_out`.  Only after `ffn_half_ok`."""
    if torch.is_grad_enabled():
        return _FFNHalf.apply(h, a, nw, wup, wdown, eps, swiglu, add_out)
    x2, y = _ext.C().ffn_half_fwd(h, a, nw, eps, _operand(wup), _operand(wdown), swiglu, add_out)[:2]
    _count(h, wup.shape[0] + wdown.shape[1], 4 if add_out else 3)
    return y.view(h.shape) if add_out else (x2.view(h.shape), y.view(h.shape))
