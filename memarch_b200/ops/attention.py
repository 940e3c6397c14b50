"""Causal / sliding-window attention with RoPE for the light and final blocks.

Reference behaviour: `F.scaled_dot_product_attention(rope(q), rope(k), v, is_causal=True)` when the text fits the
window (full.py:156-157); block-masked window attention `kv <= q and q - kv < window` otherwise (FlexAttention with
an O(T) block list, full2.py:153-181; two-block variants lm.py:448-554).

GPU body, head dim 64, where `own_core` says so: the own tcgen05 kernels on the packed projections (`_QkvAttn`, `csrc/attn_fwd.cu`,
`csrc/attn_bwd.cu`: q and k rotated, v read in place, gradients written rotated back into the packed layout).  Otherwise
`rope_qk` (rotation of the q and k thirds of the packed qkv activations, `rope_merge_bwd`
packs and rotates the three gradients back in one pass) around the library flash kernel.
"""
from __future__ import annotations

import os

import torch
import torch.nn.functional as F

from . import _ext, ref
from .basic import dense

ATTN_CORE = os.environ.get("MEMARCH_ATTN", "auto")             # auto | own | lib: see `own_core`
OWN_WINDOW_EVAL = os.environ.get("MEMARCH_ATTN_EVAL", "own") == "own"
OWN_CAUSAL_T, OWN_CAUSAL_WORK = 512, 100_000                   # plain causal texts: length, words x heads in all; see `own_core`
OWN_BWD = os.environ.get("MEMARCH_ATTN_BWD", "own") == "own"
WINDOW_BODY = os.environ.get("MEMARCH_WINDOW", "flash")        # library body of windowed attention with backward: flash | block


_tables = {}


def rope_tables(T, hd, device):
    """(T, hd/2) fp32 cos / sin tables, built once per (T, hd, device)."""
    key = (T, hd, str(device))
    if key not in _tables:
        cos, sin = ref.rope_angles(T, hd, device)
        _tables[key] = (cos.contiguous(), sin.contiguous())
    return _tables[key]


class _RopeQK(torch.autograd.Function):
    """Rotate the q and k slices of qkv (B,T,3,H,hd); v passes through.  Backward rotates the grads back."""

    @staticmethod
    def forward(ctx, qkv, half):
        ctx.half = half
        cos, sin = rope_tables(qkv.shape[1], qkv.shape[4], qkv.device)
        _ext.count()
        return _ext.C().rope_qk(dense(qkv), cos, sin, 1.0, bool(half))

    @staticmethod
    def backward(ctx, g):
        cos, sin = rope_tables(g.shape[1], g.shape[4], g.device)
        _ext.count()
        return _ext.C().rope_qk(dense(g), cos, sin, -1.0, bool(ctx.half)), None


class _RopeSplit(torch.autograd.Function):
    """Rotate q,k and hand q,k,v to the attention core as (B,H,T,hd) views of one packed tensor.  Backward takes the
    three separate gradients (any batch/head/token strides), rotates back and packs them in one pass."""

    @staticmethod
    def forward(ctx, qkv, half):
        ctx.half = half
        cos, sin = rope_tables(qkv.shape[1], qkv.shape[4], qkv.device)
        _ext.count()
        r = _ext.C().rope_qk(dense(qkv), cos, sin, 1.0, bool(half))
        return r[:, :, 0].transpose(1, 2), r[:, :, 1].transpose(1, 2), r[:, :, 2].transpose(1, 2)

    @staticmethod
    def backward(ctx, dq, dk, dv):
        cos, sin = rope_tables(dq.shape[2], dq.shape[3], dq.device)
        fix = lambda t: t if (t.stride(3) == 1 and t.stride(0) % 8 == 0 and t.stride(1) % 8 == 0 and t.stride(2) % 8 == 0
                            and t.data_ptr() % 16 == 0) else dense(t)
        _ext.count()
        return _ext.C().rope_merge_bwd(fix(dq), fix(dk), fix(dv), cos, sin, bool(ctx.half)), None


class _OwnAttn(torch.autograd.Function):
    """Attention core on the own tcgen05 kernels (`csrc/attn_fwd.cu`, `csrc/attn_bwd.cu`): S = QKt, O = PV and the five
    backward products on the tensor cores with TMEM accumulators, block lists from window arithmetic, exact LSE.  `MEMARCH_ATTN_BWD=lib` makes backward recompute through the library instead."""

    @staticmethod
    def forward(ctx, q, k, v, window):
        C = _ext.C()
        qc, kc, vc = q.contiguous(), k.contiguous(), v.contiguous()
        o, lse = C.attn_fwd_tc(qc, kc, vc, int(window), float(q.shape[-1]) ** -0.5)
        _ext.count()
        ctx.save_for_backward(qc, kc, vc, o, lse)
        ctx.window = int(window)
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse = ctx.saved_tensors
        if OWN_BWD:
            dq, dk, dv = _ext.C().attn_bwd_tc(q, k, v, o, do.contiguous(), lse, ctx.window, float(q.shape[-1]) ** -0.5)
            _ext.count(3)
            return dq, dk, dv, None
        q, k, v = (t.detach().requires_grad_() for t in (q, k, v))
        with torch.enable_grad():
            o2 = F.scaled_dot_product_attention(q, k, v, is_causal=True) if ctx.window == 0 else _lib_window(q, k, v, ctx.window)
        dq, dk, dv = torch.autograd.grad(o2, (q, k, v), do)
        return dq, dk, dv, None


def own_attention(q, k, v, window=0):
    """q, k, v (B,H,T,64) bf16 with RoPE applied -> o (B,H,T,64); `window` 0 = plain causal."""
    return _OwnAttn.apply(q, k, v, int(window or 0))


class _QkvAttn(torch.autograd.Function):
    """RoPE + causal / sliding-window attention on packed projections qkv (B,T,3,H,64) -> (B,T,H*64), window 0 = plain
    causal.  Forward rotates q and k; for a backward pass one packed array is kept, with v beside them (without one, v is read
    where the projection left it).  Backward writes dq, dk (rotated back) and dv straight into one packed gradient."""

    @staticmethod
    def forward(ctx, qkv, window, half):
        B, T, _, H, hd = qkv.shape
        cos, sin = rope_tables(T, hd, qkv.device)
        keep = ctx.needs_input_grad[0]
        o, lse, rot = _ext.C().attn_qkv_fwd(qkv, cos, sin, bool(half), int(window), keep, False)
        _ext.count(2)
        if keep:
            ctx.save_for_backward(o, lse, rot)
        ctx.window, ctx.half = int(window), bool(half)
        return o.view(B, T, H * hd)

    @staticmethod
    def backward(ctx, do):
        o, lse, rot = ctx.saved_tensors
        cos, sin = rope_tables(rot.shape[1], rot.shape[4], rot.device)
        _ext.count(3)
        return _ext.C().attn_qkv_bwd(dense(do), o, lse, rot, cos, sin, ctx.half, ctx.window), None, None


def _lib_window(q, k, v, window):
    """Two-block dense-mask window attention through SDPA: each block of `window` queries sees itself and the
    previous block (2·window keys); linear cost in T."""
    B, H, T, D = q.shape
    W = window
    nb = -(-T // W)
    pad = nb * W - T
    if pad:
        q, k, v = (F.pad(t, (0, 0, 0, pad)) for t in (q, k, v))
    qb, kb, vb = (t.reshape(B, H, nb, W, D) for t in (q, k, v))
    prev = lambda t: torch.cat([torch.zeros_like(t[:, :, :1]), t[:, :, :-1]], 2)
    kk, vv = torch.cat([prev(kb), kb], 3), torch.cat([prev(vb), vb], 3)
    i = torch.arange(W, device=q.device)[:, None]
    j = torch.arange(2 * W, device=q.device)[None]
    ok = (j > i) & (j <= i + W)
    first = torch.arange(nb, device=q.device)[:, None, None] > 0
    mask = ok[None] & (first | (j >= W)[None])
    qb, kk, vv = qb.reshape(B, H * nb, W, D), kk.reshape(B, H * nb, 2 * W, D), vv.reshape(B, H * nb, 2 * W, D)
    mask = mask[None].expand(H, nb, W, 2 * W).reshape(1, H * nb, W, 2 * W)
    out = F.scaled_dot_product_attention(qb, kk, vv, attn_mask=mask)
    return out.reshape(B, H, nb * W, D)[:, :, :T]


_flash_window_ok = [None]


def _flash_window(q, k, v, window):
    """Sliding-window causal attention through the library flash kernel's own window arguments (key j is visible to
    query i iff 0 <= i - j < window): cost proportional to the window, forward and backward.  q, k, v (B,H,T,hd).
    Falls back to the two-block dense-mask form if this build of the library has no windowed flash kernel."""
    if _flash_window_ok[0] is not False and WINDOW_BODY == "flash":
        try:
            T = q.shape[2]
            o = torch.ops.aten._flash_attention_forward(
                q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), None, None, T, T, 0.0, True, False,
                scale=None, window_size_left=int(window) - 1, window_size_right=0)[0]
            _flash_window_ok[0] = True
            return o.transpose(1, 2)
        except Exception:   # noqa: BLE001 - older library: no window arguments / unsupported head size
            if _flash_window_ok[0] is True:
                raise
            _flash_window_ok[0] = False
    return _lib_window(q, k, v, window)


def own_core(B, T, H, windowed, no_grad):
    """Whether head-dim-64 attention runs on the own kernels.  `MEMARCH_ATTN=own`: always.  `lib`: only windows without a backward
    pass, and those only with `MEMARCH_ATTN_EVAL=own` (the default).  `auto`, the default: windows and short causal texts (with a backward pass
    only few of them), but windows without a backward pass as `MEMARCH_ATTN_EVAL` says."""
    # Us, own against library core, forward + backward.  Windows: 2 x 16 384 words, 16 heads, window 256: 700 / 1221; 4 x 4096, window
    # 1024: 635 / 1242.  Causal, 4 texts, 8 heads, 256, 512, 768 and 1024 words: 70 / 184, 76 / 162, 101 / 158, 117 / 159 (the library's
    # time is the host's); 16 texts, 12 heads, 256, 384, 512, 640 and 1024 words: 101 / 175, 157 / 163, 177 / 182, 212 / 206,
    # 372 / 288; 32 texts, 32 heads, 256, 384, 512 and 1024 words: 303 / 289, 536 / 473, 632 / 582, 1594 / 1364: full, the chip does the
    # library's one backward kernel faster.  Forward alone, 32 texts, 32 heads, 256, 384 and 512 words: 73 / 87, 143 / 169, 181 / 175.
    if ATTN_CORE == "own":
        return True
    if windowed and no_grad:
        return OWN_WINDOW_EVAL
    return ATTN_CORE != "lib" and (windowed or (T <= OWN_CAUSAL_T and (no_grad or B * T * H <= OWN_CAUSAL_WORK)))


def attention(qkv, window=None, rope_half=False, qk_norm=False):
    """qkv (B,T,3,H,hd) -> (B,T,H·hd).  `window` None or >= T means plain causal."""
    B, T, _, H, hd = qkv.shape
    win = None if (window is None or window >= T) else int(window)
    if _ext.use_cuda(qkv) and qkv.dtype == torch.bfloat16 and not qk_norm and hd % 8 == 0:
        no_grad = not (torch.is_grad_enabled() and qkv.requires_grad)
        own = own_core(B, T, H, win is not None, no_grad)
        if hd == 64 and own and (no_grad or OWN_BWD):
            return _QkvAttn.apply(dense(qkv.detach() if no_grad else qkv), win or 0, rope_half)
        q, k, v = _RopeSplit.apply(qkv, rope_half)
        if hd == 64 and own:
            return own_attention(q, k, v, win or 0).transpose(1, 2).reshape(B, T, H * hd)
        o = F.scaled_dot_product_attention(q, k, v, is_causal=True) if win is None else _flash_window(q, k, v, win)
        return o.transpose(1, 2).reshape(B, T, H * hd)
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    o = ref.window_attention(q, k, v, win, rope_half, qk_norm=qk_norm)
    return o.reshape(B, T, H * hd)
