"""Autograd wrapper of the tcgen05 flash-attention forward (csrc/kernels/flash_attn_sm100.cu).

Forward and backward are the hand-written kernels of csrc/kernels/flash2_sm100.cu; the LSE convention (natural log of
the softmax denominator of the scaled scores) is the one ring attention and the reference implementation use, so blocks
computed here can be merged with or differentiated against a global LSE.
"""
from __future__ import annotations

import ctypes
import math

import torch

from . import gemm as G
from . import loader
from .rope import rope_packed_qkv_

def _group_strides(q, nkv):
    """(seq, batch, group, head) strides of q given as [s, b, nq, d] or, by groups of the heads that share a KV head, as
    [s, b, nkv, nq / nkv, d]."""
    if q.dim() == 5:
        return q.stride()[:4]
    return q.stride(0), q.stride(1), q.stride(2) * (q.shape[2] // nkv), q.stride(2)


def flash_fwd(q, k, v, causal, scale, q_offset=None, kernel=2):
    """q [sq,b,nq,128] (or [sq,b,nkv,nq/nkv,128]), k/v [sk,b,nkv,128] bf16 (strided views allowed) -> (o [sq,b,nq,128], lse [b,nq,sq]
    fp32).  ``kernel`` 2 = two query tiles per CTA with P in tensor memory (default), 1 = the single-tile kernel."""
    L = loader.require_lib()
    sq, b = q.shape[:2]
    sk, nkv, d = k.shape[0], k.shape[2], k.shape[3]
    nq = q.shape[2] if q.dim() == 4 else q.shape[2] * q.shape[3]
    for t in (q, k, v):
        if t.stride(-1) != 1 or any((s * 2) % 16 for s in t.stride()[:-1]) or t.data_ptr() % 16:
            raise ValueError("flash_fwd: operands need a contiguous last dim and 16-byte aligned strides")
    o = torch.empty(sq, b, nq, d, dtype=torch.bfloat16, device=q.device)
    lse = torch.empty(b, nq, sq, dtype=torch.float32, device=q.device)
    if q_offset is None:
        q_offset = sk - sq if causal else 0
    ll = ctypes.c_longlong
    st = G.status_word(q.device)
    q_str = _group_strides(q, nkv) if kernel == 2 else q.stride()[:3]
    fn = L.msb_flash_fwd2 if kernel == 2 else L.msb_flash_fwd
    loader.check(fn(loader.p(q), loader.p(k), loader.p(v), loader.p(o), loader.p(lse), sq, sk, b, nq, nkv,
                    *map(ll, (*q_str, *k.stride()[:3], *v.stride()[:3])), int(causal), int(q_offset),
                    ctypes.c_float(scale), loader.p(st), ctypes.c_void_p(loader.stream_ptr())), "flash_fwd")
    return o, lse


def flash_bwd(dout, q, k, v, o, lse, causal, scale, q_offset=None, out=None):
    """Gradients (dq, dk, dv) on the tcgen05 backward kernel.  Shapes as ``flash_fwd``; ``o`` contiguous, ``lse`` the
    forward's (or, for ring attention, the global) log-sum-exp.  dQ is accumulated in fp32 by the key tiles (TMA
    reduce-adds, so its low bits can differ between runs) and rounded to bf16 once at the end.  ``out``: bf16 tensors of the
    shapes of q, k and v (strided views allowed, rows 16-byte aligned) to write into."""
    L = loader.require_lib()
    sq, b = q.shape[:2]
    sk, nkv, d = k.shape[0], k.shape[2], k.shape[3]
    nq = q.shape[2] if q.dim() == 4 else q.shape[2] * q.shape[3]
    if q_offset is None:
        q_offset = sk - sq if causal else 0
    if dout.stride(-1) != 1 or any((st * 2) % 16 for st in dout.stride()[:-1]) or dout.data_ptr() % 16:
        dout = dout.contiguous()
    o = o if o.is_contiguous() else o.contiguous()
    lse = lse if lse.is_contiguous() else lse.contiguous()
    dev = q.device
    sq_pad = (sq + 127) // 128 * 128
    # few (key tile, KV head) pairs would leave most SMs idle: then one CTA per QUERY head, partial dK / dV summed in fp32
    n_ctas = ((sk + 127) // 128) * nkv * b
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    split = nq > nkv and n_ctas < 2 * sms
    acc = torch.empty((sq * nq + (2 * sk * nkv if split else 0)) * b * d, dtype=torch.float32, device=dev)
    dq, dk, dv = out or (torch.empty(t.shape, dtype=torch.bfloat16, device=dev) for t in (q, k, v))
    stats = torch.empty(2, b, nq, sq_pad, dtype=torch.float32, device=dev)
    ll = ctypes.c_longlong
    st = G.status_word(dev)
    strides = (*_group_strides(q, nkv), *k.stride()[:3], *v.stride()[:3], *dout.stride()[:3], *_group_strides(dq, nkv), *dk.stride()[:3],
               *dv.stride()[:3])
    loader.check(L.msb_flash_bwd(loader.p(q), loader.p(k), loader.p(v), loader.p(o), loader.p(dout), loader.p(lse), loader.p(acc),
                                 loader.p(dq), loader.p(dk), loader.p(dv), loader.p(stats[0]), loader.p(stats[1]), int(split), sq, sk, b, nq, nkv,
                                 *map(ll, strides), int(causal), int(q_offset), ctypes.c_float(scale), loader.p(st),
                                 ctypes.c_void_p(loader.stream_ptr())), "flash_bwd")
    return dq, dk, dv


class _FlashFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, causal, scale):
        o, lse = flash_fwd(q, k, v, causal, scale)
        ctx.save_for_backward(q, k, v, o, lse)
        ctx.meta = (causal, scale)
        ctx.mark_non_differentiable(lse)
        return o, lse

    @staticmethod
    def backward(ctx, do, _dlse):
        q, k, v, o, lse = ctx.saved_tensors
        causal, scale = ctx.meta
        dq, dk, dv = flash_bwd(do, q, k, v, o, lse, causal, scale)
        return dq, dk, dv, None, None


def flash_attention(q, k, v, causal, softmax_scale, return_lse):
    scale = softmax_scale if softmax_scale is not None else 1.0 / math.sqrt(q.shape[-1])
    o, lse = _FlashFn.apply(q, k, v, bool(causal), float(scale))
    return (o, lse) if return_lse else o


class _PackedFlash(torch.autograd.Function):
    """Rotary embedding (in place) and attention on a packed QKV activation [s, b, groups * (q_per_group + 2) * d].  The kernels read the
    query heads of a group, its key and its value where they lie, and backward writes the three gradients into one packed tensor."""

    @staticmethod
    def _views(t, groups, qpg):
        v5 = t.view(t.shape[0], t.shape[1], groups, qpg + 2, -1)
        return v5[:, :, :, :qpg], v5[:, :, :, qpg], v5[:, :, :, qpg + 1]

    @staticmethod
    def forward(ctx, qkv, cos, sin, groups, qpg, interleaved, causal, scale):
        ctx.meta = (groups, qpg, interleaved, causal, scale)
        ctx.rope = cos is not None
        if ctx.rope:
            d = qkv.shape[-1] // (groups * (qpg + 2))
            rope_packed_qkv_(qkv, cos, sin, groups, qpg, d, interleaved)
            ctx.mark_dirty(qkv)
        o, lse = flash_fwd(*_PackedFlash._views(qkv, groups, qpg), causal, scale)
        ctx.save_for_backward(qkv, o, lse, *((cos, sin) if ctx.rope else ()))
        ctx.set_materialize_grads(False)
        return (o, qkv) if ctx.rope else (o, None)

    @staticmethod
    def backward(ctx, do, d_rotated):
        groups, qpg, interleaved, causal, scale = ctx.meta
        qkv, o, lse, *angles = ctx.saved_tensors
        if do is None:
            grad = None if d_rotated is None else d_rotated.clone(memory_format=torch.contiguous_format)
        else:
            grad = torch.empty_like(qkv)
            flash_bwd(do, *_PackedFlash._views(qkv, groups, qpg), o, lse, causal, scale, out=_PackedFlash._views(grad, groups, qpg))
            if d_rotated is not None:
                grad += d_rotated
        if grad is not None and ctx.rope:
            rope_packed_qkv_(grad, *angles, groups, qpg, qkv.shape[-1] // (groups * (qpg + 2)), interleaved, backward=True)
        return grad, None, None, None, None, None, None, None


def packed_supports(qkv, groups, qpg) -> bool:
    return (loader.use_kernels(qkv) and qkv.dtype == torch.bfloat16 and qkv.is_contiguous() and qkv.data_ptr() % 16 == 0
            and qkv.numel() > 0 and qkv.shape[-1] == groups * (qpg + 2) * 128)


def flash_attention_packed(qkv, cos, sin, groups, qpg, interleaved, causal, scale):
    """Self attention [s, b, groups * qpg, 128] of a packed QKV activation (see ``packed_supports``), which the rotary embedding (unless
    ``cos`` is None) changes in place."""
    return _PackedFlash.apply(qkv, cos, sin, groups, qpg, bool(interleaved), bool(causal), float(scale))[0]
