"""Query, key and value heads of multi-head latent attention from the up-projections (csrc/kernels/mla_heads.cu).

  mla_heads(q, kv, k_pe, cos, sin, nope)   q [s, b, n, nope + rope], kv [s, b, n, nope + vd], k_pe [s, b, rope]
        -> q and k [s, b, n, nope + rope] with the last ``rope`` columns rotated (the key's shared by all heads), v [s, b, n, vd]
The PyTorch form is the oracle and serves CPU tensors.
reference: mindspeed/core/transformer/multi_head_latent_attention/adaptor.py:23-139.
"""
from __future__ import annotations

import ctypes

import torch

from . import loader
from ._dtypes import CODE, code
from .rope import apply_rope_ref


def mla_heads_ref(q, kv, k_pe, cos, sin, nope, interleaved=False):
    s, b, n, _ = q.shape
    rope = k_pe.shape[-1]
    q_pe = apply_rope_ref(q[..., nope:], cos, sin, interleaved)
    k_pe = apply_rope_ref(k_pe.reshape(s, b, 1, rope), cos, sin, interleaved)
    qf = torch.cat((q[..., :nope], q_pe), dim=-1)
    kf = torch.cat((kv[..., :nope], k_pe.expand(s, b, n, rope)), dim=-1)
    return qf, kf, kv[..., nope:].contiguous()


def _rows_ok(t):
    """Last dimension contiguous, every row on a 16-byte boundary."""
    e = t.element_size()
    return t.stride(-1) == 1 and t.data_ptr() % 16 == 0 and all(st * e % 16 == 0 for st in t.stride()[:-1])


def supports(q, kv, k_pe, cos, sin, nope) -> bool:
    rope, vd = k_pe.shape[-1], kv.shape[-1] - nope
    return (loader.use_kernels(q) and q.dtype == kv.dtype == k_pe.dtype and q.dtype in CODE and q.numel() > 0
            and nope % 8 == 0 and vd > 0 and vd % 8 == 0 and rope % 16 == 0 and 0 < rope <= 2048
            and kv.is_cuda and k_pe.is_cuda and cos.is_cuda and sin.is_cuda
            # what the kernel indexes without asking: the same tokens and heads everywhere, one row of angles per position
            and q.dim() == 4 and q.shape[3] == nope + rope and kv.shape[:3] == q.shape[:3] and k_pe.shape[:-1] == q.shape[:2]
            and tuple(cos.shape) == tuple(sin.shape) == (q.shape[0], rope))


class _MlaHeads(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, kv, k_pe, cos, sin, nope, interleaved):
        q, kv = (t if t.is_contiguous() and t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format) for t in (q, kv))
        if not _rows_ok(k_pe):
            k_pe = k_pe.clone(memory_format=torch.contiguous_format)
        s, b, n, qk = q.shape
        rope, vd = k_pe.shape[-1], kv.shape[-1] - nope
        qf, kf, v = torch.empty_like(q), torch.empty_like(q), torch.empty(s, b, n, vd, dtype=q.dtype, device=q.device)
        ll, L = ctypes.c_longlong, loader.require_lib()
        loader.check(L.msb_mla_heads_fwd(loader.p(q), loader.p(kv), loader.p(k_pe), ll(k_pe.stride(0)), ll(k_pe.stride(1)), loader.p(cos), loader.p(sin),
                                         loader.p(qf), loader.p(kf), loader.p(v), ll(s * b), b, n, nope, rope, vd, int(interleaved), code(q.dtype),
                                         ctypes.c_void_p(loader.stream_ptr())), "mla_heads_fwd")
        ctx.save_for_backward(cos, sin)
        ctx.meta = (nope, rope, vd, interleaved)
        return qf, kf, v

    @staticmethod
    def backward(ctx, dqf, dkf, dv):
        cos, sin = ctx.saved_tensors
        nope, rope, vd, interleaved = ctx.meta
        s, b, n, qk = dqf.shape
        dqf, dkf, dv = (t if _rows_ok(t) else t.clone(memory_format=torch.contiguous_format) for t in (dqf, dkf, dv))
        new = lambda *shape: torch.empty(*shape, dtype=dqf.dtype, device=dqf.device)
        dq, dkv, dk_pe = new(s, b, n, qk), new(s, b, n, nope + vd), new(s, b, rope)
        ll, L = ctypes.c_longlong, loader.require_lib()
        loader.check(L.msb_mla_heads_bwd(*(x for t in (dqf, dkf, dv) for x in (loader.p(t), ll(t.stride(0)), ll(t.stride(1)), ll(t.stride(2)))),
                                         loader.p(cos), loader.p(sin), loader.p(dq), loader.p(dkv), loader.p(dk_pe), ll(s * b), b, n, nope, rope, vd,
                                         int(interleaved), code(dqf.dtype), ctypes.c_void_p(loader.stream_ptr())), "mla_heads_bwd")
        return dq, dkv, dk_pe, None, None, None, None


def mla_heads(q, kv, k_pe, cos, sin, nope, interleaved=False):
    if supports(q, kv, k_pe, cos, sin, nope):
        return _MlaHeads.apply(q, kv, k_pe, cos.float().contiguous(), sin.float().contiguous(), nope, bool(interleaved))
    return mla_heads_ref(q, kv, k_pe, cos, sin, nope, interleaved)
