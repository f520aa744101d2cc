"""Row gather / weighted scatter-add for MoE token permutation (csrc/kernels/permute.cu)."""
from __future__ import annotations

import ctypes

import torch

from . import gemm as G
from . import loader
from ._dtypes import CODE, code


class _Gather(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, idx):
        L = loader.require_lib()
        x = x.contiguous()
        idx = idx.contiguous().long()
        out = torch.empty(idx.numel(), x.shape[1], dtype=x.dtype, device=x.device)
        loader.check(L.msb_gather_rows(loader.p(x), loader.p(idx), loader.p(out), ctypes.c_longlong(idx.numel()), x.shape[1],
                                       code(x.dtype), ctypes.c_void_p(loader.stream_ptr())), "gather_rows")
        ctx.save_for_backward(idx)
        ctx.rows = x.shape[0]
        return out

    @staticmethod
    def backward(ctx, g):
        (idx,) = ctx.saved_tensors
        return _scatter(g.contiguous(), idx, ctx.rows, None), None


def _scatter(src, idx, rows, weight):
    L = loader.require_lib()
    out = torch.empty(rows, src.shape[1], dtype=src.dtype, device=src.device)
    n, cols = idx.numel(), src.shape[1]
    full = min(rows, n // 9)                  # most output rows that more than eight source rows can name
    scratch = torch.empty(full * ((cols + 7) // 8 * 4) + 10 * rows + 3 + 5 * full + 2 * n + 2 * (n // 32), dtype=torch.int64, device=src.device)
    loader.check(L.msb_scatter_add_rows(loader.p(src), loader.p(idx), loader.p(weight), loader.p(out), loader.p(scratch), ctypes.c_longlong(n),
                                        ctypes.c_longlong(rows), cols, code(src.dtype), ctypes.c_void_p(loader.stream_ptr())), "scatter_add_rows")
    return out


class _ScatterAdd(torch.autograd.Function):
    @staticmethod
    def forward(ctx, src, idx, rows, weight):
        idx = idx.contiguous().long()
        src = src.contiguous()
        w = None if weight is None else weight.float().contiguous()
        ctx.save_for_backward(src, idx, w if w is not None else torch.empty(0, device=src.device))
        ctx.has_w = w is not None
        ctx.wdtype = None if weight is None else weight.dtype
        return _scatter(src, idx, rows, w)

    @staticmethod
    def backward(ctx, g):
        src, idx, w = ctx.saved_tensors
        g = g.contiguous()
        gs = _Gather.apply(g, idx)
        dw = None
        if ctx.has_w:
            dw = (gs.float() * src.float()).sum(-1).to(ctx.wdtype)
            gs = gs * w.unsqueeze(-1).to(gs.dtype)
        return gs, None, None, dw


def gather_rows(x, idx):
    return _Gather.apply(x, idx)


def scatter_add_rows(src, idx, rows, weight=None):
    return _ScatterAdd.apply(src, idx, rows, weight)


def add_rows_(out, idx, src):
    """out[idx[r]] += src[r] where idx[r] >= 0; ``out`` fp32 contiguous [rows, cols], rows may repeat (sums in no fixed order)."""
    L = loader.require_lib()
    loader.check(L.msb_add_rows_f32(loader.p(src), loader.p(idx), loader.p(out), ctypes.c_longlong(idx.numel()), src.shape[1],
                                    code(src.dtype), ctypes.c_void_p(loader.stream_ptr())), "add_rows_f32")
    return out


class _RouteTables(torch.autograd.Function):
    @staticmethod
    def forward(ctx, probs, routing_map, rows):
        L = loader.require_lib()
        T, E = routing_map.shape
        probs = probs.contiguous()
        found, counts = (torch.empty(E, dtype=torch.int64, device=probs.device) for _ in range(2))
        idx = torch.zeros(rows, dtype=torch.int64, device=probs.device)
        row_prob = torch.zeros(rows, dtype=probs.dtype, device=probs.device)
        loader.check(L.msb_moe_route(loader.p(routing_map.contiguous()), loader.p(probs), loader.p(found), loader.p(counts), loader.p(idx),
                                     loader.p(row_prob), ctypes.c_longlong(T), E, ctypes.c_longlong(rows), code(probs.dtype),
                                     loader.p(G.status_word(probs.device)), ctypes.c_void_p(loader.stream_ptr())), "moe_route")
        ctx.save_for_backward(idx, counts)
        ctx.shape = (T, E)
        ctx.mark_non_differentiable(idx, counts)
        return idx, row_prob, counts

    @staticmethod
    def backward(ctx, _didx, g, _dcounts):
        idx, counts = ctx.saved_tensors
        L = loader.require_lib()
        T, E = ctx.shape
        g = g.contiguous()
        dprobs = torch.empty(T, E, dtype=g.dtype, device=g.device)
        loader.check(L.msb_moe_route_bwd(loader.p(g), loader.p(idx), loader.p(counts), loader.p(dprobs), ctypes.c_longlong(T), E,
                                         ctypes.c_longlong(idx.numel()), code(g.dtype), ctypes.c_void_p(loader.stream_ptr())), "moe_route_bwd")
        return dprobs, None, None


def route_supports(probs, routing_map) -> bool:
    return (loader.use_kernels(probs) and routing_map.is_cuda and routing_map.dtype == torch.bool and routing_map.dim() == 2
            and probs.shape == routing_map.shape and probs.dtype in CODE and routing_map.numel() > 0)


def route_tables(probs, routing_map, rows):
    """probs / routing_map [T, E], ``rows`` = number of entries of the map -> (token of every dispatched row, expert after expert and
    inside an expert by token [rows]; its probability [rows], differentiable; rows per expert [E]), all on the device.  Where the map has
    another number of entries, what does not fit is left out and ``ops.gemm.check_status`` raises."""
    return _RouteTables.apply(probs, routing_map, rows)
