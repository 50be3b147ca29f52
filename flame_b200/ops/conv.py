"""Depthwise causal short convolution over packed sequences (``csrc/conv.cu``).

``short_conv(x, weight, bias, meta, activation)``: x ``[T, D]``, weight ``[D, 1, W]`` (the layout of
``nn.Conv1d(D, D, W, groups=D)``), optional SiLU.  Replaces the Triton kernels behind
``fla.modules.ShortConvolution`` (fla/modules/conv/triton/kernels.py:37-345).
"""
from __future__ import annotations

import ctypes
from ctypes import c_int, c_longlong, c_void_p
from typing import Optional

import torch

from . import _lib, linear_attn as la, slots
from .varlen import VarlenMeta

vp, i32, i64 = c_void_p, c_int, c_longlong
_lib.register("fb_short_conv_strips", [i64, i32, i32])
_lib.register("fb_short_conv_fwd", [vp, vp, vp, vp, vp, i64, i32, i32, i64, i64, i32, vp])
_lib.register("fb_short_conv_bwd", [vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, i64, i32, i32, i64, i64, i32, i32, vp])
_lib.register("fb_short_conv4_strips", [i32, vp, i32])
_lib.register("fb_short_conv4_fwd", [i32, vp, i32, vp, vp, i64, i32, vp])
_lib.register("fb_short_conv4_bwd", [i32, vp, i32, vp, vp, vp, i64, i32, i32, vp])
MAX_TOGETHER = 3  # convolutions of one launch


def _ld(x: torch.Tensor) -> int:
    """The distance of the rows of a matrix.  The stride of a single row says nothing: torch takes a ``[1, D]`` block of a wider
    matrix for contiguous and leaves it the wider stride."""
    return x.stride(0) if x.shape[0] > 1 else x.shape[1]


def _rows16(x: torch.Tensor) -> torch.Tensor:
    """``x``, or a dense copy of it: rows whole 16-byte vectors apart, on a 16-byte boundary."""
    ok = x.stride(1) == 1 and _ld(x) % 8 == 0 and _ld(x) >= x.shape[1] and x.data_ptr() % 16 == 0
    return x if ok else _lib.dense(x)


def _table(rows) -> ctypes.Array:
    flat = [v for r in rows for v in r]
    return (i64 * len(flat))(*flat)


class _ShortConv4(torch.autograd.Function):
    """Width 4, up to ``MAX_TOGETHER`` convolutions of the same rows in one launch.  With ``lay`` (``chunked.ChunkLayout``) the
    results come in its padded rows (zeros in the padding) and so do the gradients that come back."""

    @staticmethod
    def forward(ctx, meta, silu, lay, n, *tensors):
        xs, weights, biases = tensors[:n], tensors[n:2 * n], tensors[2 * n:]
        ctx.slots = [slots.of(x) for x in xs]
        T = xs[0].shape[0]
        xs = [_rows16(x) for x in xs]
        (rows, src), pos = (T, None) if lay is None else (lay.Tp, lay.inv_i32), meta.position_ids
        ys = [torch.empty(rows, x.shape[1], dtype=x.dtype, device=x.device) for x in xs]
        ws = [_lib.dense(w.detach()) for w in weights]
        bs = [_lib.dense(b.detach()) if b is not None else None for b in biases]
        table = _table((x.data_ptr(), w.data_ptr(), _lib.ptr(b), y.data_ptr(), x.shape[1], _ld(x), x.shape[1])
                       for x, w, b, y in zip(xs, ws, bs, ys))
        rc = _lib.lib().fb_short_conv4_fwd(n, table, rows, _lib.ptr(src), pos.data_ptr(), T, 1 if silu else 0, _lib.stream_ptr())
        _lib.check(rc, "fb_short_conv4_fwd")
        _lib.count_launch()
        ctx.save_for_backward(*xs, *weights, *biases)
        # the parameters themselves: a recomputation hands back detached tensors without the ``main_grad`` attribute
        ctx.params = weights, biases
        ctx.cfg = silu, n, rows, src, pos, T
        return tuple(ys)

    @staticmethod
    def backward(ctx, *dys):
        silu, n, rows, src, pos, T = ctx.cfg
        saved = ctx.saved_tensors
        xs, weights, biases = [_rows16(x) for x in saved[:n]], saved[n:2 * n], saved[2 * n:]
        L = _lib.lib()
        dxs, gws, gbs = [None] * n, [None] * n, [None] * n
        into_main = [getattr(w, "main_grad", None) is not None and (b is None or getattr(b, "main_grad", None) is not None)
                     for w, b in zip(*ctx.params)]
        for main in (True, False):
            mine = [i for i in range(n) if into_main[i] == main]
            if not mine:
                continue
            table, keep, width = [], [], 0
            for i in mine:
                x, D = xs[i], xs[i].shape[1]
                dy = torch.zeros(rows, D, dtype=x.dtype, device=x.device) if dys[i] is None else _lib.dense(dys[i])
                w, b = _lib.dense(weights[i].detach()), None if biases[i] is None else _lib.dense(biases[i].detach())
                dx = None if ctx.slots[i] is None else ctx.slots[i].take(T, D, x.dtype, x.device)
                if dx is None or _ld(dx) % 2 or dx.data_ptr() % 4:
                    dx = torch.empty(T, D, dtype=x.dtype, device=x.device)
                if main:
                    pw, pb = ctx.params[0][i], ctx.params[1][i]
                    dw, db = pw.main_grad.view(D, 4), None if pb is None else pb.main_grad
                else:
                    dw = torch.empty(D, 4, dtype=torch.float32, device=x.device)
                    db = None if b is None else torch.empty(D, dtype=torch.float32, device=x.device)
                    gws[i], gbs[i] = dw, db
                dxs[i] = dx
                keep += [dy, w, b]
                table.append((x.data_ptr(), dy.data_ptr(), w.data_ptr(), _lib.ptr(b), dx.data_ptr(), dw.data_ptr(), _lib.ptr(db), D,
                              _ld(x), D, _ld(dx)))
                width += D
            table = _table(table)
            partial = torch.empty(L.fb_short_conv4_strips(len(mine), table, rows), width, 5, dtype=torch.float32, device=xs[0].device)
            rc = L.fb_short_conv4_bwd(len(mine), table, rows, _lib.ptr(src), pos.data_ptr(), partial.data_ptr(), T, 1 if silu else 0,
                                      1 if main else 0, _lib.stream_ptr())
            _lib.check(rc, "fb_short_conv4_bwd")
            _lib.count_launch(2)
        gws = [None if g is None else g.view_as(w).to(w.dtype) for g, w in zip(gws, weights)]
        gbs = [None if g is None else g.to(b.dtype) for g, b in zip(gbs, biases)]
        return (None, None, None, None, *dxs, *gws, *gbs)


class _ShortConvFn(torch.autograd.Function):
    """Every other width."""

    @staticmethod
    def forward(ctx, x, weight, bias, meta: VarlenMeta, silu: bool):
        T, D = x.shape
        W = weight.shape[-1]
        x = _rows16(x)
        w2 = _lib.dense(weight.detach().reshape(D, W))
        b2 = _lib.dense(bias.detach()) if bias is not None else None
        y = torch.empty(T, D, dtype=x.dtype, device=x.device)
        pos = meta.position_ids
        rc = _lib.lib().fb_short_conv_fwd(x.data_ptr(), w2.data_ptr(), _lib.ptr(b2), pos.data_ptr(), y.data_ptr(), T, D,
                                          W, _ld(x), _ld(y), 1 if silu else 0, _lib.stream_ptr())
        _lib.check(rc, "fb_short_conv_fwd")
        _lib.count_launch()
        ctx.save_for_backward(x, weight, bias)
        ctx.meta, ctx.silu = meta, silu
        return y

    @staticmethod
    def backward(ctx, dy):
        x, weight, bias = ctx.saved_tensors
        T, D = x.shape
        W = weight.shape[-1]
        L = _lib.lib()
        dy = _lib.dense(dy)
        w2 = _lib.dense(weight.detach().reshape(D, W))
        b2 = _lib.dense(bias.detach()) if bias is not None else None
        dx = torch.empty(T, D, dtype=x.dtype, device=x.device)
        dpre = torch.empty(T, D, dtype=x.dtype, device=x.device)
        strips = int(L.fb_short_conv_strips(T, D, W))
        part = torch.empty(strips, D, W + 1, dtype=torch.float32, device=x.device)
        mg_w = getattr(weight, "main_grad", None)
        mg_b = getattr(bias, "main_grad", None) if bias is not None else None
        use_main = mg_w is not None and (bias is None or mg_b is not None)
        dw = mg_w.view(D, W) if use_main else torch.empty(D, W, dtype=torch.float32, device=x.device)
        db = None
        if bias is not None:
            db = mg_b if use_main else torch.empty(D, dtype=torch.float32, device=x.device)
        # dx is written with the row stride of x
        xs = x if x.is_contiguous() else x.contiguous()
        rc = L.fb_short_conv_bwd(dy.data_ptr(), xs.data_ptr(), w2.data_ptr(), _lib.ptr(b2), ctx.meta.position_ids.data_ptr(),
                                 dx.data_ptr(), dpre.data_ptr(), part.data_ptr(), dw.data_ptr(), _lib.ptr(db), T, D, W,
                                 _ld(xs), _ld(dy), 1 if ctx.silu else 0, 1 if use_main else 0, _lib.stream_ptr())
        _lib.check(rc, "fb_short_conv_bwd")
        _lib.count_launch(3)
        gw = None if use_main else dw.view_as(weight).to(weight.dtype)
        gb = None if (bias is None or use_main) else db.to(bias.dtype)
        return dx, gw, gb, None, None


def _kernel_ok(x: torch.Tensor, weight: torch.Tensor) -> bool:
    return (_lib.available() and x.is_cuda and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16
            and x.shape[1] % 8 == 0 and weight.shape[-1] <= 8)


def short_conv(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], meta: VarlenMeta,
               activation: Optional[str] = "silu") -> torch.Tensor:
    sl = getattr(meta, "sequence_slice", None)
    if sl is not None and weight.shape[-1] > 1:
        return _short_conv_with_halo(x, weight, bias, meta, activation, sl)
    if _kernel_ok(x, weight):
        silu = activation in ("silu", "swish")
        if weight.shape[-1] == 4 and x.shape[0] > 0:
            return _ShortConv4.apply(meta, silu, None, 1, x, weight, bias)[0]
        return _ShortConvFn.apply(x, weight, bias, meta, silu)
    return la.short_conv(x, weight, bias, meta, activation)


def short_convs_in_chunks(xs, weights, biases, meta: VarlenMeta, activation: Optional[str], chunk: int):
    """Several width-4 convolutions of the same rows in one launch, their results ``[Tp, D]`` in the padded rows of
    ``ChunkLayout.of(meta, chunk)`` (zeros in the padding), or None where the kernel does not apply."""
    if (getattr(meta, "sequence_slice", None) is not None or not 0 < len(xs) <= MAX_TOGETHER or xs[0].shape[0] == 0
            or not all(_kernel_ok(x, w) and w.shape[-1] == 4 for x, w in zip(xs, weights))):
        return None
    from .chunked import ChunkLayout
    lay = ChunkLayout.of(meta, chunk)
    if lay.T != xs[0].shape[0]:
        return None
    return _ShortConv4.apply(meta, activation in ("silu", "swish"), None if lay.aligned else lay, len(xs), *xs, *weights, *biases)


class _PositionsOnly:
    """The part of a ``VarlenMeta`` the convolution reads."""

    def __init__(self, position_ids: torch.Tensor) -> None:
        self.position_ids = position_ids


def _short_conv_with_halo(x, weight, bias, meta, activation, sl) -> torch.Tensor:
    """The convolution on one rank's slice of a row that context parallelism cut inside documents: the ``W - 1`` rows
    in front of the slice come from the previous rank (every rank contributes its last ``W - 1`` rows to one
    differentiable all-gather), are put in front of the local rows with the document positions they have, and their
    outputs are dropped.  ``meta.position_ids`` count from the start of the whole document, so the taps' own validity
    rule (a tap reaches back at most ``position`` rows) also decides what the halo may contribute.  Counterpart of fla's
    convolution tail exchange, also an all-gather followed by an index (fla/ops/cp/comm.py:64-169)."""
    from ..parallel.context_parallel import _AllGatherRows
    h = weight.shape[-1] - 1
    assert x.shape[0] >= h, "a context-parallel slice shorter than the convolution"
    tails = _AllGatherRows.apply(x[-h:].contiguous(), sl.group)          # [world * h, D]
    if sl.rank > 0 and sl.continues[sl.rank]:
        halo = tails[(sl.rank - 1) * h: sl.rank * h]
    else:
        halo = torch.zeros(h, x.shape[1], dtype=x.dtype, device=x.device)
    pos = meta.position_ids
    front = pos[:1] - h + torch.arange(h, device=pos.device, dtype=pos.dtype)   # negative: rows of an earlier document
    ext = _PositionsOnly(torch.cat([front, pos]).contiguous())
    y = short_conv(torch.cat([halo, x], 0), weight, bias, ext, activation)[h:]
    # every rank takes part in the gather's backward collective, also one that uses nobody's rows
    return y + tails[:0].sum().to(y.dtype)   # an empty slice: connected to the gather, independent of its values
