"""RMSNorm with optional fused residual add and optional output gate.

``rms_norm(x, weight, eps, residual=None, prenorm=False)`` follows the reference module's contract
(fla/modules/layernorm.py:1084-1134): with ``prenorm`` it returns ``(y, residual_out)`` where
``residual_out = x + residual`` is what gets normalised, so a block needs one kernel for "add, then norm".
``rms_norm_gated(x, gate, weight, eps, activation)`` computes ``norm(x) * w * act(gate)`` as
fla/modules/fused_norm_gate.py:992 does for the output of the linear-attention layers.
"""
from __future__ import annotations

from ctypes import c_float, c_int, c_longlong, c_void_p
from typing import Optional

import torch

from . import _lib, slots

vp, i32, i64, f32 = c_void_p, c_int, c_longlong, c_float
_lib.register("fb_rmsnorm_fwd", [vp, vp, vp, vp, vp, vp, vp, i64, i32, f32, i32, vp, i32, i64, vp])
_lib.register("fb_rmsnorm_bwd_rows", [vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, i64, i32, i32, i32, vp, i32, i64, i64, vp])
_lib.register("fb_rmsnorm_bwd_parts", [i64])

_GATE = {None: 0, "swish": 1, "silu": 1, "sigmoid": 2}


def rms_norm_reference(x, weight, eps, residual=None, prenorm=False, gate=None, activation=None):
    r = x if residual is None else x + residual
    rf = r.float()
    y = rf * torch.rsqrt(rf.pow(2).mean(-1, keepdim=True) + eps)
    if weight is not None:
        y = y * weight.float()
    if gate is not None:
        g = gate.float()
        y = y * (g * torch.sigmoid(g) if _GATE[activation] == 1 else torch.sigmoid(g))
    y = y.to(x.dtype)
    return (y, r) if prenorm else y


def _kernel_ok(x: torch.Tensor) -> bool:
    return _lib.available() and x.is_cuda and x.dtype == torch.bfloat16 and x.shape[-1] % 8 == 0


def _gate_rows(gate: torch.Tensor, T: int, heads: int, D: int):
    """``(gate, distance of its tokens)``: ``[T, heads, D]`` as it lies where the kernels can read it (a column block of a wider
    matrix, say), else a dense copy."""
    g = gate.reshape(T, heads, D)
    ld = g.stride(0) if T > 1 else heads * D
    if ld >= heads * D and ld % 8 == 0 and g.data_ptr() % 16 == 0 and g.stride(2) == 1 and (heads == 1 or g.stride(1) == D):
        return g, ld
    return _lib.dense(g), heads * D


class _RMSNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, residual, gate, eps, prenorm, gate_mode, lay):
        """``lay`` (``chunked.ChunkLayout``): x is ``[Tp, heads, D]`` in its padded rows, the result ``[T, heads, D]``; the gradient of x
        comes back padded, with zeros."""
        shape = x.shape
        D = shape[-1]
        x2 = _lib.dense(x.reshape(-1, D))
        heads = 1 if lay is None and gate is None or x.dim() < 3 else shape[-2]
        rows = x2.shape[0] if lay is None else lay.T * heads
        out_shape = shape if lay is None else (lay.T, *shape[1:])
        res2 = None
        if residual is not None:
            res2 = _lib.dense(residual.reshape(-1, D))
        g2, ldg, ctx.slot = None, 0, None
        if gate is not None:
            ctx.slot = slots.of(gate)
            g2, ldg = _gate_rows(gate, rows // heads, heads, D)
        y = torch.empty(rows, D, dtype=x.dtype, device=x.device)
        res_out = torch.empty_like(x2) if (res2 is not None) else None
        rstd = torch.empty(rows, dtype=torch.float32, device=x.device)
        rc = _lib.lib().fb_rmsnorm_fwd(x2.data_ptr(), _lib.ptr(res2), _lib.ptr(weight), _lib.ptr(g2), y.data_ptr(),
                                       _lib.ptr(res_out), rstd.data_ptr(), rows, D, float(eps), gate_mode,
                                       0 if lay is None else lay.rows_i32.data_ptr(), heads, 0 if ldg == heads * D else ldg, _lib.stream_ptr())
        _lib.check(rc, "fb_rmsnorm_fwd")
        _lib.count_launch()
        xin = res_out if res_out is not None else x2
        ctx.save_for_backward(xin, weight, rstd, g2)
        ctx.shape, ctx.gate_mode, ctx.prenorm, ctx.has_res = shape, gate_mode, prenorm, residual is not None
        ctx.lay, ctx.heads, ctx.gate_shape = lay, heads, None if gate is None else gate.shape
        ctx.mark_non_differentiable(rstd)
        if prenorm:
            return y.view(shape), (res_out if res_out is not None else x2).view(shape)
        return y.view(out_shape)

    @staticmethod
    def backward(ctx, dy, dres_out=None):
        xin, weight, rstd, g2 = ctx.saved_tensors
        D, lay, heads = ctx.shape[-1], ctx.lay, ctx.heads
        rows = xin.shape[0]
        dy2 = _lib.dense(dy.reshape(-1, D))
        dres2 = None
        if ctx.prenorm and dres_out is not None:
            dres2 = _lib.dense(dres_out.reshape(-1, D))
        L = _lib.lib()
        dx = torch.empty_like(xin)
        dgate, ldg, lddg = None, 0, 0
        if g2 is not None:
            T = dy2.shape[0] // heads
            g2, ldg = _gate_rows(g2, T, heads, D)
            dgate = None if ctx.slot is None else ctx.slot.take(T, heads * D, xin.dtype, xin.device)
            lddg = heads * D if dgate is None or T == 1 else dgate.stride(0)
            if dgate is None or lddg % 8 or dgate.data_ptr() % 16:
                dgate, lddg = torch.empty(T, heads * D, dtype=xin.dtype, device=xin.device), heads * D
        dw = None
        dw_part = None
        if weight is not None:
            parts = int(L.fb_rmsnorm_bwd_parts(rows))
            dw_part = torch.empty(parts, D, dtype=torch.float32, device=xin.device)
            mg = getattr(weight, "main_grad", None)
            dw = mg if mg is not None else torch.empty(D, dtype=torch.float32, device=xin.device)
        rc = L.fb_rmsnorm_bwd_rows(dy2.data_ptr(), xin.data_ptr(), _lib.ptr(weight), rstd.data_ptr(), _lib.ptr(g2),
                              _lib.ptr(dres2), dx.data_ptr(), _lib.ptr(dgate), _lib.ptr(dw_part), _lib.ptr(dw), rows, D,
                              ctx.gate_mode, 1 if (weight is not None and hasattr(weight, "main_grad")) else 0,
                              0 if lay is None else lay.inv_i32.data_ptr(), heads, 0 if ldg == heads * D else ldg,
                                   0 if lddg == heads * D else lddg, _lib.stream_ptr())
        _lib.check(rc, "fb_rmsnorm_bwd_rows")
        _lib.count_launch(2 if weight is not None else 1)
        dxv = dx.view(ctx.shape)
        gw = None
        if weight is not None and not hasattr(weight, "main_grad"):
            gw = dw.to(weight.dtype)
        gres = dxv if ctx.has_res else None
        ggate = dgate.view(ctx.gate_shape) if dgate is not None else None
        return dxv, gw, gres, ggate, None, None, None, None


def rms_norm(x: torch.Tensor, weight: Optional[torch.Tensor], eps: float = 1e-6,
             residual: Optional[torch.Tensor] = None, prenorm: bool = False):
    if _kernel_ok(x):
        return _RMSNormFn.apply(x, weight, residual, None, eps, prenorm, 0, None)
    return rms_norm_reference(x, weight, eps, residual, prenorm)


def rms_norm_gated(x: torch.Tensor, gate: torch.Tensor, weight: Optional[torch.Tensor], eps: float = 1e-6,
                   activation: str = "swish"):
    if _kernel_ok(x):
        return _RMSNormFn.apply(x, weight, None, gate, eps, False, _GATE[activation], None)
    return rms_norm_reference(x, weight, eps, gate=gate, activation=activation)


def rms_norm_chunks(x: torch.Tensor, lay, weight: Optional[torch.Tensor], eps: float = 1e-6, gate: Optional[torch.Tensor] = None,
                    activation: str = "swish") -> torch.Tensor:
    """The norm of ``x [NC, chunk, heads, D]`` in the rows of ``lay`` (``chunked.ChunkLayout``), gated or not, as ``[T, heads, D]``."""
    if not _kernel_ok(x):
        x = lay.unpack(x)
        return rms_norm(x, weight, eps) if gate is None else rms_norm_gated(x, gate, weight, eps, activation)
    x = x.reshape(lay.Tp, *x.shape[2:])
    return _RMSNormFn.apply(x, weight, None, gate, eps, False, 0 if gate is None else _GATE[activation], None if lay.aligned else lay)
