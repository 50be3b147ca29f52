"""SwiGLU on a fused ``[T, 2I]`` gate/up buffer: ``a = silu(gate) * up``.

The backward writes ``d_gate`` and ``d_up`` side by side into one ``[T, 2I]`` buffer so the weight gradient
of the fused gate/up projection is a single GEMM.  Same math as fla/modules/activations.py:553-628.
"""
from __future__ import annotations

from ctypes import c_int, c_longlong, c_void_p

import torch
import torch.nn.functional as F

from . import _lib, slots

vp, i32, i64 = c_void_p, c_int, c_longlong
_lib.register("fb_swiglu_fwd", [vp, vp, vp, i64, i32, i64, i64, i64, vp])
_lib.register("fb_swiglu_bwd", [vp, vp, vp, vp, vp, vp, i64, i32, i64, i64, i64, i64, i64, i64, vp])


def swiglu_reference(gu: torch.Tensor) -> torch.Tensor:
    g, u = gu.chunk(2, dim=-1)
    return F.silu(g) * u


class _SwiGLUFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gu):
        shape = gu.shape
        I = shape[-1] // 2
        gu2 = _lib.dense(gu.reshape(-1, 2 * I))
        T = gu2.shape[0]
        a = swiglu_forward(gu2, torch.empty(T, I, dtype=gu.dtype, device=gu.device))
        ctx.save_for_backward(gu2)
        ctx.shape = shape
        return a.view(*shape[:-1], I)

    @staticmethod
    def backward(ctx, da):
        (gu2,) = ctx.saved_tensors
        return swiglu_backward(_lib.dense(da.reshape(-1, gu2.shape[1] // 2)), _lib.dense(gu2)).view(ctx.shape)


def swiglu_forward(gu2: torch.Tensor, a: torch.Tensor) -> torch.Tensor:
    """``a [T, I] = silu(gate) * up`` of ``[gate | up] [T, 2 I]``, both contiguous."""
    T, I = a.shape
    rc = _lib.lib().fb_swiglu_fwd(gu2.data_ptr(), gu2.data_ptr() + 2 * I, a.data_ptr(), T, I, 2 * I, 2 * I, I, _lib.stream_ptr())
    _lib.check(rc, "fb_swiglu_fwd")
    _lib.count_launch()
    return a


def swiglu_backward(da2: torch.Tensor, gu2: torch.Tensor) -> torch.Tensor:
    """``[d_gate | d_up]`` for ``a = silu(gate) * up`` from ``da [T, I]`` and the saved ``[gate | up] [T, 2 I]``."""
    T, I2 = gu2.shape
    I = I2 // 2
    dgu = torch.empty_like(gu2)
    rc = _lib.lib().fb_swiglu_bwd(da2.data_ptr(), gu2.data_ptr(), gu2.data_ptr() + 2 * I, dgu.data_ptr(),
                                  dgu.data_ptr() + 2 * I, 0, T, I, I, I2, I2, I2, I2, I, _lib.stream_ptr())
    _lib.check(rc, "fb_swiglu_bwd")
    _lib.count_launch()
    return dgu


def swiglu(gu: torch.Tensor) -> torch.Tensor:
    if _lib.available() and gu.is_cuda and gu.dtype == torch.bfloat16 and (gu.shape[-1] // 2) % 8 == 0:
        return _SwiGLUFn.apply(gu)
    return swiglu_reference(gu)


_lib.register("fb_silu_rows", [vp, i64, vp, i64, i32, vp, vp, vp, i64, i32, vp])


class _SiluRows(torch.autograd.Function):
    """SiLU of neighbouring column blocks of ``x [rows, *]``, each to a matrix of its own: ``y_p[r] = silu(x[there[r], block p])``, zero rows where
    ``there`` is negative; ``back`` is the inverse map (both None: the same rows)."""

    @staticmethod
    def forward(ctx, x, sizes, rows, there, back, slot):
        ys = [torch.empty(rows, n, dtype=x.dtype, device=x.device) for n in sizes]
        _SiluRows._launch(x, None, ys, there, rows, 0)
        ctx.save_for_backward(x)
        ctx.cfg = sizes, rows, back, slot
        return tuple(ys)

    @staticmethod
    def _launch(x, dx, ys, rows_map, rows, backward):
        p = (vp * len(ys))(*(y.data_ptr() for y in ys))
        n = (i32 * len(ys))(*(y.shape[1] for y in ys))
        ld = lambda t: t.stride(0) if t.shape[0] > 1 else -(-t.shape[1] // 8) * 8  # noqa: E731
        rc = _lib.lib().fb_silu_rows(x.data_ptr(), ld(x), _lib.ptr(dx), 0 if dx is None else ld(dx), len(ys), p, n, _lib.ptr(rows_map), rows,
                                     backward, _lib.stream_ptr())
        _lib.check(rc, "fb_silu_rows")
        _lib.count_launch()

    @staticmethod
    def backward(ctx, *dys):
        x, = ctx.saved_tensors
        sizes, rows, back, slot = ctx.cfg
        x = x if _rows_ok(x) else x.contiguous()
        dys = [torch.zeros(rows, n, dtype=x.dtype, device=x.device) if d is None else _lib.dense(d) for d, n in zip(dys, sizes)]
        dx = None if slot is None else slot.take(x.shape[0], x.shape[1], x.dtype, x.device)
        if dx is None or not _rows_ok(dx):
            dx = torch.empty(x.shape, dtype=x.dtype, device=x.device)
        _SiluRows._launch(x, dx, dys, back, x.shape[0], 1)
        return dx, None, None, None, None, None


def _rows_ok(x: torch.Tensor) -> bool:
    return x.stride(1) == 1 and (x.shape[0] == 1 or (x.stride(0) % 8 == 0 and x.stride(0) >= x.shape[1])) and x.data_ptr() % 16 == 0


def silu_blocks_to_chunks(x: torch.Tensor, sizes, lay):
    """SiLU of the column blocks of ``x [T, sum(sizes)]`` (up to three) in the padded rows of ``lay`` (``chunked.ChunkLayout``), ``[Tp, n]`` each, zeros
    in the padding; None where the kernel does not apply."""
    if not (_lib.available() and x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2 and x.shape == (lay.T, sum(sizes)) and len(sizes) <= 3
            and all(n % 8 == 0 for n in sizes) and _rows_ok(x)):
        return None
    maps = (None, None) if lay.aligned else (lay.inv_i32, lay.rows_i32)
    return _SiluRows.apply(x, tuple(sizes), lay.Tp, *maps, slots.of(x))


def silu_out_of_chunks(o: torch.Tensor, lay) -> torch.Tensor:
    """``silu(lay.unpack(o))`` as ``[T, n]`` for ``o [NC, chunk, ...]`` in the rows of ``lay``."""
    o = o.reshape(lay.Tp, -1)
    if not (_lib.available() and o.is_cuda and o.dtype == torch.bfloat16 and o.shape[1] % 8 == 0 and _rows_ok(o)):
        return F.silu(lay.unpack(o.reshape(lay.NC, lay.chunk, -1)))
    maps = (None, None) if lay.aligned else (lay.rows_i32, lay.inv_i32)
    return _SiluRows.apply(o, (o.shape[1],), lay.T, *maps, None)[0]
