"""Fused gate arithmetic of the linear-attention layers (one kernel pass each way instead of a chain of elementwise
framework kernels).

``hgrn2_gates(q_raw, f_raw, lower_bound)`` returns ``(q, k, g)`` of fla/layers/hgrn2.py:160-190:
``q = silu(q_raw)``, ``g = logsigmoid(f_raw)`` (with a lower bound: ``g = log(lb + (1 - lb) sigmoid(f_raw))``, the closed
form of the reference's ``logaddexp(log lb, log1p(-lb) + logsigmoid f)``), ``k = 1 - exp(g)``; ``g`` in fp32.

``logsigmoid_gate(x, normalizer, slots)`` returns ``g = logsigmoid(x) / normalizer`` in fp32 and, with ``slots``,
``1 - exp(g)`` (fla/layers/gla.py:205-212, fla/layers/gsa.py:173-176).
"""
from __future__ import annotations

from ctypes import c_float, c_int, c_longlong, c_void_p
from typing import Optional, Tuple

import torch
import torch.nn.functional as F

from . import _lib, linear_attn as la, slots
from .slots import split_columns  # noqa: F401 - part of this module's interface

_lib.register("fb_hgrn2_gate_tiles", [c_longlong])
_lib.register("fb_hgrn2_gate_fwd", [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_void_p])
_lib.register("fb_hgrn2_gate_bwd", [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                    c_void_p, c_longlong, c_int, c_void_p])


_lib.register("fb_logsigmoid_gate_fwd", [c_void_p, c_longlong] + [c_void_p] * 3 + [c_float] + [c_longlong] * 2 + [c_void_p])
_lib.register("fb_logsigmoid_gate_bwd", [c_void_p, c_longlong] + [c_void_p] * 4 + [c_longlong, c_float] + [c_longlong] * 2 + [c_void_p])


def hgrn2_gates_reference(q_raw: torch.Tensor, f_raw: torch.Tensor,
                          lower_bound: Optional[torch.Tensor]) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    q = F.silu(q_raw)
    g = F.logsigmoid(f_raw.float())
    if lower_bound is not None:
        lb = lower_bound.float()
        g = torch.logaddexp(lb.log(), torch.log1p(-lb) + g)
    k = (1 - g.exp()).to(q_raw.dtype)
    return q, k, g


def logsigmoid_gate_reference(x: torch.Tensor, normalizer: float, with_slots: bool = False):
    g = F.logsigmoid(x.float()) / normalizer
    return (g, 1 - g.exp()) if with_slots else g


def _gate_rows(x: torch.Tensor):
    """``(rows, columns, distance of rows)`` of a gate's argument as the kernels read it, None if they cannot."""
    if x.data_ptr() % 16 or x.dim() < 2 or x.numel() == 0:
        return None
    T, cols = x.shape[0], x.numel() // x.shape[0]
    if x.is_contiguous() and cols % 8 == 0:
        return T, cols, cols
    try:
        ld = x.view(T, cols).stride(0) if T > 1 else cols
    except RuntimeError:
        return None
    return (T, cols, ld) if cols % 8 == 0 and ld % 8 == 0 and ld >= cols else None


class _LogSigmoidGate(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, normalizer, with_slots, lay):
        """``lay`` (``chunked.ChunkLayout``): the results are in its padded rows ``[NC, chunk, ...]``, zeros in the padding."""
        ctx.slot = slots.of(x)
        T, cols, ld = _gate_rows(x) or (1, x.numel(), x.numel())
        shape = x.shape if lay is None else (lay.NC, lay.chunk, *x.shape[1:])
        src = None if lay is None or lay.aligned else lay.inv_i32
        g = torch.empty(shape, dtype=torch.float32, device=x.device)
        s = torch.empty_like(g) if with_slots else None
        rc = _lib.lib().fb_logsigmoid_gate_fwd(x.data_ptr(), ld, _lib.ptr(src), g.data_ptr(), _lib.ptr(s), normalizer, T if lay is None else lay.Tp, cols,
                                               _lib.stream_ptr())
        _lib.check(rc, "fb_logsigmoid_gate_fwd")
        _lib.count_launch()
        ctx.save_for_backward(x)
        ctx.cfg = normalizer, with_slots, lay, shape
        return (g, s) if with_slots else g

    @staticmethod
    def backward(ctx, dg, ds=None):
        x, = ctx.saved_tensors
        normalizer, with_slots, lay, shape = ctx.cfg

        def full(d):
            return torch.zeros(shape, dtype=torch.float32, device=x.device) if d is None else _lib.dense(d.float())

        dg, ds = full(dg), full(ds) if with_slots else None
        rows = _gate_rows(x)
        if rows is None:
            x = x.contiguous()
            rows = _gate_rows(x) or (1, x.numel(), x.numel())
        T, cols, ld = rows
        dx = None if ctx.slot is None or T != x.shape[0] else ctx.slot.take(T, cols, x.dtype, x.device)
        if dx is None or (T > 1 and dx.stride(0) % 8) or dx.data_ptr() % 16:
            dx = torch.empty(T, cols, dtype=x.dtype, device=x.device)
        src = None if lay is None or lay.aligned else lay.rows_i32
        rc = _lib.lib().fb_logsigmoid_gate_bwd(x.data_ptr(), ld, _lib.ptr(src), dg.data_ptr(), _lib.ptr(ds), dx.data_ptr(),
                                               dx.stride(0) if T > 1 else cols, normalizer, T, cols, _lib.stream_ptr())
        _lib.check(rc, "fb_logsigmoid_gate_bwd")
        _lib.count_launch()
        return dx.view(x.shape), None, None, None


def logsigmoid_gate(x: torch.Tensor, normalizer: float, with_slots: bool = False, lay=None):
    """``logsigmoid(x) / normalizer`` in fp32, and ``1 - exp`` of it with ``with_slots``.  One pass for bf16 on the GPU, contiguous or a
    column block whose rows are whole vectors; anything else (other types, odd sizes) takes torch's chain.  ``lay``: results in the
    padded rows of a ``chunked.ChunkLayout``."""
    if _lib.available() and x.is_cuda and x.dtype == torch.bfloat16 and (lay is None or x.shape[0] == lay.T) and \
            (_gate_rows(x) is not None or (lay is None and x.is_contiguous() and x.numel() % 8 == 0 and x.data_ptr() % 16 == 0)):
        return _LogSigmoidGate.apply(x, float(normalizer), with_slots, lay)
    out = logsigmoid_gate_reference(x, normalizer, with_slots)
    if lay is None:
        return out
    return tuple(lay.pack(t) for t in out) if with_slots else lay.pack(out)


class _Hgrn2Gates(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q_raw, f_raw, lb):
        rows, D = q_raw.shape
        q_raw, f_raw = _lib.dense(q_raw), _lib.dense(f_raw)
        lbf = lb.detach().float().contiguous() if lb is not None else None
        q, k = torch.empty_like(q_raw), torch.empty_like(q_raw)
        g = torch.empty(rows, D, dtype=torch.float32, device=q_raw.device)
        rc = _lib.lib().fb_hgrn2_gate_fwd(q_raw.data_ptr(), f_raw.data_ptr(), _lib.ptr(lbf), q.data_ptr(), k.data_ptr(),
                                          g.data_ptr(), rows, D, _lib.stream_ptr())
        _lib.check(rc, "fb_hgrn2_gate_fwd")
        _lib.count_launch()
        ctx.save_for_backward(q_raw, f_raw, lbf)
        ctx.lb_dtype = lb.dtype if lb is not None else None
        return q, k, g

    @staticmethod
    def backward(ctx, dq, dk, dg):
        q_raw, f_raw, lbf = ctx.saved_tensors
        rows, D = q_raw.shape
        L = _lib.lib()
        dq = torch.zeros_like(q_raw) if dq is None else _lib.dense(dq)
        dk = torch.zeros_like(q_raw) if dk is None else _lib.dense(dk)
        dg = torch.zeros(rows, D, dtype=torch.float32, device=q_raw.device) if dg is None else _lib.dense(dg.float())
        dq_raw, df_raw = torch.empty_like(q_raw), torch.empty_like(f_raw)
        part = dlb = None
        if lbf is not None:
            part = torch.empty(int(L.fb_hgrn2_gate_tiles(rows)), D, dtype=torch.float32, device=q_raw.device)
            dlb = torch.empty(D, dtype=torch.float32, device=q_raw.device)
        rc = L.fb_hgrn2_gate_bwd(q_raw.data_ptr(), f_raw.data_ptr(), _lib.ptr(lbf), dq.data_ptr(), dk.data_ptr(), dg.data_ptr(),
                                 dq_raw.data_ptr(), df_raw.data_ptr(), _lib.ptr(part), _lib.ptr(dlb), rows, D, _lib.stream_ptr())
        _lib.check(rc, "fb_hgrn2_gate_bwd")
        _lib.count_launch(2 if lbf is not None else 1)
        return dq_raw, df_raw, (dlb.to(ctx.lb_dtype) if dlb is not None else None)


def hgrn2_gates(q_raw: torch.Tensor, f_raw: torch.Tensor,
                lower_bound: Optional[torch.Tensor] = None) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """``[T, D]`` bf16 projections (and an optional ``[D]`` lower bound) -> ``q`` bf16, ``k`` bf16, ``g`` fp32, all ``[T, D]``."""
    if (_lib.available() and q_raw.is_cuda and q_raw.dtype == torch.bfloat16 and f_raw.dtype == torch.bfloat16
            and q_raw.dim() == 2 and q_raw.shape == f_raw.shape and q_raw.shape[1] % 8 == 0):
        return _Hgrn2Gates.apply(q_raw, f_raw, lower_bound)
    return hgrn2_gates_reference(q_raw, f_raw, lower_bound)


# ----------------------------------------------------------------------------------------------------------------------
# Mamba2: the elementwise work around the SSD core (fla/layers/mamba2.py:241-331)
# ----------------------------------------------------------------------------------------------------------------------
_lib.register("fb_mamba2_pre_fwd", [c_void_p, c_longlong, c_void_p, c_longlong, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                    c_void_p, c_longlong, c_int, c_int, c_void_p])
_lib.register("fb_mamba2_pre_bwd", [c_void_p, c_longlong, c_void_p, c_longlong, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                    c_void_p, c_longlong, c_void_p, c_void_p, c_longlong, c_int, c_int, c_void_p])
_lib.register("fb_mamba2_post_fwd", [c_void_p, c_void_p, c_longlong, c_void_p, c_longlong, c_void_p, c_void_p, c_void_p, c_longlong, c_int,
                                     c_int, c_void_p])
_lib.register("fb_mamba2_post_bwd", [c_void_p, c_void_p, c_longlong, c_void_p, c_longlong, c_void_p, c_void_p, c_void_p, c_void_p,
                                     c_void_p, c_longlong, c_void_p, c_void_p, c_longlong, c_int, c_int, c_void_p])


def _views_ok(*ts: torch.Tensor) -> bool:
    return all(t.is_cuda and t.dtype == torch.bfloat16 and t.dim() == 2 and t.stride(1) == 1 and t.stride(0) % 8 == 0
               and t.data_ptr() % 16 == 0 for t in ts)


class _Mamba2Pre(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, dt_raw, dt_bias, A_log, H, P, lay):
        """``lay`` (``chunked.ChunkLayout``): x and the results are in its padded rows, ``dt_raw`` is per token.  The last result is x
        itself for its other reader, whose gradient the backward kernel adds."""
        ctx.set_materialize_grads(False)
        T = x.shape[0]
        ctx.src = None if lay is None or lay.aligned else lay.inv_i32
        bias32, alog32 = dt_bias.detach().float().contiguous(), A_log.detach().float().contiguous()
        xv = torch.empty(T, H, P, dtype=x.dtype, device=x.device)
        dt = torch.empty(T, H, dtype=torch.float32, device=x.device)
        g = torch.empty(T, H, dtype=torch.float32, device=x.device)
        rc = _lib.lib().fb_mamba2_pre_fwd(x.data_ptr(), x.stride(0), dt_raw.data_ptr(), dt_raw.stride(0), bias32.data_ptr(),
                                          alog32.data_ptr(), xv.data_ptr(), dt.data_ptr(), g.data_ptr(), _lib.ptr(ctx.src), T, H, P,
                                          _lib.stream_ptr())
        _lib.check(rc, "fb_mamba2_pre_fwd")
        _lib.count_launch()
        ctx.save_for_backward(x, dt_raw, bias32, alog32, dt)
        ctx.dims, ctx.x_slot = (H, P), slots.of(x)
        ctx.dtypes = (dt_bias.dtype, A_log.dtype, dt_raw.dtype)
        return xv, dt, g, x.view_as(x)

    @staticmethod
    def backward(ctx, dxv, ddt, dg, dskip):
        x, dt_raw, bias32, alog32, dt = ctx.saved_tensors
        H, P = ctx.dims
        T = x.shape[0]
        dxv = torch.zeros(T, H, P, dtype=x.dtype, device=x.device) if dxv is None else _lib.dense(dxv)
        dg = torch.zeros(T, H, dtype=torch.float32, device=x.device) if dg is None else _lib.dense(dg.float())
        ddt = None if ddt is None else ddt.float().contiguous()
        dskip = None if dskip is None else _lib.dense(dskip.to(x.dtype))
        dx = None if ctx.x_slot is None else ctx.x_slot.take(T, H * P, x.dtype, x.device)
        if dx is None or not _views_ok(dx):
            dx = torch.empty(T, H * P, dtype=x.dtype, device=x.device)
        d_raw = torch.empty(dt_raw.shape[0], H, dtype=torch.float32, device=x.device)
        rc = _lib.lib().fb_mamba2_pre_bwd(x.data_ptr(), x.stride(0), dt_raw.data_ptr(), dt_raw.stride(0), bias32.data_ptr(),
                                          alog32.data_ptr(), dxv.data_ptr(), dg.data_ptr(), _lib.ptr(ddt), _lib.ptr(dskip),
                                          dx.data_ptr(), dx.stride(0), d_raw.data_ptr(), _lib.ptr(ctx.src), T, H, P, _lib.stream_ptr())
        _lib.check(rc, "fb_mamba2_pre_bwd")
        _lib.count_launch()
        d_bias = d_raw.sum(0)
        d_alog = (dg * dt).sum(0) * (-alog32.exp())     # g = A dt with A = -exp(A_log): dA_log = dA * A
        return (dx, d_raw.to(ctx.dtypes[2]), d_bias.to(ctx.dtypes[0]), d_alog.to(ctx.dtypes[1]), None, None, None)


class _Mamba2Post(torch.autograd.Function):
    @staticmethod
    def forward(ctx, y, x, z, D, H, P, lay):
        """``lay``: y and x are in its padded rows, z and the result per token."""
        T = x.shape[0]
        ctx.src = None if lay is None or lay.aligned else lay.inv_i32
        y = _lib.dense(y)
        d32 = D.detach().float().contiguous()
        out = torch.empty(z.shape[0], H * P, dtype=x.dtype, device=x.device)
        rc = _lib.lib().fb_mamba2_post_fwd(y.data_ptr(), x.data_ptr(), x.stride(0), z.data_ptr(), z.stride(0), d32.data_ptr(),
                                           out.data_ptr(), _lib.ptr(ctx.src), T, H, P, _lib.stream_ptr())
        _lib.check(rc, "fb_mamba2_post_fwd")
        _lib.count_launch()
        ctx.save_for_backward(y, x, z, d32)
        ctx.dims, ctx.d_dtype, ctx.z_slot = (H, P), D.dtype, slots.of(z)
        return out

    @staticmethod
    def backward(ctx, dout):
        y, x, z, d32 = ctx.saved_tensors
        H, P = ctx.dims
        T = x.shape[0]
        dout = _lib.dense(dout)
        dy = torch.empty(T, H, P, dtype=x.dtype, device=x.device)
        dx = torch.empty(T, H * P, dtype=x.dtype, device=x.device)
        n = z.shape[0]
        dz = ctx.z_slot.take(n, H * P, x.dtype, x.device) if ctx.z_slot is not None else torch.empty(n, H * P, dtype=x.dtype, device=x.device)
        if not _views_ok(dz):
            dz = torch.empty(n, H * P, dtype=x.dtype, device=x.device)
        part = torch.empty(T, H, dtype=torch.float32, device=x.device)
        rc = _lib.lib().fb_mamba2_post_bwd(y.data_ptr(), x.data_ptr(), x.stride(0), z.data_ptr(), z.stride(0), d32.data_ptr(),
                                           dout.data_ptr(), dy.data_ptr(), dx.data_ptr(), dz.data_ptr(), dz.stride(0), part.data_ptr(), _lib.ptr(ctx.src), T, H, P,
                                           _lib.stream_ptr())
        _lib.check(rc, "fb_mamba2_post_bwd")
        _lib.count_launch()
        return dy, dx, dz, part.sum(0).to(ctx.d_dtype), None, None, None


def mamba2_pre_reference(x, dt_raw, dt_bias, A_log, H: int, P: int):
    T = x.shape[0]
    dt = F.softplus(dt_raw.float() + dt_bias.float())
    g = dt * (-torch.exp(A_log.float()))[None, :]
    xv = (x.reshape(T, H, P).float() * dt[..., None]).to(x.dtype)
    return xv, dt, g


def mamba2_post_reference(y, x, z, D, H: int, P: int):
    T = x.shape[0]
    u = y.reshape(T, H, P).float() + x.reshape(T, H, P).float() * D.float()[None, :, None]
    return (u.reshape(T, H * P) * F.silu(z.float())).to(x.dtype)


def mamba2_kernels(x, dt_raw, z, P: int) -> bool:
    """Whether both of the functions below run on their kernels, which also take padded rows (``lay``)."""
    return _lib.available() and P in (64, 128, 256) and _views_ok(x, z) and dt_raw.is_cuda and dt_raw.dtype == torch.bfloat16 and dt_raw.stride(1) == 1


def mamba2_pre(x, dt_raw, dt_bias, A_log, H: int, P: int, lay=None):
    """``x [T, H * P]`` and ``dt_raw [T, H]`` (strided views are fine) -> ``xv = x dt`` ``[T, H, P]``, ``dt = softplus(dt_raw +
    dt_bias)`` and the log decay ``g = -exp(A_log) dt`` (both fp32 ``[T, H]``), in one kernel."""
    return mamba2_pre_skip(x, dt_raw, dt_bias, A_log, H, P, lay)[:3]


def mamba2_pre_skip(x, dt_raw, dt_bias, A_log, H: int, P: int, lay=None):
    """``mamba2_pre`` and x once more: the skip connection reads that, and x's two gradients meet in the backward kernel."""
    if mamba2_kernels(x, dt_raw, x, P):
        return _Mamba2Pre.apply(x, dt_raw, dt_bias, A_log, H, P, lay)
    if lay is None:
        return (*mamba2_pre_reference(x, dt_raw, dt_bias, A_log, H, P), x)
    out = mamba2_pre_reference(x.index_select(0, lay.rows), dt_raw, dt_bias, A_log, H, P)
    return (*(lay.pack(t).flatten(0, 1) for t in out), x)


def mamba2_post(y, x, z, D, H: int, P: int, lay=None):
    """``(y + D x) silu(z)`` as ``[T, H * P]`` in one kernel; ``x`` and ``z`` may be strided views."""
    if _lib.available() and P in (64, 128, 256) and _views_ok(x, z) and y.is_cuda and y.dtype == torch.bfloat16:
        return _Mamba2Post.apply(y, x, z, D, H, P, lay)
    if lay is not None:
        y, x = y.index_select(0, lay.rows), x.index_select(0, lay.rows)
    return mamba2_post_reference(y, x, z, D, H, P)


_lib.register("fb_delta_gates_blocks", [c_longlong, c_int])
_lib.register("fb_delta_gates_fwd", [c_void_p, c_longlong] * 2 + [c_void_p] * 2 + [c_int, c_void_p, c_longlong, c_int, c_float] + [c_void_p] * 3)
_lib.register("fb_delta_gates_bwd", [c_void_p, c_longlong] * 2 + [c_void_p] * 2 + [c_int, c_void_p, c_longlong, c_int, c_float] + [c_void_p] * 2
              + [c_void_p, c_longlong] * 2 + [c_void_p] * 3 + [c_int, c_void_p])
_DELTA_GATES_MAX_HEADS = 128


class _DeltaGates(torch.autograd.Function):
    @staticmethod
    def forward(ctx, b, a, A_log, dt_bias, mul, lay):
        ctx.slots = slots.of(b), None if a is None else slots.of(a)
        rows, H = lay.Tp, b.shape[1]
        src = None if lay.aligned else lay.inv_i32
        beta = torch.empty(lay.NC, lay.chunk, H, dtype=torch.float32, device=b.device)
        g = None if a is None else torch.empty_like(beta)
        rc = _lib.lib().fb_delta_gates_fwd(*_DeltaGates._inputs(b, a, A_log, dt_bias), _lib.ptr(src), rows, H, mul, beta.data_ptr(),
                                           _lib.ptr(g), _lib.stream_ptr())
        _lib.check(rc, "fb_delta_gates_fwd")
        _lib.count_launch()
        ctx.save_for_backward(b, a, A_log, dt_bias)
        ctx.params, ctx.cfg = (A_log, dt_bias), (mul, lay, src)
        return beta, g

    @staticmethod
    def _inputs(b, a, A_log, dt_bias):
        return (b.data_ptr(), b.stride(0), _lib.ptr(a), 0 if a is None else a.stride(0), _lib.ptr(A_log), _lib.ptr(dt_bias),
                int(A_log is not None and A_log.dtype == torch.bfloat16))

    @staticmethod
    def backward(ctx, dbeta, dg):
        b, a, A_log, dt_bias = ctx.saved_tensors
        (mul, lay, src), H, dev = ctx.cfg, b.shape[1], b.device
        rows = lay.Tp

        def dense(d):
            return torch.zeros(rows, H, dtype=torch.float32, device=dev) if d is None else _lib.dense(d.float())

        def out(x, slot):
            y = None if slot is None else slot.take(lay.T, H, x.dtype, dev)
            return torch.empty(lay.T, H, dtype=x.dtype, device=dev) if y is None else y
        dbeta, db = dense(dbeta), out(b, ctx.slots[0])
        dA = ddt = da = part = None
        main = False
        L = _lib.lib()
        if a is not None:
            dg, da = dense(dg), out(a, ctx.slots[1])
            need = ctx.needs_input_grad[2:4]
            main = all(getattr(p, "main_grad", None) is not None for p, n in zip(ctx.params, need) if n)
            dA, ddt = (None if not n else p.main_grad if main else torch.empty(H, dtype=torch.float32, device=dev) for p, n in zip(ctx.params, need))
            part = torch.empty(L.fb_delta_gates_blocks(rows, H), 2, H, dtype=torch.float32, device=dev)
        rc = L.fb_delta_gates_bwd(*_DeltaGates._inputs(b, a, A_log, dt_bias), _lib.ptr(src), rows, H, mul, dbeta.data_ptr(), _lib.ptr(dg) if a is not None else 0,
                                  db.data_ptr(), db.stride(0), _lib.ptr(da), 0 if da is None else da.stride(0), _lib.ptr(part),
                                  _lib.ptr(dA), _lib.ptr(ddt), int(main), _lib.stream_ptr())
        _lib.check(rc, "fb_delta_gates_bwd")
        _lib.count_launch(1 if a is None else 2)
        gA, gdt = (None if main or d is None else d.to(p.dtype) for d, p in ((dA, A_log), (ddt, dt_bias)))
        return db, da, gA, gdt, None, None


def delta_gates_torch(b: torch.Tensor, a: Optional[torch.Tensor], A_log, dt_bias, mul: float):
    """The same per token, ``[T, H]``."""
    beta = b.float().sigmoid()
    if mul != 1.0:
        beta = beta * mul
    return beta, None if a is None else la.gdn_gate(a, A_log, dt_bias)


def delta_gates(b: torch.Tensor, a: Optional[torch.Tensor], A_log, dt_bias, mul: float, lay):
    """``beta = mul sigmoid(b)`` and, with ``a``, the log decay ``-exp(A_log) softplus(a + dt_bias)`` of ``[T, H]`` bf16 projections, in fp32
    ``[NC, chunk, H]`` in the rows of ``lay`` (``chunked.ChunkLayout``); None where the kernel does not apply."""
    ok = _lib.available() and b.is_cuda and b.dtype == torch.bfloat16 and b.stride(-1) == 1 and b.shape[0] == lay.T and b.shape[1] <= _DELTA_GATES_MAX_HEADS
    if a is not None:
        ok = ok and (a.dtype, a.shape, a.stride(-1)) == (b.dtype, b.shape, 1) and A_log.dtype == dt_bias.dtype and \
            A_log.dtype in (torch.bfloat16, torch.float32) and A_log.is_contiguous() and dt_bias.is_contiguous()
    return _DeltaGates.apply(b, a, A_log, dt_bias, float(mul), lay) if ok else None
