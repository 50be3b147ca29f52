"""Column blocks of one matrix whose gradients are written where they belong.

``split_columns(x, sizes)`` hands out column blocks of ``x [T, N]`` as views.  Autograd's own slices zero-fill a full-width matrix
per block and add them up; writing the blocks' gradients side by side afterwards still copies each of them once.  Here every
view carries a ``Slot``: the operator that consumes the view may ask it, in its backward, for the block's columns of the
shared gradient buffer and write there (``take``); what comes back to ``split_columns`` in place needs no copy, anything else is
copied in.

A slot serves ONE consumer: two operators reading the same view would overwrite each other's gradient before autograd adds
them, so a slot is given away once (``of``) and later askers get none.  The buffer belongs to one run of the backward: it
is allocated by that run's first ``take`` and handed to autograd at the end of it; a run that stopped short of it (gradients
asked for at the views only) leaves its buffer to whoever got those gradients, and the next run makes its own.  It also belongs
to the stream it was allocated on: a consumer on another stream gets a matrix of its own, which is copied in.  Runs of one
retained graph in several threads take turns at the holder, so that a run is never handed another one's buffer.
"""
from __future__ import annotations

import threading
from typing import Optional, Tuple

import torch

from . import _lib


class _Holder:
    def __init__(self, width: int) -> None:
        self.width, self.buffer, self.run, self.stream, self.lock = width, None, -1, 0, threading.Lock()

    def give(self, run: int) -> Optional[torch.Tensor]:
        """The buffer of this run, which the holder lets go of; None if it has none (or another run's)."""
        with self.lock:
            if self.run != run:
                return None
            b, self.buffer = self.buffer, None
            return b


class Slot:
    def __init__(self, holder: _Holder, col: int, n: int) -> None:
        self.holder, self.col, self.n, self.given = holder, col, n, False

    def take(self, rows: int, n: int, dtype: torch.dtype, device: torch.device) -> torch.Tensor:
        """``[rows, n]`` columns of the shared gradient buffer (a fresh matrix if they do not match the block)."""
        h = self.holder
        run = torch._C._current_graph_task_id()
        if run == -1:  # not inside a backward run
            return torch.empty(rows, n, dtype=dtype, device=device)
        stream = _lib.stream_ptr() if device.type == "cuda" else 0
        with h.lock:
            if h.buffer is None or h.run != run:
                # rows whole 16-byte vectors apart (of two-byte values), as the projection's GEMMs read them
                h.buffer = torch.empty(rows, -(-h.width // 8) * 8, dtype=dtype, device=device)[:, :h.width]
                h.run, h.stream = run, stream
            b, owner = h.buffer, h.stream
        if n != self.n or owner != stream or b.shape[0] != rows or b.dtype != dtype or b.device != device:
            return torch.empty(rows, n, dtype=dtype, device=device)
        return b[:, self.col:self.col + n]


def of(x: torch.Tensor) -> Optional[Slot]:
    """The slot of a view from ``split_columns``, for its first consumer; None for the others and for every other tensor."""
    s = getattr(x, "_grad_slot", None)
    if s is None or s.given:
        return None
    s.given = True
    return s


def reshaped(x: torch.Tensor, *shape: int) -> torch.Tensor:
    """``x.reshape(shape)`` of a block's rows; the slot goes along."""
    y = x.reshape(*shape)
    s = getattr(x, "_grad_slot", None)
    if s is not None and y.data_ptr() == x.data_ptr():
        y._grad_slot = s
    return y


def _same_place(a: torch.Tensor, b: torch.Tensor) -> bool:
    """Whether two ``[T, n]`` matrices are the same memory (a single row's stride says nothing)."""
    return (a.data_ptr() == b.data_ptr() and a.dtype == b.dtype and a.shape == b.shape
            and all(n == 1 or s == t for n, s, t in zip(a.shape, a.stride(), b.stride())))


class _SplitColumns(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, holder, *sizes):
        ctx.sizes, ctx.dtype, ctx.holder = sizes, x.dtype, holder
        outs, c = [], 0
        for n in sizes:
            outs.append(x[:, c:c + n])
            c += n
        assert c == x.shape[1], (sizes, x.shape)
        return tuple(outs)

    @staticmethod
    def backward(ctx, *grads):
        T = next(g.shape[0] for g in grads if g is not None)
        dev = next(g.device for g in grads if g is not None)
        buf = ctx.holder.give(torch._C._current_graph_task_id())
        if buf is None or buf.shape[0] != T or buf.dtype != ctx.dtype or buf.device != dev:
            parts = [g.to(ctx.dtype) if g is not None else torch.zeros(T, n, dtype=ctx.dtype, device=dev)
                     for g, n in zip(grads, ctx.sizes)]
            return (torch.cat(parts, dim=1), None, *([None] * len(ctx.sizes)))
        c = 0
        for g, n in zip(grads, ctx.sizes):
            dst = buf[:, c:c + n]
            if g is None:
                dst.zero_()
            elif not _same_place(g, dst):
                dst.copy_(g)
            c += n
        return (buf, None, *([None] * len(ctx.sizes)))


def split_columns(x: torch.Tensor, sizes) -> Tuple[torch.Tensor, ...]:
    """Column blocks of ``x [T, sum(sizes)]`` as views (see the module's head)."""
    holder = _Holder(sum(sizes))
    outs = _SplitColumns.apply(x, holder, *sizes)
    c = 0
    for o, n in zip(outs, sizes):
        o._grad_slot = Slot(holder, c, n)
        c += n
    return outs
