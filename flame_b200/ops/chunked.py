"""Chunk-parallel token mixers on the batched tcgen05 GEMM: gated delta rule, delta rule, scalar-gated linear
attention (Mamba2 SSD).

Layout.  Packed tokens ``[T, H, d]`` are re-packed so that every document starts on a chunk boundary (``ChunkLayout``;
chunks of C = 64 or 128 tokens, fewer than C zero rows per document).  In that layout ``[NC, C, H, d]`` every chunk of every head is
one batch of a strided batched GEMM, a zero row contributes nothing (k = v = 0, decay 1), and the whole algorithm
is a short list of batched GEMMs plus elementwise work:

  scores      Akk = strict_tril(beta k k^T e^{b_i-b_j}),  Aqk = tril(scale q k^T e^{b_i-b_j})   (decay + mask in the epilogue)
  WY          T = (I + Akk)^-1,  u = T (beta v),  w = T (beta e^{b} k)
  transition  M_c = khat_c^T w_c,  B_c = khat_c^T u_c          khat = k e^{b_last - b}
  recurrence  S_{c+1} = e^{b_last} S_c - M_c S_c + B_c         one batched GEMM per chunk position, all documents at once
  output      v_new = u - w S,   o = (scale q e^{b}) S + Aqk v_new

The recurrence is the only sequential part; writing the chunk transition as the matrix ``M_c`` turns each step into
a plain GEMM on the state, so it also runs on the batched kernel (state kept in fp32, bf16 mirror as the operand).
The reverse recurrence of the backward pass uses the same launches with ``M_c^T``.

Covers the reference's chunk_gated_delta_rule / chunk_delta_rule / Mamba2 SSD paths
(fla/ops/gated_delta_rule/chunk.py, fla/ops/delta_rule/chunk.py, fla/ops/common/chunk_delta_h.py,
fla/ops/common/chunk_o.py, fla/layers/mamba2.py).
"""
from __future__ import annotations

import math
from typing import List, Optional

import torch

from ctypes import c_int, c_longlong, c_void_p

from . import _lib, slots
from .bgemm import MASK_STRICT, MASK_TRIL, _mask, bgemm, bmm
from .varlen import VarlenMeta

CHUNK = 64
_lib.register("fb_gather_rows", [c_void_p, c_void_p, c_void_p, c_longlong, c_longlong, c_longlong, c_longlong, c_void_p])
_lib.register("fb_delta_scan", [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int,
                                c_int, c_void_p])


# --------------------------------------------------------------------------------------------------------
# recomputation of a token mixer in the backward pass
# --------------------------------------------------------------------------------------------------------
_recompute_mixers = False


def set_mixer_recompute(flag: bool) -> None:
    """With the flag set, the chunk-parallel token mixers below keep only their inputs for the backward pass and run
    their chunk pipeline again there (``--activation_checkpoint.mode selective --activation_checkpoint.selective_ac_option
    mixer``): the pipeline's intermediates - packed operands, WY factors and above all one ``dk x dv`` state per chunk
    and head - are most of what a linear-attention block holds on to (34 GB of states alone for gated_deltanet_1B at
    65,536 tokens), while the projections, norms and the MLP around it are kept as without checkpointing."""
    global _recompute_mixers
    _recompute_mixers = bool(flag)


def _recomputable(fn):
    import functools

    @functools.wraps(fn)
    def wrapper(*args, **kw):
        if (_recompute_mixers and torch.is_grad_enabled()
                and any(isinstance(a, torch.Tensor) and a.requires_grad for a in args)):
            from torch.utils.checkpoint import checkpoint
            return checkpoint(lambda *t: fn(*t, **kw), *args, use_reentrant=False, preserve_rng_state=False)
        return fn(*args, **kw)
    return wrapper


# --------------------------------------------------------------------------------------------------------
# chunk-aligned layout
# --------------------------------------------------------------------------------------------------------
class ChunkLayout:
    """Where each packed token lives once every document is padded to a multiple of the chunk size."""

    def __init__(self, meta: VarlenMeta, chunk: int = CHUNK) -> None:
        import numpy as np
        lens = np.asarray([n for n in meta.lengths_list() if n > 0], dtype=np.int64)
        dev = meta.device
        self.chunk = chunk
        nchunks = (lens + chunk - 1) // chunk
        self.NC = int(nchunks.sum())
        self.T = int(lens.sum())
        self.Tp = self.NC * chunk
        self.aligned = bool((lens % chunk == 0).all())
        self.n_docs = int(lens.shape[0])
        # built with array operations on the host (a per-token Python loop would sit on the critical path of every step
        # of the linear-attention families): a token's padded row is its packed index plus the padding in front of its
        # document
        first = np.concatenate([[0], np.cumsum(nchunks)[:-1]])
        starts = np.concatenate([[0], np.cumsum(lens)[:-1]])
        rows = np.arange(self.T, dtype=np.int64) + np.repeat(first * chunk - starts, lens)
        last = first + nchunks - 1
        inv = np.full(self.Tp, -1, dtype=np.int32)
        inv[rows] = np.arange(self.T, dtype=np.int32)
        self._first_np, self._nchunks_np = first, nchunks
        self.rows = torch.from_numpy(rows).to(dev)                            # packed token -> padded row
        self.first = torch.from_numpy(first).to(dev)                          # first chunk of every document
        self.last = torch.from_numpy(last).to(dev)                            # last chunk of every document
        self.first_i32, self.last_i32 = self.first.to(torch.int32), self.last.to(torch.int32)
        self.rows_i32 = self.rows.to(torch.int32)
        self.inv_i32 = torch.from_numpy(inv).to(dev)                          # padded row -> packed token, -1 = padding
        self._steps = None
        self.longest = int(nchunks.max()) if self.n_docs else 0               # chunks of the longest document

    def _build_steps(self) -> None:
        # chunks at in-document position s that have a successor, and the documents they belong to (only the
        # per-position fallback of the state recurrences walks these)
        import numpy as np
        dev = self.first.device
        docs_all = np.arange(self.n_docs)
        steps, docs = [], []
        for s_ in range(int(self._nchunks_np.max()) - 1 if self.n_docs else 0):
            sel = docs_all[self._nchunks_np > s_ + 1]
            steps.append(torch.from_numpy((self._first_np[sel] + s_).astype(np.int32)).to(dev))
            docs.append(torch.from_numpy(sel.astype(np.int32)).to(dev))
        self._steps, self._step_docs = steps, docs

    @property
    def steps(self):
        if self._steps is None:
            self._build_steps()
        return self._steps

    @property
    def step_docs(self):
        if self._steps is None:
            self._build_steps()
        return self._step_docs

    @staticmethod
    def of(meta: VarlenMeta, chunk: int = CHUNK) -> "ChunkLayout":
        key = ("chunk_layout", chunk)
        lay = meta.cache.get(key)
        if lay is None:
            lay = ChunkLayout(meta, chunk)
            meta.cache[key] = lay
        return lay

    def pack(self, x: torch.Tensor) -> torch.Tensor:
        """[T, ...] -> [NC, chunk, ...] (zero rows where a document is padded)."""
        if self.aligned and (x.is_contiguous() or not _rows_strided(x)):
            return x.reshape(self.NC, self.chunk, *x.shape[1:])
        return _Pack.apply(x, self, slots.of(x)).reshape(self.NC, self.chunk, *x.shape[1:])

    def unpack(self, y: torch.Tensor) -> torch.Tensor:
        """[NC, chunk, ...] -> [T, ...]."""
        y = y.reshape(self.Tp, *y.shape[2:])
        return y if self.aligned else _Unpack.apply(y, self)


def _row_distance(x: torch.Tensor) -> int:
    """Elements between the rows of ``x``; of one row its length, whatever stride torch keeps for it."""
    return x.stride(0) if x.shape[0] > 1 else x.numel()


def _rows_strided(x: torch.Tensor) -> bool:
    """Rows that are contiguous and whole 16-byte vectors, at any distance that is one too, or the same with 4-byte words (a
    few scalars per token): what the gather kernel reads."""
    n = x.numel() // max(x.shape[0], 1)
    inner = list(x.stride()[1:]) == [math.prod(x.shape[i + 1:]) for i in range(1, x.dim())]
    ld = _row_distance(x)
    unit = 16 if n * x.element_size() % 16 == 0 else 4
    return inner and n * x.element_size() % unit == 0 and ld * x.element_size() % unit == 0 and x.data_ptr() % unit == 0 and ld >= n


def _gather_rows(x: torch.Tensor, idx: torch.Tensor, n_out: int, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``out[r] = x[idx[r]]`` (zero where ``idx[r] < 0``) in one pass of the row-gather kernel."""
    x = x if _rows_strided(x) else x.contiguous()
    row_bytes = (x.numel() // max(x.shape[0], 1)) * x.element_size()
    unit = 16 if row_bytes % 16 == 0 else 4
    if not (_lib.available() and x.is_cuda and row_bytes % unit == 0 and x.shape[0] > 0 and x.data_ptr() % unit == 0):
        safe = idx.clamp_min(0).long()
        r = x.index_select(0, safe)
        r = r * (idx >= 0).to(x.dtype).view(-1, *([1] * (x.dim() - 1)))
        return r if out is None else out.copy_(r)
    if out is None:
        out = torch.empty(n_out, *x.shape[1:], dtype=x.dtype, device=x.device)
    rc = _lib.lib().fb_gather_rows(x.data_ptr(), out.data_ptr(), idx.data_ptr(), n_out, row_bytes,
                                   _row_distance(x) * x.element_size(), _row_distance(out) * out.element_size(), _lib.stream_ptr())
    _lib.check(rc, "fb_gather_rows")
    _lib.count_launch()
    return out


class _Pack(torch.autograd.Function):
    """Packed rows into the padded layout (zero rows where a document is padded): a gather through the inverse row map;
    the map is injective, so the backward is a plain gather too.  ``slot``: where the gradient of ``x`` belongs (``ops/slots.py``)."""

    @staticmethod
    def forward(ctx, x, lay, slot):
        ctx.lay, ctx.slot = lay, slot
        return _gather_rows(x, lay.inv_i32, lay.Tp)

    @staticmethod
    def backward(ctx, dy):
        lay = ctx.lay
        out = None
        if ctx.slot is not None and dy.numel():
            out = ctx.slot.take(lay.T, dy.numel() // dy.shape[0], dy.dtype, dy.device)
            out = out.view(lay.T, *dy.shape[1:])
            if not _rows_strided(out):
                out = None
        return _gather_rows(dy, lay.rows_i32, lay.T, out), None, None


class _Unpack(torch.autograd.Function):
    @staticmethod
    def forward(ctx, y, lay):
        ctx.lay = lay
        return _gather_rows(y, lay.rows_i32, lay.T)

    @staticmethod
    def backward(ctx, dx):
        return _gather_rows(dx, ctx.lay.inv_i32, ctx.lay.Tp), None


def _hm(x: torch.Tensor) -> torch.Tensor:
    """[NC, 64, H, d] -> the [NC, H, 64, d] operand view."""
    return x.permute(0, 2, 1, 3)


# --------------------------------------------------------------------------------------------------------
# differentiable pieces
# --------------------------------------------------------------------------------------------------------
class _Scores(torch.autograd.Function):
    """``C = mask(alpha * A B^T * exp(d_i - d_j))`` for 64 x 64 score blocks; ``d`` is the within-chunk cumulative log decay."""

    @staticmethod
    def forward(ctx, a, b, d, alpha, mask, out_dtype):
        # a, b: [NC, H, C, dk] views; d: [NC, H, C] fp32
        out = bgemm(a, b, alpha=alpha, mask=mask, decay=d, out_dtype=out_dtype)
        ctx.save_for_backward(a, b, d, out)
        ctx.cfg = (alpha, mask)
        return out

    @staticmethod
    def backward(ctx, dc):
        a, b, d, out = ctx.saved_tensors
        alpha, mask = ctx.cfg
        C = out.shape[-1]
        if _lib.available() and out.is_cuda and out.dtype in (torch.float32, torch.bfloat16) and C % 32 == 0 and C <= 128 \
                and d.dtype == torch.float32:
            from . import chunk_kernels
            g, dd = chunk_kernels.scores_bwd_prep(dc, out, d, mask)       # one pass instead of eight elementwise ones
        else:
            dcf = dc.float()
            dd = None
            if ctx.needs_input_grad[2]:
                e = dcf * out.float()
                dd = e.sum(-1) - e.sum(-2)
            m = _mask(out.shape[-2], out.shape[-1], mask, dc.device)
            w = (d[..., :, None] - d[..., None, :]).masked_fill(~m, float("-inf")).exp()
            g = dcf * w
        g = g.to(a.dtype)
        da = db = None
        if ctx.needs_input_grad[0]:
            da = _like(a)
            bgemm(g, b, b_mn=True, out=da, alpha=alpha)
        if ctx.needs_input_grad[1]:
            db = _like(b)
            bgemm(g, a, a_mn=True, b_mn=True, out=db, alpha=alpha)
        return da, db, dd, None, None, None


def _like(t: torch.Tensor) -> torch.Tensor:
    from .bgemm import _empty_like_layout
    return _empty_like_layout(t)


class _DecayStates(torch.autograd.Function):
    """States at the start of every chunk for ``S_{c+1} = alpha_c S_c + khat_c^T u_c`` (S = 0 at the first chunk of a
    document); ``alpha`` is ``[NC, H]`` or ``[NC, H, dk]`` (one decay per key channel).  The increments and the running state
    are fp32, the states handed out bf16."""

    @staticmethod
    def forward(ctx, alpha, khat, u, lay: ChunkLayout):
        # alpha fp32; khat [NC, H, C, dk]; u [NC, H, C, dv] (operand views)
        alpha = alpha.contiguous()
        S = _decay_states(lay, alpha, khat, u, reverse=False)
        ctx.save_for_backward(alpha, khat, u, S)
        ctx.lay = lay
        return S

    @staticmethod
    def backward(ctx, dS):
        alpha, khat, u, S = ctx.saved_tensors
        lay = ctx.lay
        NC, H, _, dk = khat.shape
        # adjoint of the state entering the NEXT chunk; zero where the next chunk belongs to another document
        Ln = _state_scan(lay, alpha, _lib.dense(dS.to(khat.dtype)), khat.dtype, reverse=True)
        dalpha = dkhat = du = None
        if ctx.needs_input_grad[0]:
            dalpha = _pair_dot(Ln, S, per_row=alpha.dim() == 3)
        if ctx.needs_input_grad[2]:
            du = _like(u)
            bgemm(khat, Ln, b_mn=True, out=du)
        if ctx.needs_input_grad[1]:
            dkhat = bgemm(u, Ln, out=_token_major(NC, H, lay.chunk, dk, khat.dtype, khat.device))
        return dalpha, dkhat, du, None


def _state_scan(lay: ChunkLayout, alpha, x, dtype, reverse: bool) -> torch.Tensor:
    """``s = 0; for every chunk of a document (backwards when ``reverse``): out_c = s; s = alpha_c s + x_c``."""
    if _lib.available() and x.is_cuda:
        from . import chunk_kernels
        return chunk_kernels.state_scan(lay.first, lay.last, alpha, x, reverse)
    al = alpha[..., None] if alpha.dim() == 3 else alpha[..., None, None]
    out = torch.zeros(x.shape, dtype=torch.float32, device=x.device)
    for idx in (lay.steps[::-1] if reverse else lay.steps):
        i = idx.long()
        src, dst = (i + 1, i) if reverse else (i, i + 1)
        out[dst] = al[src] * out[src] + x[src].float()
    return out.to(dtype)


_lib.register("fb_decay_scan", ([c_void_p] + [c_longlong] * 3 + [c_int]) * 2 + [c_void_p, c_int] + [c_void_p] * 5 + [c_int] * 6 + [c_void_p])


# Where the one kernel pays, without and with the decay's gradient, in microseconds: it takes a time per chunk of the longest document, however
# many documents and heads there are beside it (until memory bounds it, far below the other form); product and scan have all chunks'
# products side by side and take a time per state element, and some microseconds more of launches.  Measured at 161 combinations of 1,024 to
# 65,536 tokens in 1 to 32 documents and 2 x 64 x 64 (heads x rows x columns), 4 x 64 x 256, 4 x 64 x 512, 4 x 128 x 256, 16 x 128 x 512,
# 32 x 128 x 64 and 64 x 128 x 64 states: the rule's choice is the faster one or within 1 % of it forward, and the faster one or within 7 us
# with the gradient (the worst: 24 for 18 at 1,024 tokens of 32 x 128 x 64).  4 x 128 x 256 at 65,536
# tokens, one kernel and the other form: 8 documents 103 and 276 us, with the gradient 142 and 263; 2 documents 295 and 302, 489 and 322.
# 2 x 64 x 64 at 16,384 tokens: 16 documents 13 and 14, 22 and 21; 4 documents 36 and 22, 63 and 28.
# The two differ by roundings: going backwards the other form rounds the increments to bf16, this one keeps them in fp32.
WALK_US = (0.55, 8.0, 2.1e-6), (1.05, 14.0, 1.9e-6)   # per chunk; launches, per state element


def _rows_of_vectors(t: torch.Tensor) -> torch.Tensor:
    """``t`` (four dimensions, bf16), as it lies if the kernels' tile copies can read it there: rows of consecutive elements on 16-byte
    boundaries."""
    s = t.stride()
    ok = s[3] == 1 and min(s) > 0 and not (s[0] | s[1] | s[2]) & 7 and not t.data_ptr() & 15
    return t if ok else _lib.dense(t)


def _walk_pays(lay: ChunkLayout, elements: int, gradient: bool) -> bool:
    chunk, launches, element = WALK_US[gradient]
    return lay.longest * chunk < launches + lay.NC * elements * element


def _decay_states(lay: ChunkLayout, alpha, a, b, reverse: bool, with_state=None):
    """``_state_scan`` over the increments ``x_c = a_c^T b_c`` of operands ``[NC, heads, chunk, rows]`` and ``[NC, heads, chunk, cols]`` (heads of
    either may serve several of alpha's), in the operands' type.  ``with_state`` (contiguous, as the result): returns the pair of the result
    and alpha's gradient, the sums of their products over the columns, and over the rows if alpha has none.  For the state sizes of the
    configurations one kernel does it all (``csrc/decay_scan.cu``), others take a product, a scan and the sums."""
    rows, cols, H = a.shape[3], b.shape[3], alpha.shape[1]
    per_row = alpha.dim() == 3
    if (lay.chunk == 64 and rows in (64, 128) and cols % 64 == 0 and cols > 0 and a.is_cuda and a.dtype == b.dtype == torch.bfloat16 and _lib.available()
            and alpha.dtype == torch.float32 and alpha.is_contiguous() and max(lay.n_docs, H) <= 65535 and lay.NC * H * rows < 1 << 31
            and _walk_pays(lay, H * rows * cols, with_state is not None)):
        a, b = _rows_of_vectors(a), _rows_of_vectors(b)
        out = torch.empty(lay.NC, H, rows, cols, dtype=a.dtype, device=a.device)
        part = None
        if with_state is not None:
            with_state = _lib.dense(with_state)   # saved-tensor hooks hand back copies, which lie wherever they were put
            slices = cols // 64
            part = torch.empty((slices, lay.NC, H, rows) if per_row else (slices * (rows // 32), lay.NC, H), dtype=torch.float32, device=a.device)
        args = [x for t in (a, b) for x in (t.data_ptr(), t.stride(2), t.stride(1), t.stride(0), t.shape[1])]
        rc = _lib.lib().fb_decay_scan(*args, alpha.data_ptr(), int(per_row), out.data_ptr(), _lib.ptr(with_state), _lib.ptr(part),
                                      lay.first_i32.data_ptr(), lay.last_i32.data_ptr(), lay.n_docs, H, lay.NC, rows, cols, int(reverse),
                                      _lib.stream_ptr())
        _lib.check(rc, "fb_decay_scan")
        _lib.count_launch()
        if with_state is None:
            return out
        return out, part.sum(0)
    x = bgemm(a, b, a_mn=True, b_mn=True, out_dtype=None if reverse else torch.float32)
    out = _state_scan(lay, alpha, x, a.dtype, reverse)
    return out if with_state is None else (out, _pair_dot(out, with_state, per_row=per_row))


def _delta_states(M, B, alpha, lay: ChunkLayout) -> torch.Tensor:
    """``[NC, H, dk, dv]``: the state entering every chunk of ``S_{c+1} = alpha_c S_c - M_c S_c + B_c``."""
    NC, H, dk, dv = B.shape
    if _scan_kernel_ok(M, B, alpha, dk, dv):
        return _delta_scan(M, B, alpha, lay, reverse=False)   # one persistent launch walks every document
    # shapes the scan kernel does not cover: one batched GEMM per chunk position; the running state lives in ONE fp32
    # buffer per document, updated in place by the epilogue
    S = torch.empty(NC + 1, H, dk, dv, dtype=B.dtype, device=B.device)
    S.index_fill_(0, lay.first, 0.0)
    state = torch.zeros(lay.n_docs, H, dk, dv, dtype=torch.float32, device=B.device)
    for idx, docs in zip(lay.steps, lay.step_docs):
        bgemm(M, S, b_mn=True, a_index=idx, b_index=idx, out=state, c_index=docs, cin=state, cin_index=docs, gamma=alpha,
              alpha=-1.0, add16=B, add16_index=idx, out16=S, out16_index=idx, out16_offset=1, n_hi=len(idx))
    return S[:NC]


def _delta_adjoint(M, dS, alpha, lay: ChunkLayout) -> torch.Tensor:
    """``[NC, H, dk, dv]``: the adjoint of the state LEAVING every chunk (zero at a document's last) for the state gradients
    ``dS`` of the recurrence above."""
    NC, H, dk, dv = dS.shape
    if _scan_kernel_ok(M, dS, alpha, dk, dv):
        return _delta_scan(M, dS, alpha, lay, reverse=True)
    L = torch.empty(NC + 1, H, dk, dv, dtype=dS.dtype, device=dS.device)
    L[:NC] = dS
    L[NC] = 0
    lam = dS.index_select(0, lay.last).float()
    for idx, docs in zip(lay.steps[::-1], lay.step_docs[::-1]):
        bgemm(M, L, a_mn=True, b_mn=True, a_index=idx, b_index=idx, b_offset=1, out=lam, c_index=docs, cin=lam, cin_index=docs,
              gamma=alpha, alpha=-1.0, add16=dS, add16_index=idx, out16=L, out16_index=idx, n_hi=len(idx))
    L.index_fill_(0, lay.first, 0.0)
    return L[1:]


# the C x C stages of the delta rule: kernels of csrc/chunk.cu, or their definitions
def _delta_inverse(P, beta, b):
    if _lib.available() and P.is_cuda:
        from . import chunk_kernels
        return chunk_kernels.delta_inverse(P, beta, b, bgemm)
    C = P.shape[-1]
    br = beta.permute(0, 2, 1)
    eye = torch.eye(C, dtype=torch.float32, device=P.device)
    T = torch.linalg.solve_triangular(eye + br[..., None] * P.float(), eye.expand_as(P).contiguous(), upper=False, unitriangular=True)
    return T, T * br[..., None, :], None if b is None else T * (br * b.permute(0, 2, 1).exp())[..., None, :]


def _delta_bwd_t(T, dTu, dTw, beta, b, scale):
    if _lib.available() and T.is_cuda:
        from . import chunk_kernels
        return chunk_kernels.delta_bwd_t(T, dTu, dTw, beta, b, scale)
    br = beta.permute(0, 2, 1)[..., None, :]
    w = 0 if b is None else dTw * b.permute(0, 2, 1).exp()[..., None, :]
    dbeta = scale * (T * (dTu + w)).sum(-2).permute(0, 2, 1)
    db = None if b is None else scale * (br * T * w).sum(-2).permute(0, 2, 1)
    return br * (dTu + w), dbeta, db


def _delta_bwd_scores(dA, P, dQ, Q, beta, b, scale, dbeta, db):
    if _lib.available() and P.is_cuda:
        from . import chunk_kernels
        return chunk_kernels.delta_bwd_scores(dA, P, dQ, Q, beta, b, scale, dbeta, db)
    C = P.shape[-1]
    br = beta.permute(0, 2, 1)[..., None]
    dA = dA.masked_fill(~_mask(C, C, MASK_STRICT, P.device), 0.0)
    dbeta += scale * (dA * P).sum(-1).permute(0, 2, 1)
    if b is None:
        return dA * br, None
    d = b.permute(0, 2, 1)
    w = (d[..., :, None] - d[..., None, :]).masked_fill(~_mask(C, C, MASK_TRIL, P.device), float("-inf")).exp()
    if dQ is None:
        return br * dA * w, None
    e = br * dA * P + dQ * Q
    db += scale * (e.sum(-1) - e.sum(-2)).permute(0, 2, 1)
    return br * dA * w, dQ * w


class _GatedDelta(torch.autograd.Function):
    """The whole chunk pipeline of the (gated) delta rule on packed chunks: q, k ``[NC, C, H, dk]``, v ``[NC, C, H, dv]``, beta
    and the log decay g ``[NC, C, H]`` fp32 (g may be None).  One node instead of one per product: the terms of an output or of
    a gradient accumulate in one GEMM, nothing is added up by passes of its own, and without a decay the operands that a
    decay would rescale are the inputs themselves.  ``scale`` is a factor of the output; the backward runs without it and
    puts it into the last products."""

    @staticmethod
    def forward(ctx, q, k, v, beta, g, scale, lay):
        q, k, v, beta = (_lib.dense(t) for t in (q, k, v, beta))
        NC, C, H, dk = q.shape
        dv = v.shape[-1]
        if g is not None:
            b, khat, qbar, alpha = _scalar_prep_raw(q, k, _lib.dense(g))
            d = b.permute(0, 2, 1)
        else:
            b = d = None
            khat, qbar = k, q
            alpha = torch.ones(NC, H, dtype=torch.float32, device=q.device)
        qh, kh, vh, khh, qbh = (_hm(t) for t in (q, k, v, khat, qbar))
        P = bgemm(kh, kh, mask=MASK_STRICT, decay=d, out_dtype=torch.float32)             # [NC, H, C, C]
        Q = bgemm(qh, kh, mask=MASK_TRIL, decay=d)
        T, Tu, Tw = _delta_inverse(P, beta, b)
        T, Tu = T.to(q.dtype), Tu.to(q.dtype)
        Tw = Tu if Tw is None else Tw.to(q.dtype)
        u = bgemm(Tu, vh, b_mn=True, out=_token_major(NC, H, C, dv, q.dtype, q.device))
        w = bgemm(Tw, kh, b_mn=True, out=_token_major(NC, H, C, dk, q.dtype, q.device))
        M = bgemm(khh, w, a_mn=True, b_mn=True)                                           # [NC, H, dk, dk] chunk transition
        S = _delta_states(M, bgemm(khh, u, a_mn=True, b_mn=True), alpha, lay)             # [NC, H, dk, dv]
        # u - w S; u again as a product in the same accumulator: added from its bf16 copy it would be rounded twice
        vn = bgemm(Tu, vh, b_mn=True, more=[(w, S, False, True, -1)], out=_token_major(NC, H, C, dv, q.dtype, q.device))
        o = bgemm(qbh, S, b_mn=True, alpha=scale, more=[(Q, vn, False, True, 1)],
                  out=_token_major(NC, H, C, dv, q.dtype, q.device))
        ctx.save_for_backward(q, k, v, beta, b, khat if b is not None else None, qbar if b is not None else None, alpha, P, Q, T, Tu,
                              Tw if b is not None else None, w, M, S, vn)
        ctx.cfg = (scale, lay)
        return o.permute(0, 2, 1, 3)

    @staticmethod
    def backward(ctx, do):
        q, k, v, beta, b, khat, qbar, alpha, P, Q, T, Tu, Tw, w, M, S, vn = ctx.saved_tensors
        scale, lay = ctx.cfg
        NC, C, H, dk = q.shape
        dt, dev = q.dtype, q.device
        dv = v.shape[-1]
        gated = b is not None
        need_q, need_k, need_v, need_beta, need_g = ctx.needs_input_grad[:5]
        need_g = need_g and gated
        inner = need_k or need_beta or need_g              # what goes through the inverse and the chunk transitions
        doh = _hm(_lib.dense(do.to(dt)))
        qh, kh, vh = _hm(q), _hm(k), _hm(v)
        khh, qbh = (_hm(khat), _hm(qbar)) if gated else (kh, qh)
        Tw = Tw if gated else Tu
        tok = lambda n: _token_major(NC, H, C, n, dt, dev)                                # noqa: E731
        back = lambda t: None if t is None else t.permute(0, 2, 1, 3)                     # noqa: E731
        dq = dkk = dvv = dbeta = db = dg = gk = None
        # dQ (without a decay also the operand of its products)
        gq = bgemm(doh, vn, mask=MASK_TRIL) if need_q or need_k or need_g else None
        if inner or need_v:
            dvn = bgemm(Q, doh, a_mn=True, b_mn=True, out=tok(dv))
            Ln = _delta_adjoint(M, bgemm(qbh, doh, a_mn=True, b_mn=True, more=[(w, dvn, True, True, -1)]), alpha, lay)
            # dvn again as a product in the same accumulator: added from its bf16 copy it would be rounded twice
            du = bgemm(khh, Ln, b_mn=True, more=[(Q, doh, True, True, 1)], out=tok(dv))
            if need_v:
                dvv = bgemm(Tu, du, a_mn=True, b_mn=True, alpha=scale, out=tok(dv))
        if inner:
            # S leaves a chunk as alpha S + khat^T vn, vn = u - w S: what reaches vn reaches u and, times -S^T, w
            dw = bgemm(du, S, alpha=-1.0, out=tok(dk))
            if gated:
                dTu, dTw = bgemm(du, vh), bgemm(dw, kh)
            else:
                dTu, dTw = bgemm(du, vh, more=[(dw, kh, False, False, 1)]), None
            dT, dbeta, db = _delta_bwd_t(T, dTu, dTw, beta, b, scale)
            # T = (I + A)^-1: dA = -T^T dT T^T on the strict lower triangle
            dA = bgemm(bgemm(T, dT, a_mn=True, b_mn=True), T, alpha=-1.0, mask=MASK_STRICT, out_dtype=torch.float32)
            gk, gq2 = _delta_bwd_scores(dA, P, gq, Q, beta, b, scale, dbeta, db)
            gk = gk.to(dt)
            keys = [(gk, kh, False, True, 1), (gk, kh, True, True, 1)]
        elif gated and gq is not None:
            gq2 = _scores_bwd(gq, Q, b, None, 1.0)
        if gated and gq is not None:
            gq = gq2.to(dt)
            dqbar = bgemm(doh, S, out=tok(dk)) if need_q or need_g else None
            dkhat = bgemm(vn, Ln, alpha=scale, out=tok(dk)) if need_k or need_g else None
            dalpha = _pair_dot(Ln, S, per_row=False) * scale if need_g else None
            dq0, dk0, dg = _scalar_prep_raw_bwd(q, k, b, back(dkhat), back(dqbar), dalpha, db, scale)
            if need_q:
                dq = bgemm(gq, kh, b_mn=True, alpha=scale, add16=_hm(dq0), out=tok(dk))
            if need_k:
                dkk = bgemm(Tw, dw, a_mn=True, b_mn=True, alpha=scale, more=keys + [(gq, qh, True, True, 1)], add16=_hm(dk0), out=tok(dk))
        elif not gated:
            if need_q:
                dq = bgemm(doh, S, alpha=scale, more=[(gq, kh, False, True, 1)], out=tok(dk))
            if need_k:
                dkk = bgemm(Tu, dw, a_mn=True, b_mn=True, alpha=scale, out=tok(dk),
                            more=keys + [(gq, qh, True, True, 1), (vn, Ln, False, False, 1)])
        return back(dq), back(dkk), back(dvv), dbeta if need_beta else None, dg if need_g else None, None, None


class _GroupedScalarGla(torch.autograd.Function):
    """The chunk pipeline of scalar-gated attention whose queries and keys ``[NC, C, G, dk]`` serve groups of H / G heads
    (Mamba2's C and B), v ``[NC, C, H, dv]``, g ``[NC, C, H]`` fp32.  They are never expanded: the decay moves to the value side
    of the state update (``S += k^T (v e^{b_last - b})``) and to the rows of the output, and the gradients of q and k add the
    heads of a group up in the accumulator of one product."""

    @staticmethod
    def forward(ctx, q, k, v, g, scale, lay):
        ctx.slots = slots.of(q), slots.of(k)
        q, k = (_rows_of_vectors(t) if t.dtype == torch.bfloat16 else _lib.dense(t) for t in (q, k))  # (column blocks, as a rule)
        v, g = _lib.dense(v), _lib.dense(g)
        NC, C, H, dv = v.shape
        b, eb, alpha, vhat = _group_prep(v, g, scale)
        d = b.permute(0, 2, 1)
        qh, kh = _hm(q), _hm(k)
        Q = bgemm(qh, kh, alpha=scale, mask=MASK_TRIL, decay=d, n_lo=H)                   # [NC, H, C, C] from the shared q / k
        S = _decay_states(lay, alpha, kh, _hm(vhat), reverse=False)
        o1 = bgemm(qh, S, b_mn=True, rowscale=eb.permute(0, 2, 1), out=_token_major(NC, H, C, dv, q.dtype, q.device))
        o = bgemm(Q, _hm(v), b_mn=True, add16=o1, out=_token_major(NC, H, C, dv, q.dtype, q.device))
        ctx.save_for_backward(q, k, v, b, eb, alpha, vhat, Q, S, o1.permute(0, 2, 1, 3))
        ctx.lay, ctx.scale = lay, scale
        return o.permute(0, 2, 1, 3)

    @staticmethod
    def backward(ctx, do):
        q, k, v, b, eb, alpha, vhat, Q, S, o1 = ctx.saved_tensors
        lay = ctx.lay
        NC, C, H, dv = v.shape
        G, dk = q.shape[2:]
        dt, dev = q.dtype, q.device
        tok = lambda h, n: _token_major(NC, h, C, n, dt, dev)                             # noqa: E731

        def block(i):  # where the gradient of q or k belongs
            if ctx.slots[i] is None:
                return tok(G, dk)
            m = ctx.slots[i].take(NC * C, G * dk, dt, dev)
            if (m.data_ptr() // m.element_size() | m.stride(0) | dk) & 7:  # the product writes vectors of eight
                return tok(G, dk)
            return m.view(NC, C, G, dk).permute(0, 2, 1, 3)

        do = _lib.dense(do.to(dt))
        need_q, need_k, need_v, need_g = ctx.needs_input_grad[:4]
        dos, db = _group_bwd1(do, o1, eb)
        doh, dosh, qh, kh, vhh = _hm(do), _hm(dos), _hm(q), _hm(k), _hm(vhat)
        back = lambda t: None if t is None else t.permute(0, 2, 1, 3)                     # noqa: E731
        dq = dkk = dvv = dg = dv1 = dalpha = None
        r = H // G
        if need_q or need_k or need_g:
            # Q has the factor ``scale`` (so the gradient of b has it), its operand's gradient gets it before it is rounded
            gq = _scores_bwd(bgemm(doh, _hm(v), mask=MASK_TRIL), Q, b, db, ctx.scale).to(dt)
        if need_k or need_v or need_g:
            Ln, dalpha = _decay_states(lay, alpha, qh, dosh, True, S) if need_g else (_decay_states(lay, alpha, qh, dosh, True), None)
        if need_v or need_g:
            dvhat = bgemm(kh, Ln, b_mn=True, out=tok(H, dv))
            if need_v:
                dv1 = bgemm(Q, doh, a_mn=True, b_mn=True, out=tok(H, dv))
            dvv, dg = _group_bwd2(back(dvhat), vhat, back(dv1), b, db, alpha, dalpha)
        if need_q:
            dq = bgemm(dosh, S, more=[(gq, kh, False, True, 1)], sum_lo=r, out=block(0))
        if need_k:
            dkk = bgemm(vhh, Ln, more=[(gq, qh, True, True, 1)], sum_lo=r, out=block(1))
        return back(dq), back(dkk), dvv, dg, None, None


def _group_kernels(v) -> bool:
    if not (_lib.available() and v.is_cuda):
        return False
    from . import chunk_kernels
    return chunk_kernels.group_supported(v.shape[1], v.shape[-1])


def _group_prep(v, g, scale):
    if _group_kernels(v):
        from . import chunk_kernels
        return chunk_kernels.group_prep(v, g, scale)
    b = g.cumsum(1)
    last = b[:, -1:]
    return b, scale * b.exp(), last[:, 0].exp().contiguous(), (v.float() * (last - b).exp()[..., None]).to(v.dtype)


def _group_bwd1(do, o1, eb):
    if _group_kernels(do):
        from . import chunk_kernels
        return chunk_kernels.group_bwd1(do, o1, eb)
    return (do.float() * eb[..., None]).to(do.dtype), (do.float() * o1.float()).sum(-1)


def _group_bwd2(dvhat, vhat, dv1, b, db, alpha, dalpha):
    if _group_kernels(vhat):
        from . import chunk_kernels
        return chunk_kernels.group_bwd2(dvhat, vhat, dv1, b, db, alpha, dalpha)
    dv = dg = None
    if dv1 is not None:
        dv = (dv1.float() + dvhat.float() * (b[:, -1:] - b).exp()[..., None]).to(dv1.dtype)
    if dalpha is not None:
        s = (dvhat.float() * vhat.float()).sum(-1)
        db = db - s
        db[:, -1] += s.sum(1) + alpha * dalpha
        dg = db.flip(1).cumsum(1).flip(1)
    return dv, dg


def _scores_bwd(dQ, Q, b, db, scale):
    if _lib.available() and Q.is_cuda:
        from . import chunk_kernels
        return chunk_kernels.scores_bwd(dQ, Q, b, db, scale)
    C = Q.shape[-1]
    d = b.permute(0, 2, 1)
    w = (d[..., :, None] - d[..., None, :]).masked_fill(~_mask(C, C, MASK_TRIL, Q.device), float("-inf")).exp()
    if db is not None:
        e = dQ.float() * Q.float()
        db += (e.sum(-1) - e.sum(-2)).permute(0, 2, 1)
    return dQ * w * scale


def _scalar_prep_raw(q, k, g):
    """``b = cumsum(g)``, ``khat = k e^{b_last - b}``, ``qbar = q e^b``, ``alpha = e^{b_last}`` without autograd."""
    if _lib.available() and q.is_cuda:
        from . import chunk_kernels
        if chunk_kernels.scalar_prep_supported(q.shape[1], q.shape[-1]):
            return chunk_kernels.scalar_prep(q, k, g, 1.0)
    b = g.cumsum(1)
    return (b, k * (b[:, -1:] - b).exp().to(k.dtype)[..., None], q * b.exp().to(q.dtype)[..., None], b[:, -1].exp().contiguous())


def _scalar_prep_raw_bwd(q, k, b, dkhat, dqbar, dalpha, db, scale):
    """Gradients of ``_scalar_prep_raw``; ``scale`` multiplies ``dqbar`` (the other incoming gradients have it already).  An
    incoming gradient may be None (zero)."""
    if _lib.available() and q.is_cuda:
        from . import chunk_kernels
        if chunk_kernels.scalar_prep_supported(q.shape[1], q.shape[-1]):
            return chunk_kernels.scalar_prep_bwd(q, k, b, dkhat, dqbar, dalpha, db, scale)
    last = b[:, -1:]
    dq = torch.zeros_like(q, dtype=torch.float32) if dqbar is None else dqbar.float() * (b.exp() * scale)[..., None]
    dk = torch.zeros_like(k, dtype=torch.float32) if dkhat is None else dkhat.float() * (last - b).exp()[..., None]
    kd = (k.float() * dk).sum(-1)
    db = (0 if db is None else db) + (q.float() * dq).sum(-1) - kd
    db[:, -1] += kd.sum(1) + (0 if dalpha is None else dalpha * b[:, -1].exp())
    return dq.to(q.dtype), dk.to(k.dtype), db.flip(1).cumsum(1).flip(1)


def _scan_kernel_ok(M: torch.Tensor, add: torch.Tensor, alpha: torch.Tensor, dk: int, dv: int) -> bool:
    import os
    return (_lib.available() and M.is_cuda and M.dtype == torch.bfloat16 and add.dtype == torch.bfloat16
            and M.is_contiguous() and add.is_contiguous() and alpha.dim() == 2 and alpha.dtype == torch.float32
            and dk in (128, 256) and dv % 128 == 0 and os.environ.get("FLAME_B200_DELTA_SCAN", "1") != "0")


def _delta_scan(M: torch.Tensor, add: torch.Tensor, alpha: torch.Tensor, lay: "ChunkLayout", reverse: bool) -> torch.Tensor:
    """The chunk-state recurrence of every (document, head) in one persistent kernel (``csrc/delta_scan.cu``)."""
    NC, H, dk, _ = M.shape
    dv = add.shape[-1]
    out = torch.empty_like(add)
    rc = _lib.lib().fb_delta_scan(M.data_ptr(), add.data_ptr(), alpha.data_ptr(), out.data_ptr(), lay.first_i32.data_ptr(),
                                  lay.last_i32.data_ptr(), lay.n_docs, H, NC, dk, dv, int(reverse), _lib.stream_ptr())
    _lib.check(rc, "fb_delta_scan")
    _lib.count_launch()
    return out


def _pair_dot(x: torch.Tensor, y: torch.Tensor, per_row: bool) -> torch.Tensor:
    """``sum(x * y)`` over the last two (or the last) dimensions in fp32 without materialising fp32 copies."""
    if _lib.available() and x.is_cuda:
        from . import chunk_kernels
        return chunk_kernels.pair_dot(x, y, per_row)
    return (x.float() * y.float()).sum(-1 if per_row else (-1, -2))


def _token_major(NC, H, R, D, dtype, dev):
    return torch.empty(NC, R, H, D, dtype=dtype, device=dev).permute(0, 2, 1, 3)


# --------------------------------------------------------------------------------------------------------
# algorithms
# --------------------------------------------------------------------------------------------------------
def _scalar_prep(qp, kp, gp, scale, dt):
    """``b = cumsum(g)`` [NC, C, H], ``khat = k e^{b_last - b}``, ``qbar = scale q e^{b}``, ``alpha = e^{b_last}`` [NC, H]."""
    NC, C, H, dk = qp.shape
    if _lib.available() and qp.is_cuda:
        from . import chunk_kernels
        if chunk_kernels.scalar_prep_supported(C, dk):
            return chunk_kernels.ScalarPrep.apply(qp, kp, gp, scale)
    b = gp.cumsum(1)
    b_last = b[:, -1]
    khat = kp * (b_last[:, None] - b).exp().to(dt)[..., None]
    qbar = qp * (b.exp() * scale).to(dt)[..., None]
    return b, khat, qbar, b_last.exp()


def scalar_chunk(dk: int, dv: int) -> int:
    """Chunk length of the scalar-gated algorithms.  With a large state (dk * dv) 128 halves the number of sequential
    state steps and of stored chunk states and fills the 128-row MMA tile; with a small state the 64 x 64 score blocks
    are the cheaper side.  Every decay exponent stays <= 0 at any chunk length."""
    return 128 if dk * dv >= 32768 else 64


@_recomputable
def gated_delta_rule_tc(q, k, v, beta, g, meta: VarlenMeta, scale: Optional[float] = None,
                        chunk: Optional[int] = None) -> torch.Tensor:
    """Chunked (gated) delta rule; q, k ``[T, H, dk]`` (already normalised), v ``[T, H, dv]``, beta ``[T, H]``,
    g ``[T, H]`` log decay or None.  Same result as ``linear_attn.gated_delta_rule_recurrent``."""
    T, H, dk = q.shape
    dv = v.shape[-1]
    scale = dk ** -0.5 if scale is None else scale
    lay = ChunkLayout.of(meta, chunk or scalar_chunk(dk, dv))
    dt = torch.bfloat16 if q.is_cuda else q.dtype
    qp, kp, vp = lay.pack(q).to(dt), lay.pack(k).to(dt), lay.pack(v).to(dt)   # [NC, C, H, d]
    o = _GatedDelta.apply(qp, kp, vp, lay.pack(beta.float()), None if g is None else lay.pack(g.float()), scale, lay)
    return lay.unpack(o).to(v.dtype)


@_recomputable
def gated_delta_rule_chunks(qp, kp, vp, beta, g, lay: "ChunkLayout", scale: float) -> torch.Tensor:
    """The same on operands in the rows of ``lay``: q, k, v ``[Tp, H, d]`` bf16 (zero in the padding), beta and g ``[NC, chunk, H]`` fp32; the
    result stays there, ``[NC, chunk, H, dv]``."""
    qp, kp, vp = (t.view(lay.NC, lay.chunk, *t.shape[1:]) for t in (qp, kp, vp))
    return _GatedDelta.apply(qp, kp, vp, beta, g, scale, lay)


@_recomputable
def scalar_gla_tc(q, k, v, g, meta: VarlenMeta, scale: float = 1.0, chunk: Optional[int] = None) -> torch.Tensor:
    """``S_t = exp(g_t) S_{t-1} + k_t v_t^T,  o_t = scale q_t^T S_t`` with one log decay per head and step
    (Mamba2's SSD in its attention form).  q, k ``[T, G, dk]`` with G dividing H, v ``[T, H, dv]``, g ``[T, H]``."""
    T, G, dk = q.shape
    H = v.shape[1]
    lay = ChunkLayout.of(meta, chunk or scalar_chunk(dk, v.shape[-1]))
    dt = torch.bfloat16 if q.is_cuda else q.dtype
    qp, kp, vp = lay.pack(q).to(dt), lay.pack(k).to(dt), lay.pack(v).to(dt)
    if G < H:
        o = _GroupedScalarGla.apply(qp, kp, vp, lay.pack(g.float()), scale, lay)
        return lay.unpack(o).to(v.dtype)
    b, khat, qbar, alpha = _scalar_prep(qp, kp, lay.pack(g.float()), scale, dt)
    d = b.permute(0, 2, 1)
    Aqk = _Scores.apply(_hm(qp), _hm(kp), d, scale, MASK_TRIL, dt)
    S = _DecayStates.apply(alpha, _hm(khat), _hm(vp), lay)
    o = bmm(_hm(qbar), S, b_mn=True, token_major=True, out_dtype=dt)
    o = bmm(Aqk, _hm(vp), b_mn=True, token_major=True, out_dtype=dt, addend=o)
    return lay.unpack(o.permute(0, 2, 1, 3)).to(v.dtype)


@_recomputable
def grouped_scalar_gla_chunks(q, k, v, g, lay: "ChunkLayout") -> torch.Tensor:
    """``scalar_gla_tc`` for heads in groups on operands in the rows of ``lay``: q, k ``[Tp, G, dk]``, v ``[Tp, H, dv]`` bf16 (zero in the padding), g
    ``[Tp, H]`` fp32; the result stays there, ``[NC, chunk, H, dv]``."""
    return _GroupedScalarGla.apply(*(slots.reshaped(t, lay.NC, lay.chunk, *t.shape[1:]) for t in (q, k, v, g)), 1.0, lay)


class _Gla(torch.autograd.Function):
    """The whole chunk pipeline of gated linear attention on 64-token chunks, on the kernels: v ``[NC, 64, H, dv]`` bf16; q, k ``[NC, 64, H, dk]``
    bf16 and g fp32 there too, or with ``tokens`` packed ``[T, H, dk]`` (``norm``: g is then the bf16 argument of ``logsigmoid(g) / norm``), which
    the kernels read, and whose gradients they write, where they lie.  One node, so that the two halves of the output and of dv
    accumulate in one GEMM each, and the channel-wise backward of preparation and diagonal sub-blocks is one kernel."""

    @staticmethod
    def forward(ctx, q, k, v, g, scale, lay, tokens, norm):
        from . import chunk_kernels
        v, rows = _lib.dense(v), lay if tokens else None
        ctx.slots = None, None
        if tokens:
            ctx.slots = slots.of(q), slots.of(k)
            q, k, g = (chunk_kernels.token_rows(t) for t in (q, k, g))
        else:
            q, k, g = (_lib.dense(t) for t in (q, k, g))
        (NC, C, H, dv), dk = v.shape, q.shape[-1]
        b, khat, qbar, qt, k3, alpha = chunk_kernels.gla_prep(q, k, g, scale, rows, norm)
        vh = _hm(v)
        S = _decay_states(lay, alpha, _hm(khat), vh, reverse=False)
        # off-diagonal sub-blocks: batch (chunk, I) multiplies the 16 query rows of sub-block I, re-based on the sub-block's
        # first row, with the keys before it re-based on the same row; later keys are zero in k3
        qt3 = qt.view(NC * 3, 16, H, dk)
        k3 = k3.view(NC * 3, 48, H, dk)
        A = chunk_kernels.gla_scores(q, k, b, bgemm(_hm(qt3), _hm(k3), alpha=scale), scale, rows)
        o = bgemm(_hm(qbar), S, b_mn=True, more=[(A, vh, False, True, 1)], out=_token_major(NC, H, C, dv, q.dtype, q.device))
        ctx.save_for_backward(q, k, v, b, khat, qbar, qt3, k3, alpha, S, A, None if norm is None else g)
        ctx.cfg = (scale, lay, rows, norm)
        return o.permute(0, 2, 1, 3)

    @staticmethod
    def backward(ctx, do):
        from . import chunk_kernels
        q, k, v, b, khat, qbar, qt3, k3, alpha, S, A, raw = ctx.saved_tensors
        scale, lay, rows, norm = ctx.cfg
        if rows is not None:  # saved-tensor hooks hand back copies, which lie wherever they were put
            q, k = chunk_kernels.token_rows(q), chunk_kernels.token_rows(k)
            raw = None if raw is None else chunk_kernels.token_rows(raw)
        NC, C, H, dk = b.shape
        dv = v.shape[-1]
        dt, dev = q.dtype, q.device
        doh, vh = _hm(_lib.dense(do.to(dt))), _hm(v)
        tok = lambda n: _token_major(NC, H, C, n, dt, dev)                                # noqa: E731
        back = lambda t: None if t is None else t.permute(0, 2, 1, 3)                     # noqa: E731
        need_q, need_k, need_v, need_g = ctx.needs_input_grad[:4]
        sums = need_q or need_k or need_g
        Ln, dalpha = _decay_states(lay, alpha, _hm(qbar), doh, True, S) if sums else (_decay_states(lay, alpha, _hm(qbar), doh, True), None)
        dvv = bgemm(_hm(khat), Ln, b_mn=True, more=[(A, doh, True, True, 1)], out=tok(dv)) if need_v else None
        if not sums:
            return None, None, back(dvv), None, None, None, None, None
        # one kernel forms the other three gradients, whichever of them are wanted
        dA = bgemm(doh, vh, mask=MASK_TRIL)
        dqbar, dkhat = bgemm(doh, S, out=tok(dk)), bgemm(vh, Ln, out=tok(dk))
        dblk = dA.view(NC, H, 4, 16, 64)[:, :, 1:, :, :48].permute(0, 2, 1, 3, 4).reshape(NC * 3, H, 16, 48)
        dqt3 = bgemm(dblk, _hm(k3), b_mn=True, alpha=scale, out=_token_major(NC * 3, H, 16, dk, dt, dev))
        dk3 = bgemm(dblk, _hm(qt3), a_mn=True, b_mn=True, alpha=scale, out=_token_major(NC * 3, H, 48, dk, dt, dev))
        grads = [None if s is None else s.take(lay.T, H * dk, dt, dev).view(lay.T, H, dk) for s in (*ctx.slots, None)]
        dq, dkk, dg = chunk_kernels.gla_bwd(q, k, b, dA, back(dkhat), back(dqbar), back(dqt3), back(dk3), dalpha, scale,
                                            rows, raw, norm or 1.0, grads)
        return dq, dkk, back(dvv), dg, None, None, None, None


def _gla_diag(qp, kp, b, scale, sub: int = 16):
    """[NC, H, 64, 64] fp32 holding only the diagonal sub-blocks of A_ij = scale sum_d q_id k_jd exp(b_id - b_jd), j <= i."""
    NC, C, H, dk = qp.shape
    A = torch.zeros(NC, H, C, C, dtype=torch.float32, device=qp.device)
    tri = torch.tril(torch.ones(sub, sub, dtype=torch.bool, device=qp.device))
    for i in range(C // sub):
        rows = slice(i * sub, (i + 1) * sub)
        d = b[:, rows, None] - b[:, None, rows]                       # [NC, sub, sub, H, dk]
        d = d.masked_fill(~tri[None, :, :, None, None], float("-inf")).exp()
        A[:, :, rows, rows] = torch.einsum("nihd,njhd,nijhd->nhij", qp[:, rows].float(), kp[:, rows].float(), d) * scale
    return A


def gla_raw_gate(q, k, v, raw, norm: float, meta: VarlenMeta, scale: Optional[float] = None):
    """``gla_tc`` with the gate ``logsigmoid(raw) / norm`` formed inside, from bf16 q, k, raw ``[T, H, dk]``, v ``[T, H, dv]``: the result, still
    in the rows of the layout, and the layout; None where the kernels do not apply."""
    if not (_lib.available() and q.is_cuda and all(t.dtype == torch.bfloat16 for t in (q, k, v, raw)) and q.shape == k.shape == raw.shape
            and q.shape[2] % 2 == 0 and getattr(meta, "sequence_slice", None) is None):
        return None
    lay = ChunkLayout.of(meta)
    if q.shape[0] != lay.T:
        return None
    return _gla_raw_gate(q, k, v, raw, q.shape[-1] ** -0.5 if scale is None else scale, lay, float(norm)), lay


@_recomputable
def _gla_raw_gate(q, k, v, raw, scale: float, lay: "ChunkLayout", norm: float) -> torch.Tensor:
    return _Gla.apply(q, k, lay.pack(v), raw, scale, lay, True, norm)


@_recomputable
def gla_tc(q, k, v, g, meta: VarlenMeta, scale: Optional[float] = None, sub: int = 16) -> torch.Tensor:
    """Chunked gated linear attention with one log decay per key channel: q, k, g ``[T, H, dk]``, v ``[T, H, dv]``.
    Same result as ``linear_attn.gla_recurrent``.  Inside a chunk the scores are built from 16-row sub-blocks:
    off-diagonal sub-blocks as products re-based on the query sub-block's first row (batched GEMM), diagonal
    sub-blocks pairwise, so every exponent is <= 0 for any gate values (fla/ops/gla/chunk.py:88-170)."""
    T, H, dk = q.shape
    scale = dk ** -0.5 if scale is None else scale
    lay = ChunkLayout.of(meta)
    dt = torch.bfloat16 if q.is_cuda else q.dtype
    C = lay.chunk
    if _lib.available() and q.is_cuda and C == 64 and sub == 16:
        if q.dtype == k.dtype == dt and q.shape[0] == lay.T:
            o = _Gla.apply(q, k, lay.pack(v).to(dt), g.float(), scale, lay, True, None)
        else:
            o = _Gla.apply(*(lay.pack(t).to(dt) for t in (q, k, v)), lay.pack(g.float()), scale, lay, False, None)
        return lay.unpack(o).to(v.dtype)
    qp, kp, vp = lay.pack(q).to(dt), lay.pack(k).to(dt), lay.pack(v).to(dt)   # [NC, 64, H, d]
    nb = C // sub
    NC = qp.shape[0]
    ncol = C - sub
    b = lay.pack(g.float()).cumsum(1)                                          # [NC, 64, H, dk]
    b_last = b[:, -1]                                                          # [NC, H, dk]
    alpha = b_last.exp()
    khat = kp * (b_last[:, None] - b).exp().to(dt)
    qbar = qp * (b.exp() * scale).to(dt)
    # off-diagonal sub-blocks: batch (chunk, I) multiplies the 16 query rows of sub-block I, re-based on the
    # sub-block's first row, with the keys before it re-based on the same row; later keys are zeroed
    r = b[:, ::sub].detach()                                                   # [NC, nb, H, dk]
    qt = qp * (b - r.repeat_interleave(sub, 1)).exp().to(dt)
    expo = r[:, 1:, None] - b[:, None, :ncol]                                  # [NC, nb-1, ncol, H, dk]
    keep = (torch.arange(ncol, device=q.device)[None, :] < (torch.arange(1, nb, device=q.device) * sub)[:, None])
    keep = keep[None, :, :, None, None]
    k3 = (kp[:, None, :ncol] * torch.where(keep, expo, expo.new_full((), float("-inf"))).exp().to(dt))
    S = _DecayStates.apply(alpha, _hm(khat), _hm(vp), lay)                 # [NC, H, dk, dv]
    o = bmm(_hm(qbar), S, b_mn=True, token_major=True, out_dtype=dt)
    A = _gla_diag(qp, kp, b, scale, sub)
    # all off-diagonal sub-blocks in ONE batched GEMM
    qt3 = qt[:, sub:].reshape(NC * (nb - 1), sub, H, dk)
    k3 = k3.reshape(NC * (nb - 1), ncol, H, dk)
    blk = bmm(_hm(qt3), _hm(k3), alpha=scale, out_dtype=torch.float32)         # [NC*(nb-1), H, sub, ncol]
    blk = blk.reshape(NC, nb - 1, H, sub, ncol).permute(0, 2, 1, 3, 4).reshape(NC, H, C - sub, ncol)
    A = A + torch.nn.functional.pad(blk, (0, sub, sub, 0))
    o = bmm(A.to(dt), _hm(vp), b_mn=True, token_major=True, out_dtype=dt, addend=o)
    return lay.unpack(o.permute(0, 2, 1, 3)).to(v.dtype)


class _VDecay(torch.autograd.Function):
    """The chunk pipeline with a decay along the VALUE dimension (first pass of gated slot attention) on packed 64-token chunks,
    on the kernels: q, k ``[NC, 64, H, dk]``, v ``[NC, 64, H, M]`` bf16, g ``[NC, 64, H, M]`` fp32.  Returns ``o`` in fp32, or with
    ``softmax`` its softmax over the slots in bf16.  The state is carried transposed (``[M, dk]``)."""

    @staticmethod
    def forward(ctx, q, k, v, g, scale, softmax, lay):
        from . import chunk_kernels
        q, k, v, g = (_lib.dense(t) for t in (q, k, v, g))
        NC, C, H, dk = q.shape
        M = v.shape[-1]
        qh, kh = _hm(q), _hm(k)
        b, vhat, v3, alpha = chunk_kernels.vdecay_prep(v, g)
        v3 = v3.view(NC * 3, 48, H, M)
        S = _decay_states(lay, alpha, _hm(vhat), kh, reverse=False)
        o1 = bgemm(qh, S, out=_token_major(NC, H, C, M, torch.float32, q.device))
        P16 = torch.empty(NC, H, C, C, dtype=q.dtype, device=q.device)
        P = bgemm(qh, kh, mask=MASK_TRIL, out_dtype=torch.float32, out16=P16)
        P3 = P16.view(NC, H, 4, 16, C)[:, :, 1:, :, :48].permute(0, 2, 1, 3, 4).reshape(NC * 3, H, 16, 48)
        acc = bgemm(P3, _hm(v3), b_mn=True, out=_token_major(NC * 3, H, 16, M, torch.float32, q.device))
        o, qv = chunk_kernels.vdecay_out(o1.permute(0, 2, 1, 3), acc.permute(0, 2, 1, 3), P, v, b, scale, softmax)
        ctx.save_for_backward(q, k, v, b, vhat, v3, alpha, S, P, P3, o)
        ctx.cfg = (scale, softmax, lay)
        return qv if softmax else o

    @staticmethod
    def backward(ctx, dout):
        from . import chunk_kernels
        q, k, v, b, vhat, v3, alpha, S, P, P3, o = ctx.saved_tensors
        scale, softmax, lay = ctx.cfg
        NC, C, H, dk = q.shape
        M = v.shape[-1]
        dt, dev = q.dtype, q.device
        need_q, need_k, need_v, need_g = ctx.needs_input_grad[:4]
        qh, kh = _hm(q), _hm(k)
        back = lambda t: None if t is None else t.permute(0, 2, 1, 3)                     # noqa: E731
        dq = dkk = dvv = dg = None
        dqv, d32 = (_lib.dense(dout.to(dt)), None) if softmax else (None, _lib.dense(dout.float()))
        do, do1, dacc = chunk_kernels.vdecay_bwd1(o, dqv, d32, b, scale)
        do1h, dacch = _hm(do1), _hm(dacc.view(NC * 3, 16, H, M))
        if need_k or need_v or need_g:
            sums = need_v or need_g
            Ln, dalpha = _decay_states(lay, alpha, do1h, qh, True, S) if sums else (_decay_states(lay, alpha, do1h, qh, True), None)
        if need_q or need_k:
            # gradient of the scores: off-diagonal sub-blocks by GEMM, the diagonal ones are pairwise sums like GLA's own scores
            dP = chunk_kernels.gla_scores(do, v, b, bgemm(dacch, _hm(v3)), 1.0)
        if need_q:
            dq = bgemm(do1h, S, b_mn=True, more=[(dP, kh, False, True, 1)], out=_token_major(NC, H, C, dk, dt, dev))
        if need_k:
            dkk = bgemm(_hm(vhat), Ln, b_mn=True, more=[(dP, qh, True, True, 1)], out=_token_major(NC, H, C, dk, dt, dev))
        if need_v or need_g:  # one kernel forms both
            dvhat = bgemm(kh, Ln, out=_token_major(NC, H, C, M, dt, dev))
            dv3 = bgemm(P3, dacch, a_mn=True, b_mn=True, out=_token_major(NC * 3, H, 48, M, dt, dev))
            dvv, dg = chunk_kernels.vdecay_bwd2(P, v, b, do, o, back(dvhat), back(dv3), dalpha, scale)
        return back(dq), back(dkk), dvv, dg, None, None, None


class _TwoReaders(torch.autograd.Function):
    """``x`` in ``dtype`` for two readers; their gradients are added in fp32 (autograd would add them in ``dtype``)."""

    @staticmethod
    def forward(ctx, x, dtype):
        ctx.dtype = x.dtype
        y = x.to(dtype)
        return y, y.detach()

    @staticmethod
    def backward(ctx, a, b):
        if a is None or b is None:
            d = b if a is None else a
            return None if d is None else d.to(ctx.dtype), None
        if _lib.available() and a.is_cuda and a.dtype == b.dtype == torch.bfloat16:
            from . import chunk_kernels
            return chunk_kernels.add_to_f32(a, b).to(ctx.dtype), None
        return torch.add(a.float(), b).to(ctx.dtype), None


def gsa_chunks(q, k, v, s, g, meta: VarlenMeta, scale: float) -> Optional[torch.Tensor]:
    """Both passes of gated slot attention without leaving the chunk layout between them (the slots' softmax rides on the first
    pass); None where the kernels do not apply."""
    from . import chunk_kernels
    M = s.shape[-1]
    if not (_lib.available() and q.is_cuda and M <= chunk_kernels.VDECAY_SOFTMAX_MAX and M % 8 == 0 and v.dtype == torch.bfloat16):
        return None
    return _gsa_chunks(q, k, v, s, g, meta, scale)


@_recomputable
def _gsa_chunks(q, k, v, s, g, meta: VarlenMeta, scale: float) -> torch.Tensor:
    lay = ChunkLayout.of(meta)
    qp, kp, vp = (lay.pack(t).to(torch.bfloat16) for t in (q, k, v))
    return lay.unpack(_gsa_padded.__wrapped__(qp, kp, vp, lay.pack(s), lay.pack(g.float()), lay, scale)).to(v.dtype)


def gsa_in_chunks_ok(slots: int, meta: VarlenMeta) -> bool:
    """Whether ``gsa_in_chunks`` takes bf16 operands with this many slots; asked before the projections are made."""
    from . import chunk_kernels
    return _lib.available() and slots <= chunk_kernels.VDECAY_SOFTMAX_MAX and slots % 8 == 0 and getattr(meta, "sequence_slice", None) is None


def gsa_in_chunks(qkv, sizes, heads: int, f, normalizer: float, meta: VarlenMeta, scale: float):
    """Both passes on q, k, v = the SiLU of column blocks of ``qkv [T, sum(sizes)]`` and the slots' gates from their bf16 argument ``f [T, heads, M]``;
    activation and gates go into the chunk layout on the way.  The result, still in the rows of the layout, and the layout; None where
    the kernels do not apply."""
    from .activations import silu_blocks_to_chunks
    from .gates import logsigmoid_gate
    if not (gsa_in_chunks_ok(f.shape[-1], meta) and qkv.is_cuda):
        return None
    lay = ChunkLayout.of(meta)
    qkv = silu_blocks_to_chunks(qkv, sizes, lay)
    if qkv is None:
        return None
    g, s = logsigmoid_gate(f, normalizer, True, lay)
    return _gsa_padded(*(t.view(lay.NC, lay.chunk, heads, -1) for t in qkv), s, g, lay, scale), lay


@_recomputable
def _gsa_padded(qp, kp, vp, sp, gp, lay: "ChunkLayout", scale: float) -> torch.Tensor:
    written, read = _TwoReaders.apply(sp, torch.bfloat16)
    qv = _VDecay.apply(qp, kp, written, gp, scale, True, lay)
    return _Gla.apply(qv, read, vp, gp, 1.0, lay, False, None)


@_recomputable
def gla_vdecay_tc(q, k, v, gv, meta: VarlenMeta, scale: float, sub: int = 16) -> torch.Tensor:
    """``S_t = S_{t-1} diag(exp gv_t) + k_t v_t^T,  o_t = scale q_t^T S_t``: the state decays along its VALUE dimension
    (first pass of gated slot attention, fla/ops/gsa/chunk.py).  q, k ``[T, H, dk]``, v, gv ``[T, H, dv]``; returns fp32.
    The state is carried transposed (``[dv, dk]``) so that the decay is per state row like in ``gla_tc``."""
    T, H, dk = q.shape
    lay = ChunkLayout.of(meta)
    dt = torch.bfloat16 if q.is_cuda else q.dtype
    C = lay.chunk
    qp, kp, vp = lay.pack(q).to(dt), lay.pack(k).to(dt), lay.pack(v).to(dt)
    if _lib.available() and q.is_cuda and C == 64 and sub == 16 and vp.shape[-1] % 8 == 0:
        return lay.unpack(_VDecay.apply(qp, kp, vp, lay.pack(gv.float()), scale, False, lay))
    b = lay.pack(gv.float()).cumsum(1)                                         # [NC, 64, H, dv]
    b_last = b[:, -1]
    vhat = vp * (b_last[:, None] - b).exp().to(dt)
    St = _DecayStates.apply(b_last.exp(), _hm(vhat), _hm(kp), lay)         # [NC, H, dv, dk]
    o = bmm(_hm(qp), St, token_major=True, out_dtype=torch.float32).permute(0, 2, 1, 3) * b.exp()   # [NC, 64, H, dv]
    P = bgemm_scores_plain(qp, kp)                                             # [NC, H, 64, 64] tril(q k^T)
    nb, ncol, NC = C // sub, C - sub, qp.shape[0]
    dv = vp.shape[-1]
    # off-diagonal sub-blocks, all in ONE batched GEMM: batch (chunk, I) multiplies the 16 score rows of sub-block I with
    # the values before it, re-based on the sub-block's first row r_I (every exponent is <= 0); values from sub-block I
    # on are zeroed, so the product may run over all 48 columns
    r = b[:, ::sub].detach()                                                   # [NC, nb, H, dv]
    expo = r[:, 1:, None] - b[:, None, :ncol]                                  # [NC, nb-1, ncol, H, dv]
    keep = (torch.arange(ncol, device=q.device)[None, :] < (torch.arange(1, nb, device=q.device) * sub)[:, None])
    keep = keep[None, :, :, None, None]
    v3 = vp[:, None, :ncol] * torch.where(keep, expo, expo.new_full((), float("-inf"))).exp().to(dt)
    P3 = P[:, :, sub:, :ncol].reshape(NC, H, nb - 1, sub, ncol).permute(0, 2, 1, 3, 4).reshape(NC * (nb - 1), H, sub, ncol)
    acc = bmm(P3.to(dt), _hm(v3.reshape(NC * (nb - 1), ncol, H, dv)), b_mn=True, token_major=True,
              out_dtype=torch.float32)                                         # [NC*(nb-1), H, sub, dv] over [.., sub, H, dv]
    acc = acc.permute(0, 2, 1, 3).reshape(NC, ncol, H, dv) * (b[:, sub:] - r[:, 1:].repeat_interleave(sub, 1)).exp()
    o = o + torch.nn.functional.pad(acc, (0, 0, 0, 0, sub, 0))
    tri = torch.tril(torch.ones(sub, sub, dtype=torch.bool, device=q.device))
    parts = []
    for i in range(nb):
        rows = slice(i * sub, (i + 1) * sub)
        dd = (b[:, rows, None] - b[:, None, rows]).masked_fill(~tri[None, :, :, None, None], float("-inf")).exp()
        parts.append(torch.einsum("nhij,njhc,nijhc->nihc", P[:, :, rows, rows].float(), vp[:, rows].float(), dd))
    o = o + torch.cat(parts, 1)
    o = o * scale
    return lay.unpack(o)


def bgemm_scores_plain(qp, kp):
    """``tril(q k^T)`` per chunk and head, differentiable: [NC, H, 64, 64] fp32."""
    zero = torch.zeros(qp.shape[0], qp.shape[2], qp.shape[1], dtype=torch.float32, device=qp.device)
    return _Scores.apply(_hm(qp), _hm(kp), zero, 1.0, MASK_TRIL, torch.float32)
