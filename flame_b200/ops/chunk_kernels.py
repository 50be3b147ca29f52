"""ctypes wrappers of the CUDA-core helper kernels of the chunk algorithms (``csrc/chunk.cu``)."""
from __future__ import annotations

from ctypes import c_float, c_int, c_longlong, c_void_p

import torch

from . import _lib, slots

_lib.register("fb_delta_inverse", [c_void_p] * 3 + [c_int] * 3 + [c_void_p] * 5)
_lib.register("fb_delta_scale", [c_void_p] * 3 + [c_int] * 3 + [c_void_p] * 3)
_lib.register("fb_delta_bwd_t", [c_void_p] * 5 + [c_int] * 3 + [c_float] + [c_void_p] * 4)
_lib.register("fb_delta_bwd_scores", [c_void_p] * 6 + [c_int] * 3 + [c_float] * 2 + [c_void_p] * 5)


def delta_inverse(P: torch.Tensor, beta: torch.Tensor, b, bgemm):
    """``T = (I + diag(beta) P)^-1``, ``Tu = T diag(beta)`` and, with a decay ``b``, ``Tw = T diag(beta e^b)`` (bf16) for the
    strictly lower-triangular fp32 ``P [NC, H, C, C]``, C = 64 or 128; beta, b ``[NC, C, H]`` fp32 contiguous.  At C = 128 the
    diagonal blocks are inverted and ``T21 = -T22 A21 T11`` comes from two batched GEMMs."""
    NC, H, C, _ = P.shape
    new = lambda: torch.empty(P.shape, dtype=torch.bfloat16, device=P.device)  # noqa: E731
    T, Tu, Tw = new(), new(), None if b is None else new()
    A21 = torch.empty(NC, H, 64, 64, dtype=torch.bfloat16, device=P.device) if C == 128 else None
    L = _lib.lib()
    _lib.check(L.fb_delta_inverse(P.data_ptr(), beta.data_ptr(), _lib.ptr(b), NC, H, C, T.data_ptr(), Tu.data_ptr(), _lib.ptr(Tw),
                                  _lib.ptr(A21), _lib.stream_ptr()), "fb_delta_inverse")
    _lib.count_launch()
    if C == 128:
        X = bgemm(T[..., 64:, 64:], A21, b_mn=True)
        bgemm(X, T[..., :64, :64], b_mn=True, alpha=-1.0, out=T[..., 64:, :64])
        _lib.check(L.fb_delta_scale(T.data_ptr(), beta.data_ptr(), _lib.ptr(b), NC, H, C, Tu.data_ptr(), _lib.ptr(Tw), _lib.stream_ptr()),
                   "fb_delta_scale")
        _lib.count_launch()
    return T, Tu, Tw


def delta_bwd_t(T, dTu, dTw, beta, b, scale: float):
    """``dT`` (bf16) from the gradients of ``Tu`` and ``Tw``, and the parts of ``dbeta``, ``db`` (``[NC, C, H]`` fp32, times
    ``scale``) that come from the column factors.  ``dTw`` and ``b`` are None without a decay."""
    NC, H, C, _ = T.shape
    dT = torch.empty_like(T)
    dbeta = torch.empty_like(beta)
    db = None if b is None else torch.empty_like(b)
    _lib.check(_lib.lib().fb_delta_bwd_t(T.data_ptr(), dTu.data_ptr(), _lib.ptr(dTw), beta.data_ptr(), _lib.ptr(b), NC, H, C, float(scale),
                                         dT.data_ptr(), dbeta.data_ptr(), _lib.ptr(db), _lib.stream_ptr()), "fb_delta_bwd_t")
    _lib.count_launch()
    return dT, dbeta, db


def delta_bwd_scores(dA, P, dQ, Q, beta, b, scale: float, dbeta, db):
    """The bf16 operands ``g`` (of k k^T) and, with a decay and ``dQ``, ``gq`` (of q k^T) of the dq / dk products; adds to ``dbeta``
    and ``db``."""
    NC, H, C, _ = P.shape
    g = torch.empty(P.shape, dtype=torch.bfloat16, device=P.device)
    both = b is not None and dQ is not None
    gq = torch.empty_like(g) if both else None
    _lib.check(_lib.lib().fb_delta_bwd_scores(dA.data_ptr(), P.data_ptr(), dQ.data_ptr() if both else 0, Q.data_ptr() if both else 0,
                                              beta.data_ptr(), _lib.ptr(b), NC, H, C, float(scale), 1.0, g.data_ptr(), _lib.ptr(gq),
                                              dbeta.data_ptr(), _lib.ptr(db), _lib.stream_ptr()), "fb_delta_bwd_scores")
    _lib.count_launch()
    return g, gq


_lib.register("fb_group_prep_fwd", [c_void_p] * 2 + [c_int] * 4 + [c_float] + [c_void_p] * 5)
_lib.register("fb_group_bwd1", [c_void_p] * 3 + [c_int] * 4 + [c_void_p] * 3)
_lib.register("fb_group_bwd2", [c_void_p] * 7 + [c_int] * 4 + [c_void_p] * 3)


def group_supported(C: int, dv: int) -> bool:
    n = dv // 8
    return C in (64, 128) and dv % 8 == 0 and 1 <= n <= 32 and (n & (n - 1)) == 0


def group_prep(v, g, scale: float):
    """``b = cumsum(g)``, ``eb = scale e^b``, ``alpha = e^{b_last}``, ``vhat = v e^{b_last - b}`` for v ``[NC, C, H, dv]`` bf16 and g
    ``[NC, C, H]`` fp32, both contiguous."""
    NC, C, H, dv = v.shape
    b, eb = torch.empty_like(g), torch.empty_like(g)
    alpha = torch.empty(NC, H, dtype=torch.float32, device=v.device)
    vhat = torch.empty_like(v)
    _lib.check(_lib.lib().fb_group_prep_fwd(v.data_ptr(), g.data_ptr(), NC, C, H, dv, float(scale), b.data_ptr(), eb.data_ptr(),
                                            alpha.data_ptr(), vhat.data_ptr(), _lib.stream_ptr()), "fb_group_prep_fwd")
    _lib.count_launch()
    return b, eb, alpha, vhat


def group_bwd1(do, o1, eb):
    """``do eb`` and the row sums of ``do o1``."""
    NC, C, H, dv = do.shape
    dos, db = torch.empty_like(do), torch.empty_like(eb)
    _lib.check(_lib.lib().fb_group_bwd1(do.data_ptr(), o1.data_ptr(), eb.data_ptr(), NC, C, H, dv, dos.data_ptr(), db.data_ptr(),
                                        _lib.stream_ptr()), "fb_group_bwd1")
    _lib.count_launch()
    return dos, db


def group_bwd2(dvhat, vhat, dv1, b, db, alpha, dalpha):
    """``dv`` and ``dg`` (see ``csrc/chunk.cu: group_bwd2_kernel``), each None without ``dv1`` and ``dalpha``."""
    NC, C, H, dv = vhat.shape
    dvo = None if dv1 is None else torch.empty_like(vhat)
    dg = None if dalpha is None else torch.empty_like(b)
    _lib.check(_lib.lib().fb_group_bwd2(dvhat.data_ptr(), vhat.data_ptr(), _lib.ptr(dv1), b.data_ptr(), db.data_ptr(), alpha.data_ptr(),
                                        _lib.ptr(dalpha), NC, C, H, dv, _lib.ptr(dvo), _lib.ptr(dg), _lib.stream_ptr()), "fb_group_bwd2")
    _lib.count_launch()
    return dvo, dg


def scores_bwd(dQ, Q, b, db, scale: float):
    """bf16 ``scale dQ_ij e^{b_i - b_j}`` (j <= i) and, added to ``db [NC, C, H]``, the gradient of ``b`` through ``Q``: the part of
    ``delta_bwd_scores`` that attention without a delta rule has."""
    NC, H, C, _ = Q.shape
    gq = torch.empty_like(Q)
    _lib.check(_lib.lib().fb_delta_bwd_scores(0, 0, dQ.data_ptr(), Q.data_ptr(), 0, b.data_ptr(), NC, H, C, 1.0, float(scale), 0, gq.data_ptr(), 0,
                                              _lib.ptr(db), _lib.stream_ptr()), "fb_delta_bwd_scores")
    _lib.count_launch()
    return gq


_lib.register("fb_gla_scores", [c_void_p, c_int] + [c_void_p] * 5 + [c_longlong] * 2 + [c_int] * 3 + [c_float, c_void_p])
_lib.register("fb_gla_bwd", [c_void_p] * 13 + [c_float, c_void_p] + [c_longlong] * 6 + [c_int] * 3 + [c_float, c_void_p])


def _token_ld(x: torch.Tensor) -> int:
    """Elements between the tokens of ``[T, H, d]`` (of one token its length, whatever stride torch keeps for it)."""
    return x.stride(0) if x.shape[0] > 1 else x.shape[1] * x.shape[2]


def token_rows(x: torch.Tensor) -> torch.Tensor:
    """``x [T, H, d]``, or a dense copy: a token's values side by side, tokens whole 16-byte vectors apart, on a 16-byte boundary."""
    H, d = x.shape[1:]
    ld, e = _token_ld(x), x.element_size()
    ok = (d == 1 or x.stride(2) == 1) and (H == 1 or x.stride(1) == d) and ld >= H * d and ld * e % 16 == 0 and x.data_ptr() % 16 == 0
    return x if ok else _lib.dense(x)


def _gla_rows(q, k, lay):
    """Arguments of ``csrc/chunk.cu: GlaRows`` for q and k: packed tokens of ``lay``, or padded rows ``[NC, 64, H, d]`` (None)."""
    if lay is None:
        n = q.shape[2] * q.shape[3]
        return 0, n, n
    return lay.inv_i32.data_ptr(), _token_ld(q), _token_ld(k)


def gla_scores(q, k, b, blk, scale: float, lay=None) -> torch.Tensor:
    """bf16 ``A [NC, H, 64, 64]``: diagonal 16 x 16 sub-blocks computed here, the ones left of them from ``blk [3 NC, H, 16, 48]``
    bf16; q (or fp32), k bf16: contiguous ``[NC, 64, H, dk]``, or with ``lay`` packed ``token_rows``; b fp32 contiguous."""
    NC, _, H, dk = b.shape
    A = torch.empty(NC, H, 64, 64, dtype=torch.bfloat16, device=q.device)
    src, ldq, ldk = _gla_rows(q, k, lay)
    _lib.check(_lib.lib().fb_gla_scores(q.data_ptr(), int(q.dtype == torch.float32), k.data_ptr(), b.data_ptr(), blk.data_ptr(), A.data_ptr(),
                                        src, ldq, ldk, NC, H, dk, float(scale), _lib.stream_ptr()), "fb_gla_scores")
    _lib.count_launch()
    return A


def gla_bwd(q, k, b, dA, dkhat, dqbar, dqt, dk3, dalpha, scale: float, lay=None, raw=None, norm: float = 1.0, grads=(None, None, None)):
    """``dq, dk`` (bf16) and ``dg`` of a chunk (see ``csrc/chunk.cu: gla_bwd_kernel``): fp32, or with ``raw`` that of the gate's bf16 argument.
    With ``lay`` q, k, ``raw`` and the gradients are packed tokens; ``grads``: where dq, dk and dg belong ``[T, H, dk]``."""
    NC, _, H, dk = b.shape
    if lay is None:
        dq, dk_, dg = torch.empty_like(q), torch.empty_like(k), torch.empty_like(b)
        lds = [H * dk] * 6
    else:
        new = lambda dt: torch.empty(lay.T, H, dk, dtype=dt, device=q.device)  # noqa: E731
        dq, dk_, dg = (new(torch.float32 if i == 2 and raw is None else torch.bfloat16) if t is None else t for i, t in enumerate(grads))
        lds = [_token_ld(q), _token_ld(k), H * dk if raw is None else _token_ld(raw), *(_token_ld(t) for t in (dq, dk_, dg))]
    _lib.check(_lib.lib().fb_gla_bwd(q.data_ptr(), k.data_ptr(), b.data_ptr(), dA.data_ptr(), dkhat.data_ptr(), dqbar.data_ptr(),
                                     dqt.data_ptr(), dk3.data_ptr(), dalpha.data_ptr(), dq.data_ptr(), dk_.data_ptr(), dg.data_ptr(), _lib.ptr(raw),
                                     1.0 / float(norm), 0 if lay is None else lay.inv_i32.data_ptr(), *lds, NC, H, dk, float(scale), _lib.stream_ptr()),
               "fb_gla_bwd")
    _lib.count_launch()
    return dq, dk_, dg


_lib.register("fb_l2norm_fwd", [c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_float, c_void_p])
_lib.register("fb_l2norm_bwd", [c_void_p, c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_void_p])


class _L2Norm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, eps):
        xc = x.contiguous()
        D = xc.shape[-1]
        rows = xc.numel() // D
        y = torch.empty_like(xc)
        rstd = torch.empty(rows, dtype=torch.float32, device=x.device)
        _lib.check(_lib.lib().fb_l2norm_fwd(xc.data_ptr(), y.data_ptr(), rstd.data_ptr(), rows, D, float(eps),
                                            _lib.stream_ptr()), "fb_l2norm_fwd")
        _lib.count_launch()
        ctx.save_for_backward(xc, rstd)
        return y

    @staticmethod
    def backward(ctx, dy):
        xc, rstd = ctx.saved_tensors
        dy = dy.contiguous()
        D = xc.shape[-1]
        dx = torch.empty_like(xc)
        _lib.check(_lib.lib().fb_l2norm_bwd(xc.data_ptr(), rstd.data_ptr(), dy.data_ptr(), dx.data_ptr(), xc.numel() // D, D,
                                            _lib.stream_ptr()), "fb_l2norm_bwd")
        _lib.count_launch()
        return dx, None


def l2norm(x: torch.Tensor, eps: float = 1e-6) -> torch.Tensor:
    """``x * rsqrt(sum(x^2, -1) + eps)`` for bf16 ``x [..., D]``, D <= 1024 (fla/modules/l2norm.py)."""
    return _L2Norm.apply(x, eps)


_lib.register("fb_add_bf16_to_f32", [c_void_p] * 3 + [c_longlong, c_void_p])


def add_to_f32(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """``a + b`` in fp32 of two bf16 tensors of one shape."""
    a, b = _lib.dense(a), _lib.dense(b)
    out = torch.empty(a.shape, dtype=torch.float32, device=a.device)
    _lib.check(_lib.lib().fb_add_bf16_to_f32(a.data_ptr(), b.data_ptr(), out.data_ptr(), a.numel(), _lib.stream_ptr()), "fb_add_bf16_to_f32")
    _lib.count_launch()
    return out


_lib.register("fb_pair_dot", [c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_int, c_int, c_void_p])


def pair_dot(x: torch.Tensor, y: torch.Tensor, per_row: bool) -> torch.Tensor:
    """fp32 ``sum(x * y)`` over the last two dims (``per_row``: the last dim) of bf16 ``[..., R, C]`` tensors."""
    x, y = _lib.dense(x), _lib.dense(y)
    R, C = x.shape[-2:]
    B = x.numel() // (R * C)
    out = torch.empty(*x.shape[:-2], *([R] if per_row else []), dtype=torch.float32, device=x.device)
    _lib.check(_lib.lib().fb_pair_dot(x.data_ptr(), y.data_ptr(), out.data_ptr(), B, R, C, int(per_row), _lib.stream_ptr()),
               "fb_pair_dot")
    _lib.count_launch()
    return out


_lib.register("fb_state_scan", [c_void_p, c_void_p, c_int, c_void_p, c_int, c_void_p, c_int, c_void_p, c_int, c_int, c_int, c_int,
                                c_void_p])


def state_scan(first: torch.Tensor, last: torch.Tensor, alpha: torch.Tensor, x: torch.Tensor, reverse: bool) -> torch.Tensor:
    """bf16 ``[NC, H, rows, cols]``: the state entering every chunk (reverse: the adjoint of the state leaving it) of the
    recurrence ``s = alpha_c s + x_c`` over the chunks ``first .. last`` (int64) of every document, from zero; ``x`` fp32 or bf16."""
    x = _lib.dense(x)
    _, H, rows, cols = x.shape
    out = torch.empty(x.shape, dtype=torch.bfloat16, device=x.device)
    per_row = 1 if alpha.dim() == 3 else 0
    rc = _lib.lib().fb_state_scan(first.data_ptr(), last.data_ptr(), first.numel(), alpha.data_ptr(), per_row, x.data_ptr(),
                                  int(x.dtype == torch.bfloat16), out.data_ptr(), H, rows, cols, int(reverse), _lib.stream_ptr())
    _lib.check(rc, "fb_state_scan")
    _lib.count_launch()
    return out


_lib.register("fb_gla_prep_fwd", [c_void_p] * 3 + [c_int, c_float, c_void_p] + [c_longlong] * 3 + [c_void_p] * 6 + [c_int] * 3 + [c_float, c_void_p])


def gla_prep(q, k, g, scale: float, lay=None, norm=None):
    """One pass over a chunk's q, k, g producing the cumulative decay and every scaled operand of the GLA chunk algorithm (see
    ``csrc/chunk.cu: gla_prep_fwd_kernel``).  q, k ``[NC, 64, H, dk]`` bf16, g fp32, all contiguous; with ``lay`` they are packed
    ``token_rows [T, H, dk]``, and with ``norm`` too g is the bf16 argument of ``logsigmoid(g) / norm``.  Returns
    ``(b, khat, qbar, qt, k3, alpha)``; qt ``[NC, 48, H, dk]``."""
    NC, (H, dk), dev = q.shape[0] if lay is None else lay.NC, q.shape[-2:], q.device
    assert q.dtype == k.dtype == torch.bfloat16 and g.dtype == (torch.float32 if norm is None else torch.bfloat16)
    new = lambda *n, dt=torch.bfloat16: torch.empty(*n, H, dk, dtype=dt, device=dev)  # noqa: E731
    b, khat, qbar, qt, k3 = new(NC, 64, dt=torch.float32), new(NC, 64), new(NC, 64), new(NC, 48), new(NC, 3, 48)
    alpha = new(NC, dt=torch.float32)
    src, ldq, ldk = _gla_rows(q, k, lay)
    rc = _lib.lib().fb_gla_prep_fwd(q.data_ptr(), k.data_ptr(), g.data_ptr(), int(norm is not None), float(norm or 1.0), src, ldq, ldk,
                                    H * dk if lay is None else _token_ld(g), b.data_ptr(), khat.data_ptr(), qbar.data_ptr(), qt.data_ptr(),
                                    k3.data_ptr(), alpha.data_ptr(), NC, H, dk, float(scale), _lib.stream_ptr())
    _lib.check(rc, "fb_gla_prep_fwd")
    _lib.count_launch()
    return b, khat, qbar, qt, k3, alpha


_lib.register("fb_scalar_prep_fwd", [c_void_p] * 7 + [c_int, c_int, c_int, c_int, c_float, c_void_p])
_lib.register("fb_scalar_prep_bwd", [c_void_p] * 10 + [c_int, c_int, c_int, c_int, c_float, c_void_p])


def scalar_prep_supported(C: int, dk: int) -> bool:
    n = dk // 8
    return C in (64, 128) and dk % 8 == 0 and n > 0 and (n & (n - 1)) == 0


def scalar_prep(qp, kp, gp, scale: float):
    """``b = cumsum(g)``, ``khat = k e^{b_last - b}``, ``qbar = scale q e^{b}``, ``alpha = e^{b_last}`` in one kernel; q, k
    ``[NC, C, H, dk]`` bf16, g ``[NC, C, H]`` fp32, all contiguous."""
    NC, C, H, dk = qp.shape
    dev = qp.device
    b = torch.empty(NC, C, H, dtype=torch.float32, device=dev)
    khat, qbar = torch.empty_like(kp), torch.empty_like(qp)
    alpha = torch.empty(NC, H, dtype=torch.float32, device=dev)
    rc = _lib.lib().fb_scalar_prep_fwd(qp.data_ptr(), kp.data_ptr(), gp.data_ptr(), b.data_ptr(), khat.data_ptr(),
                                       qbar.data_ptr(), alpha.data_ptr(), NC, C, H, dk, float(scale), _lib.stream_ptr())
    _lib.check(rc, "fb_scalar_prep_fwd")
    _lib.count_launch()
    return b, khat, qbar, alpha


def scalar_prep_bwd(qp, kp, b, dkhat, dqbar, dalpha, db, scale: float):
    """``dq, dk`` (bf16) and ``dg`` (fp32) of ``scalar_prep``; the incoming gradients are contiguous (or None)."""
    NC, C, H, dk = qp.shape
    dq, dk_, dg = torch.empty_like(qp), torch.empty_like(kp), torch.empty_like(b)
    rc = _lib.lib().fb_scalar_prep_bwd(qp.data_ptr(), kp.data_ptr(), b.data_ptr(), _lib.ptr(dkhat), _lib.ptr(dqbar),
                                       _lib.ptr(dalpha), _lib.ptr(db), dq.data_ptr(), dk_.data_ptr(), dg.data_ptr(), NC,
                                       C, H, dk, float(scale), _lib.stream_ptr())
    _lib.check(rc, "fb_scalar_prep_bwd")
    _lib.count_launch()
    return dq, dk_, dg


class ScalarPrep(torch.autograd.Function):
    """``scalar_prep`` with its gradients: the token-sized operands of the scalar-gated chunk algorithms."""

    @staticmethod
    def forward(ctx, qp, kp, gp, scale):
        qp, kp = _lib.dense(qp), _lib.dense(kp)
        b, khat, qbar, alpha = scalar_prep(qp, kp, gp.float().contiguous(), scale)
        ctx.save_for_backward(qp, kp, b)
        ctx.scale = scale
        return b, khat, qbar, alpha

    @staticmethod
    def backward(ctx, db, dkhat, dqbar, dalpha):
        qp, kp, b = ctx.saved_tensors
        dkhat = None if dkhat is None else _lib.dense(dkhat.to(torch.bfloat16))
        dqbar = None if dqbar is None else _lib.dense(dqbar.to(torch.bfloat16))
        db = None if db is None else db.float().contiguous()
        dalpha = None if dalpha is None else dalpha.float().contiguous()
        dq, dk_, dg = scalar_prep_bwd(qp, kp, b, dkhat, dqbar, dalpha, db, ctx.scale)
        return dq, dk_, dg, None


_vp, _i, _ll = c_void_p, c_int, c_longlong
_SSCAN_IN = [_vp, _ll, _vp, _ll, _i, _vp, _ll, _vp, _ll, _vp, _ll, _i, _vp, _vp, _vp, _vp, _vp, _i]
_lib.register("fb_sscan_fwd", _SSCAN_IN + [_vp] * 4 + [_i] * 4 + [_vp])
_lib.register("fb_sscan_bwd", _SSCAN_IN + [_vp] * 8 + [_ll] + [_vp] * 5 + [_ll] + [_i] * 3 + [_vp])
_lib.register("fb_sscan_channel_blocks", [c_int])
_lib.register("fb_sscan_padded", [c_int])


def _rows(x: torch.Tensor) -> torch.Tensor:
    """``x`` with unit stride along its rows (the kernels take any row stride)."""
    return x if x.stride(1) == 1 or x.shape[1] == 1 else x.contiguous()


_lib.register("fb_colsum_parts", [c_void_p, c_int, c_int, c_void_p, c_void_p])


def _sum_parts(x: torch.Tensor) -> torch.Tensor:
    """``x.sum(0)`` of contiguous fp32 partials ``[parts, ...]``, in a fixed order."""
    out = torch.empty(x.shape[1:], dtype=torch.float32, device=x.device)
    _lib.check(_lib.lib().fb_colsum_parts(x.data_ptr(), x.shape[0], out.numel(), out.data_ptr(), _lib.stream_ptr()), "fb_colsum_parts")
    _lib.count_launch()
    return out


class SelectiveScan(torch.autograd.Function):
    """Mamba-1 selective scan on the chunk-parallel kernels of ``csrc/sscan.cu``, on packed tokens: u ``[T, Di]`` bf16, delta
    ``[T, Di]`` (fp32, or with ``raw`` the bf16 argument of a softplus), A ``[Di, 16]`` fp32, B, C ``[T, 16]`` (both bf16 or both
    fp32), D ``[Di]`` fp32; z ``[T, Di]`` bf16 or None.  Rows may have any stride.  Returns bf16 ``[T, Di]``: y, or ``y silu(z)``.
    ``lay``: the 64-token ``ChunkLayout`` of the documents; ``keep``: a backward may follow (known to the caller only, as inside
    of ``forward`` gradients are always off)."""

    @staticmethod
    def forward(ctx, u, delta, A, B, C, D, z, lay, raw, keep):
        u, delta, B, C = _rows(u), _rows(delta), _rows(B), _rows(C)
        ctx.z_slot = None if z is None else slots.of(z)
        z = None if z is None else _rows(z)
        A, D = _lib.dense(A), D.contiguous()
        T, Di = lay.T, u.shape[1]
        for t in (u, delta, B, C) + (() if z is None else (z,)):
            if t.shape[0] < T:
                raise ValueError(f"selective scan: {t.shape[0]} rows for documents of {T} tokens")
        dev = u.device
        L = _lib.lib()
        DiP = int(L.fb_sscan_padded(Di))
        st = torch.empty(lay.NC, 4 if keep else 1, 16, DiP, dtype=torch.float32, device=dev)
        sdl = torch.empty(lay.NC, DiP, dtype=torch.float32, device=dev)
        y = torch.empty(T, Di, dtype=torch.bfloat16, device=dev) if keep or z is None else None
        out = torch.empty(T, Di, dtype=torch.bfloat16, device=dev) if z is not None else None
        ctx.geometry = (lay, raw, DiP)
        rc = L.fb_sscan_fwd(*SelectiveScan._operands(u, delta, A, B, C, D, z, lay, raw), st.data_ptr(), sdl.data_ptr(), _lib.ptr(y),
                            _lib.ptr(out), int(keep), lay.NC, Di, A.shape[1], _lib.stream_ptr())
        _lib.check(rc, "fb_sscan_fwd")
        _lib.count_launch(3)
        ctx.save_for_backward(u, delta, A, B, C, D, z, st, sdl, y if z is not None else None)
        return y if z is None else out

    @staticmethod
    def _operands(u, delta, A, B, C, D, z, lay, raw):
        return (u.data_ptr(), u.stride(0), delta.data_ptr(), delta.stride(0), int(raw), _lib.ptr(z), 0 if z is None else z.stride(0),
                B.data_ptr(), B.stride(0), C.data_ptr(), C.stride(0), int(B.dtype == torch.bfloat16), A.data_ptr(), D.data_ptr(),
                lay.inv_i32.data_ptr(), lay.first.data_ptr(), lay.last.data_ptr(), lay.first.numel())

    @staticmethod
    def backward(ctx, dout):
        u, delta, A, B, C, D, z, st, sdl, y = ctx.saved_tensors
        assert st.shape[1] == 4, "the forward was told that no backward follows"
        lay, raw, DiP = ctx.geometry
        T, Di = lay.T, u.shape[1]
        dev = u.device
        L = _lib.lib()
        dout = dout.to(torch.bfloat16).contiguous()

        def grad(like):  # rows past the documents have no part in the result
            t = torch.empty(like.shape, dtype=like.dtype, device=dev)
            if like.shape[0] > T:
                t[T:].zero_()
            return t
        du, ddl, dB, dC = grad(u), grad(delta), grad(B), grad(C)
        dz = None
        if z is not None:
            dz = ctx.z_slot.take(T, Di, z.dtype, dev) if ctx.z_slot is not None and z.shape[0] == T else grad(z)
        nblk = int(L.fb_sscan_channel_blocks(Di))
        adj = torch.empty(lay.NC, 16, DiP, dtype=torch.float32, device=dev)
        dA = torch.empty(lay.NC, 16, DiP, dtype=torch.float32, device=dev)     # per-chunk partials, summed below
        dD = torch.empty(lay.NC, DiP, dtype=torch.float32, device=dev)
        part = torch.empty(nblk, T, 32, dtype=torch.float32, device=dev)       # per-channel-block partials of dB | dC
        rc = L.fb_sscan_bwd(*SelectiveScan._operands(u, delta, A, B, C, D, z, lay, raw), st.data_ptr(), sdl.data_ptr(), _lib.ptr(y),
                            dout.data_ptr(), adj.data_ptr(), du.data_ptr(), ddl.data_ptr(), _lib.ptr(dz),
                            0 if dz is None else dz.stride(0), dA.data_ptr(),
                            part.data_ptr(), dD.data_ptr(), dB.data_ptr(), dC.data_ptr(), T, lay.NC, Di, A.shape[1], _lib.stream_ptr())
        _lib.check(rc, "fb_sscan_bwd")
        _lib.count_launch(4)
        dA, dD = _sum_parts(dA), _sum_parts(dD)
        return du, ddl, dA[:, :Di].t(), dB, dC, dD[:Di], dz, None, None, None


_lib.register("fb_vdecay_prep", [c_void_p] * 6 + [c_int] * 3 + [c_void_p])
_lib.register("fb_vdecay_out", [c_void_p] * 5 + [c_int] * 3 + [c_float] + [c_void_p] * 3)
_lib.register("fb_vdecay_bwd1", [c_void_p] * 4 + [c_int] * 3 + [c_float] + [c_void_p] * 4)
_lib.register("fb_vdecay_bwd2", [c_void_p] * 8 + [c_int] * 3 + [c_float] + [c_void_p] * 3)
VDECAY_SOFTMAX_MAX = 512   # slots whose softmax rides on ``vdecay_out``


def vdecay_prep(v, g):
    """``b = cumsum(g)``, ``vhat = v e^{b_last - b}``, ``v3`` (values re-based for the sub-blocks behind them, ``[NC, 3, 48, H, M]``)
    and ``alpha = e^{b_last}``; v ``[NC, 64, H, M]`` bf16, g fp32, contiguous."""
    NC, C, H, M = v.shape
    assert C == 64 and v.dtype == torch.bfloat16 and g.dtype == torch.float32
    b, vhat = torch.empty_like(g), torch.empty_like(v)
    v3 = torch.empty(NC, 3, 48, H, M, dtype=v.dtype, device=v.device)
    alpha = torch.empty(NC, H, M, dtype=torch.float32, device=v.device)
    _lib.check(_lib.lib().fb_vdecay_prep(v.data_ptr(), g.data_ptr(), b.data_ptr(), vhat.data_ptr(), v3.data_ptr(), alpha.data_ptr(), NC, H,
                                         M, _lib.stream_ptr()), "fb_vdecay_prep")
    _lib.count_launch()
    return b, vhat, v3, alpha


def vdecay_out(o1, acc, P, v, b, scale: float, softmax: bool):
    """``o`` fp32 and, with ``softmax``, its softmax over the last dimension in bf16 (see ``csrc/chunk.cu: vdecay_out_kernel``)."""
    NC, C, H, M = v.shape
    o = torch.empty_like(b)
    qv = torch.empty_like(v) if softmax else None
    _lib.check(_lib.lib().fb_vdecay_out(o1.data_ptr(), acc.data_ptr(), P.data_ptr(), v.data_ptr(), b.data_ptr(), NC, H, M, float(scale),
                                        o.data_ptr(), _lib.ptr(qv), _lib.stream_ptr()), "fb_vdecay_out")
    _lib.count_launch()
    return o, qv


def vdecay_bwd1(o, dqv, d32, b, scale: float):
    """``do`` (fp32, from the gradient ``dqv`` of the softmax, or ``d32`` of ``o``), ``do e^b`` and ``do e^{b - r_I}`` (rows 16..63)."""
    NC, C, H, M = b.shape
    do = torch.empty_like(b)
    do1 = torch.empty(b.shape, dtype=torch.bfloat16, device=b.device)
    dacc = torch.empty(NC, 48, H, M, dtype=torch.bfloat16, device=b.device)
    _lib.check(_lib.lib().fb_vdecay_bwd1(o.data_ptr(), _lib.ptr(dqv), _lib.ptr(d32), b.data_ptr(), NC, H, M, float(scale), do.data_ptr(),
                                         do1.data_ptr(), dacc.data_ptr(), _lib.stream_ptr()), "fb_vdecay_bwd1")
    _lib.count_launch()
    return do, do1, dacc


def vdecay_bwd2(P, v, b, do, o, dvhat, dv3, dalpha, scale: float):
    """``dv`` (bf16) and ``dg`` (fp32).  ``o`` and ``do`` both carry ``scale``, so one is taken out (with 0 both are zero)."""
    NC, C, H, M = v.shape
    inv_scale = 1.0 / scale if scale else 0.0
    dv, dg = torch.empty_like(v), torch.empty_like(b)
    _lib.check(_lib.lib().fb_vdecay_bwd2(P.data_ptr(), v.data_ptr(), b.data_ptr(), do.data_ptr(), o.data_ptr(), dvhat.data_ptr(),
                                         dv3.data_ptr(), dalpha.data_ptr(), NC, H, M, inv_scale, dv.data_ptr(), dg.data_ptr(),
                                         _lib.stream_ptr()), "fb_vdecay_bwd2")
    _lib.count_launch()
    return dv, dg


_lib.register("fb_scores_bwd_prep", [c_void_p] * 5 + [c_longlong] * 3 + [c_int] * 4 + [c_void_p, c_void_p, c_void_p])


def scores_bwd_prep(dc: torch.Tensor, out: torch.Tensor, d: torch.Tensor, mask_mode: int):
    """For score blocks ``out = alpha (a b^T) exp(d_i - d_j)`` (masked): returns the bf16 GEMM operand
    ``dc * keep * exp(d_i - d_j)`` and the fp32 gradient of ``d``.  dc, out ``[NC, H, C, C]`` (fp32 or bf16),
    d ``[NC, H, C]`` fp32 with any strides."""
    NC, H, C, _ = out.shape
    dc, out = dc.contiguous(), out.contiguous()
    g = torch.empty(NC, H, C, C, dtype=torch.bfloat16, device=out.device)
    dd = torch.empty(NC, H, C, dtype=torch.float32, device=out.device)
    dc32, dc16 = (dc.data_ptr(), 0) if dc.dtype == torch.float32 else (0, dc.to(torch.bfloat16).data_ptr())
    c32, c16 = (out.data_ptr(), 0) if out.dtype == torch.float32 else (0, out.data_ptr())
    if dc.dtype not in (torch.float32, torch.bfloat16):
        dc = dc.float()
        dc32, dc16 = dc.data_ptr(), 0
    dh, dl, dr = d.stride()
    rc = _lib.lib().fb_scores_bwd_prep(dc32, dc16, c32, c16, d.data_ptr(), dh, dl, dr, NC, H, C, int(mask_mode), g.data_ptr(),
                                       dd.data_ptr(), _lib.stream_ptr())
    _lib.check(rc, "fb_scores_bwd_prep")
    _lib.count_launch()
    return g, dd
