"""Linear layers on the tcgen05 GEMM, with the Megatron-style "main_grad" contract.

If a weight carries a ``main_grad`` attribute (an fp32 view into the sharding engine's flat gradient buffer)
the weight-gradient GEMM accumulates straight into it and autograd sees ``None`` for that weight; otherwise
the gradient is returned to autograd as usual.

``linear_fused(x, [w_q, w_k, w_v])`` runs ONE GEMM when the weights (and their ``main_grad``s) sit back to back
in memory, which is how the engine lays out a block's parameters; the HF-style per-projection parameter names
are kept for checkpoints (fla/layers/attn.py:73-82, fla/modules/mlp.py:58-60 use separate nn.Linear calls).
"""
from __future__ import annotations

from ctypes import c_int, c_longlong, c_void_p
from typing import Optional, Sequence

import torch
import torch.nn.functional as F

from . import _lib, float8, sac, slots
from .gemm import gemm_nn, gemm_nt, gemm_tn


def _adjacent(ts: Sequence[torch.Tensor]) -> bool:
    for a, b in zip(ts[:-1], ts[1:]):
        if a.data_ptr() + a.numel() * a.element_size() != b.data_ptr():
            return False
        if not (a.is_contiguous() and b.is_contiguous()) or a.dtype != b.dtype or a.shape[1:] != b.shape[1:]:
            return False
        if a.untyped_storage().data_ptr() != b.untyped_storage().data_ptr():
            return False
    return True


def _cat_view(ts: Sequence[torch.Tensor]) -> torch.Tensor:
    """Adjacent tensors (``_adjacent``) as one."""
    first, last = ts[0], ts[-1]
    rows = sum(t.shape[0] for t in ts)
    if last.data_ptr() - first.data_ptr() != (rows - last.shape[0]) * first.stride(0) * first.element_size() or \
            first.untyped_storage().data_ptr() != last.untyped_storage().data_ptr():
        raise ValueError("not adjacent in memory")
    return first.as_strided((rows, *first.shape[1:]), first.stride())  # stays within the storage, or raises


def _operands_ok(x: torch.Tensor, w: torch.Tensor) -> bool:
    return _lib.available() and x.is_cuda and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and x.shape[-1] % 8 == 0


def _kernel_ok(x: torch.Tensor, w: torch.Tensor) -> bool:
    return _operands_ok(x, w) and w.shape[0] % 8 == 0


def _matrix(rows: int, cols: int, like: torch.Tensor) -> torch.Tensor:
    """``[rows, cols]`` whose rows are whole 16-byte vectors apart, as the GEMM's operands have to be."""
    return torch.empty(rows, -(-cols // 8) * 8, dtype=like.dtype, device=like.device)[:, :cols]


_lib.register("fb_colsum_bf16_parts", [c_longlong, c_int])
_lib.register("fb_colsum_bf16", [c_void_p, c_longlong, c_longlong, c_int, c_void_p, c_void_p, c_void_p])


def _column_sums(x: torch.Tensor) -> torch.Tensor:
    """fp32 sums over the rows of ``x [T, N]``."""
    T, N = x.shape
    if not (_lib.available() and x.is_cuda and x.dtype == torch.bfloat16 and N % 8 == 0 and N > 0 and x.stride(1) == 1
            and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0):
        return x.sum(0, dtype=torch.float32)
    L = _lib.lib()
    part = torch.empty(L.fb_colsum_bf16_parts(T, N), N, dtype=torch.float32, device=x.device)
    out = torch.empty(N, dtype=torch.float32, device=x.device)
    _lib.check(L.fb_colsum_bf16(x.data_ptr(), x.stride(0), T, N, part.data_ptr(), out.data_ptr(), _lib.stream_ptr()), "fb_colsum_bf16")
    _lib.count_launch(2)
    return out


class _LinearFn(torch.autograd.Function):
    """y = x @ cat(weights).T (+ bias); weights are passed individually so autograd can route their grads."""

    @staticmethod
    def forward(ctx, x, bias, known, *weights):
        """``known``: the output when it is already at hand (the replay pass of operator-level selective activation
        checkpointing, ``ops/sac.py``): nothing is computed, the node only saves what its backward needs."""
        shape = x.shape
        K = shape[-1]
        x2 = x.reshape(-1, K)
        ctx.slot = slots.of(x) if known is None and x.dim() == 2 and x.is_cuda else None
        fused = len(weights) == 1 or _adjacent([w.detach() for w in weights])
        ctx.fp8 = (known is None and fused and bias is None and all(getattr(w, "_fp8", False) for w in weights)
                   and float8.supported(x2) and all(w.shape[0] % 16 == 0 for w in weights))
        # the parameters themselves (not the saved copies): under activation checkpointing the tensors that come back
        # from ``saved_tensors`` are detached recomputations without the ``main_grad`` attribute
        ctx.params = weights
        if known is not None:
            ctx.save_for_backward(x2, *weights)
            ctx.fused, ctx.shape, ctx.has_bias = fused, shape, bias is not None
            return known.view(*shape[:-1], known.shape[-1])
        if ctx.fp8:
            wcat = weights[0].detach() if len(weights) == 1 else _cat_view([w.detach() for w in weights])
            recipe = getattr(weights[0], "_fp8", None)
            ctx.fp8_recipe = recipe if isinstance(recipe, str) else "tensorwise"
            y, saved = float8.float8_linear_forward(x2, wcat, ctx.fp8_recipe)
            ctx.n_fp8_saved = len(saved)
            ctx.save_for_backward(*saved, *weights)
            ctx.fused, ctx.shape, ctx.has_bias = fused, shape, False
            return y.view(*shape[:-1], y.shape[-1])
        if fused:
            wcat = weights[0].detach() if len(weights) == 1 else _cat_view([w.detach() for w in weights])
            y = gemm_nt(x2, wcat, None if wcat.shape[0] % 8 == 0 else _matrix(x2.shape[0], wcat.shape[0], x2), bias=bias)
        else:
            N = sum(w.shape[0] for w in weights)
            y = torch.empty(x2.shape[0], N, dtype=x.dtype, device=x.device)
            c = 0
            for w in weights:
                gemm_nt(x2, w.detach(), out=y[:, c:c + w.shape[0]])
                c += w.shape[0]
            if bias is not None:
                y += bias
        ctx.save_for_backward(x2, *weights)
        ctx.fused, ctx.shape, ctx.has_bias = fused, shape, bias is not None
        return y.view(*shape[:-1], y.shape[-1])

    @staticmethod
    def backward(ctx, dy):
        if ctx.fp8:
            return _LinearFn._backward_fp8(ctx, dy)
        x2, *weights = ctx.saved_tensors
        N = dy.shape[-1]
        dy2 = dy.reshape(-1, N)
        odd = N % 8 != 0 and dy2.is_cuda  # no contiguous matrix of this width is an operand
        if dy2.stride(-1) != 1 or dy2.stride(0) % 8 != 0 or (odd and (dy2.stride(0) < N or dy2.data_ptr() % 16 != 0)):
            dy2 = _matrix(dy2.shape[0], N, dy2).copy_(dy2) if odd else dy2.contiguous()
        K = x2.shape[1]
        dx = None
        if ctx.needs_input_grad[0]:
            if ctx.fused:
                # saved-tensor hooks hand back copies, which lie wherever they were put
                wcat = weights[0] if len(weights) == 1 else _cat_view(weights) if _adjacent(weights) else torch.cat(weights, 0)
                dx = None if ctx.slot is None else ctx.slot.take(x2.shape[0], K, x2.dtype, x2.device)
                if dx is not None and (dx.stride(0) % 8 or dx.data_ptr() % 16 or wcat.shape[0] != N):
                    dx = None
                dx = gemm_nn(dy2, wcat, dx)
            else:
                dx32 = None
                c = 0
                for w in weights:
                    part = gemm_nn(dy2[:, c:c + w.shape[0]], w, out_dtype=torch.float32)
                    dx32 = part if dx32 is None else dx32.add_(part)
                    c += w.shape[0]
                dx = dx32.to(x2.dtype)
            dx = dx.view(ctx.shape)
        grads = [None] * len(weights)
        mgs = [getattr(w, "main_grad", None) for w in ctx.params]
        odd = len(weights) > 1 and any(w.shape[0] % 8 for w in weights)
        if odd and not any(ctx.needs_input_grad[3:]):
            pass  # frozen, as torch's own products of such sizes would leave them
        elif odd and not (all(m is not None for m in mgs) and _adjacent(mgs)):
            # column blocks that start between vectors cannot be operands of their own
            whole = gemm_tn(dy2, x2, out_dtype=torch.float32)
            for i, (part, m) in enumerate(zip(whole.split([w.shape[0] for w in weights]), mgs)):
                if m is not None:
                    m += part
                elif ctx.needs_input_grad[3 + i]:
                    grads[i] = part.to(weights[i].dtype)
        elif all(m is not None for m in mgs):
            if ctx.fused and (len(weights) == 1 or _adjacent(mgs)):
                mg = mgs[0] if len(weights) == 1 else _cat_view(mgs)
                gemm_tn(dy2, x2, out=mg, accumulate=True)
            else:
                c = 0
                for w, m in zip(weights, mgs):
                    gemm_tn(dy2[:, c:c + w.shape[0]], x2, out=m, accumulate=True)
                    c += w.shape[0]
        else:
            c = 0
            for i, w in enumerate(weights):
                if ctx.needs_input_grad[3 + i]:
                    grads[i] = gemm_tn(dy2[:, c:c + w.shape[0]], x2, out_dtype=torch.float32).to(w.dtype)
                c += w.shape[0]
        gb = None
        if ctx.has_bias and ctx.needs_input_grad[1]:
            gb = _column_sums(dy2).to(dy.dtype)
        return (dx, gb, None, *grads)


def _backward_fp8(ctx, dy):
    saved = tuple(ctx.saved_tensors[:ctx.n_fp8_saved])
    weights = list(ctx.saved_tensors[ctx.n_fp8_saved:])
    recipe = ctx.fp8_recipe
    dy2 = dy.reshape(-1, dy.shape[-1])
    need_dx = ctx.needs_input_grad[0]
    mgs = [getattr(w, "main_grad", None) for w in ctx.params]
    grads = [None] * len(weights)
    if all(m is not None for m in mgs) and (len(weights) == 1 or _adjacent(mgs)):
        mg = mgs[0] if len(weights) == 1 else _cat_view(mgs)
        dx, _ = float8.float8_linear_backward(dy2, saved, need_dx, wgrad_out=mg, recipe=recipe)
    else:
        need_dw = any(ctx.needs_input_grad[3:])
        dx, dw = float8.float8_linear_backward(dy2, saved, need_dx, need_dw=need_dw, recipe=recipe)
        c = 0
        for i, (w, m) in enumerate(zip(weights, mgs)):
            if dw is not None:
                part = dw[c:c + w.shape[0]]
                if m is not None:
                    m += part
                elif ctx.needs_input_grad[3 + i]:
                    grads[i] = part.to(w.dtype)
            c += w.shape[0]
    if dx is not None:
        dx = dx.view(ctx.shape)
    return (dx, None, None, *grads)


_LinearFn._backward_fp8 = staticmethod(_backward_fp8)


def _cpu_fp8(x: torch.Tensor, weights: Sequence[torch.Tensor]) -> bool:
    # without CUDA the fp8 path still runs (torch float8 dtypes) so that converted models behave the same everywhere
    return (all(getattr(w, "_fp8", False) for w in weights) and x.shape[-1] % 16 == 0
            and x.numel() // x.shape[-1] % 16 == 0)


def _with_tape(x: torch.Tensor, bias, weights: Sequence[torch.Tensor], compute):
    """Runs ``compute()`` unless a selective-checkpointing tape is active (``ops/sac.py``).  Under a tape both passes go
    through ``_LinearFn`` - with the output computed in the record pass and handed over in the replay pass - because the
    checkpoint machinery requires the recomputation to save the same tensors, in the same order, as the forward."""
    tape = sac.current()
    if tape is None or not torch.is_grad_enabled() or any(getattr(w, "_fp8", False) for w in weights):
        return compute()
    if tape.mode == "record":
        tape.decide("mm")
        y = _LinearFn.apply(x, bias, None, *weights)
        if tape._keep:
            # a private copy: the consumer may rework the output in place (the rotary embedding does, on q and k), and
            # the replay pass must hand back what the GEMM produced
            tape.store(y.detach().clone())
        return y
    return _LinearFn.apply(x, bias, tape.fetch(), *weights)


def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    if _kernel_ok(x, weight) or (bias is None and not x.is_cuda and x.dtype == torch.bfloat16 and _cpu_fp8(x, [weight])):
        return _with_tape(x, bias, [weight], lambda: _LinearFn.apply(x, bias, None, weight))
    return _with_tape(x, bias, [weight], lambda: F.linear(x, weight, bias))


def side_by_side(x: torch.Tensor, weights: Sequence[torch.Tensor]) -> bool:
    """Whether one GEMM may stand for the products of ``x`` with these weights: adjacent in memory (their ``main_grad``s too, or
    none has one), bf16 on the GPU, no fp8 scaling per tensor, no tape that counts products (selective checkpointing)."""
    mgs = [getattr(w, "main_grad", None) for w in weights]
    return (x.dim() == 2 and all(_operands_ok(x, w) and not getattr(w, "_fp8", False) for w in weights) and sac.current() is None
            and _adjacent([w.detach() for w in weights])
            and (all(m is None for m in mgs) or (all(m is not None for m in mgs) and _adjacent(mgs))))


def linear_fused(x: torch.Tensor, weights: Sequence[torch.Tensor]) -> torch.Tensor:
    """``x @ cat(weights, 0).T`` as one ``[..., sum(N_i)]`` tensor."""
    if all(_kernel_ok(x, w) for w in weights) or side_by_side(x, weights):
        return _with_tape(x, None, weights, lambda: _LinearFn.apply(x, None, None, *weights))
    if not x.is_cuda and x.dtype == torch.bfloat16 and _cpu_fp8(x, weights):
        return torch.cat([_LinearFn.apply(x, None, None, w) for w in weights], dim=-1)
    return _with_tape(x, None, weights, lambda: torch.cat([F.linear(x, w) for w in weights], dim=-1))


# --------------------------------------------------------------------------------------------------------------
# SwiGLU in the epilogues of the products around it
# --------------------------------------------------------------------------------------------------------------
_lib.register("fb_gemm2_swiglu", [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_longlong, c_longlong,
                                  c_longlong, c_longlong, c_int, c_void_p])
_lib.register("fb_gemm2_swiglu_bwd", [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_longlong, c_longlong,
                                      c_longlong, c_longlong, c_int, c_void_p])


def _rows(x: torch.Tensor) -> torch.Tensor:
    """``x [..., N]`` as a matrix the GEMM kernels read: rows of whole 16-byte vectors."""
    x = x.reshape(-1, x.shape[-1])
    if x.stride(1) != 1 or x.stride(0) % 8 or x.data_ptr() % 16 or (x.shape[0] > 1 and x.stride(0) < x.shape[1]):
        x = x.clone(memory_format=torch.contiguous_format)
    return x


def _gate_up(x2: torch.Tensor, wg: torch.Tensor, wu: torch.Tensor):
    """``gate | up [T, 2 I]`` and ``z = silu(gate) * up`` from ONE kernel: the GEMM's epilogue holds gate_j and up_j of the same hidden
    index side by side (the two CTAs of a pair load the gate rows and the up rows of the fused weight) and writes both, which the
    backward needs, and the activation."""
    from . import gemm as gemm_ops
    T, K = x2.shape
    I = wg.shape[0]
    wcat = _cat_view([wg.detach(), wu.detach()])
    gu = torch.empty(T, 2 * I, dtype=x2.dtype, device=x2.device)
    z = torch.empty(T, I, dtype=x2.dtype, device=x2.device)
    pend = gemm_ops.pending_gather()
    if pend is not None and not pend.done and pend.touches(wcat):  # a plain product may fetch the weights on its way
        from .activations import swiglu_forward
        return gemm_nt(x2, wcat, gu), swiglu_forward(gu, z)
    rc = _lib.lib().fb_gemm2_swiglu(x2.data_ptr(), wcat.data_ptr(), gu.data_ptr(), z.data_ptr(), T, I, K, x2.stride(0),
                                    wcat.stride(0), gu.stride(0), z.stride(0), gemm_ops._sm_count(x2.device),
                                    _lib.stream_ptr())
    _lib.check(rc, "fb_gemm2_swiglu")
    _lib.count_launch()
    return gu, z


def _gate_up_grads(dgu, x2, wg, wu, params, need, dx=None):
    """Gradients of the input and, unless they went to ``main_grad``, of the two weights; ``need`` as ``needs_input_grad`` of
    (x, gate, up); ``dx``: where the input's gradient is wanted, or None."""
    I = wg.shape[0]
    if need[0]:
        dx = gemm_nn(dgu, _cat_view([wg, wu]) if _adjacent([wg, wu]) else torch.cat([wg, wu], 0), dx)
    mgs = [getattr(w, "main_grad", None) for w in params]
    if all(m is not None for m in mgs) and _adjacent(mgs):
        gemm_tn(dgu, x2, out=_cat_view(mgs), accumulate=True)
        return dx, None, None
    grads = []
    for w, m, d, n in zip(params, mgs, (dgu[:, :I], dgu[:, I:]), need[1:]):
        if m is not None:
            gemm_tn(d, x2, out=m, accumulate=True)
        grads.append(gemm_tn(d, x2, out_dtype=torch.float32).to(w.dtype) if m is None and n else None)
    return (dx, *grads)


class _GateUpSwiGLU(torch.autograd.Function):
    """``z = silu(x @ Wg.T) * (x @ Wu.T)``, see ``_gate_up``; what is left of ``_GatedMLP`` where the down projection is a call of its own."""

    @staticmethod
    def forward(ctx, x, wg, wu):
        shape = x.shape
        x2 = _rows(x)
        gu, z = _gate_up(x2, wg, wu)
        ctx.save_for_backward(x2, gu, wg, wu)
        ctx.params = (wg, wu)
        ctx.shape = shape
        return z.view(*shape[:-1], z.shape[1])

    @staticmethod
    def backward(ctx, dz):
        from .activations import swiglu_backward
        x2, gu, wg, wu = ctx.saved_tensors
        dgu = swiglu_backward(_lib.dense(dz.reshape(-1, wg.shape[0])), _lib.dense(gu))
        dx, gg, gu_ = _gate_up_grads(dgu, x2, wg, wu, ctx.params, ctx.needs_input_grad)
        return None if dx is None else dx.view(ctx.shape), gg, gu_


class _GatedMLP(torch.autograd.Function):
    """``(silu(x @ Wg.T) * (x @ Wu.T)) @ Wd.T`` as one node: the activation is formed in the epilogue of the first product, and its backward
    in the epilogue of the down projection's data gradient, which never goes to memory."""

    @staticmethod
    def forward(ctx, x, wg, wu, wd):
        shape = x.shape
        ctx.slot = slots.of(x) if x.dim() == 2 else None
        x2 = _rows(x)
        gu, z = _gate_up(x2, wg, wu)
        y = gemm_nt(z, wd.detach())
        ctx.save_for_backward(x2, gu, z, wg, wu, wd)
        ctx.params = (wg, wu, wd)
        ctx.shape = shape
        return y.view(*shape[:-1], y.shape[1])

    @staticmethod
    def backward(ctx, dy):
        from . import gemm as gemm_ops
        from .activations import swiglu_backward
        x2, gu, z, wg, wu, wd = ctx.saved_tensors
        T, I, D = z.shape[0], z.shape[1], wd.shape[0]
        need_x, need_g, need_u, need_d = ctx.needs_input_grad
        dy2 = _rows(dy)
        dgu = None
        if need_x or need_g or need_u:
            wd2, gu = _rows(wd), _rows(gu)  # saved-tensor hooks hand back copies, which lie wherever they were put
            pend = gemm_ops.pending_gather()
            if pend is not None and not pend.done and pend.touches(wd2):  # a plain product may fetch the weights on its way
                dgu = swiglu_backward(gemm_nn(dy2, wd2), gu)
            else:
                dgu = torch.empty(T, 2 * I, dtype=gu.dtype, device=gu.device)
                rc = _lib.lib().fb_gemm2_swiglu_bwd(dy2.data_ptr(), wd2.data_ptr(), gu.data_ptr(), dgu.data_ptr(), T, I, D, dy2.stride(0),
                                                    wd2.stride(0), gu.stride(0), dgu.stride(0), gemm_ops._sm_count(gu.device),
                                                    _lib.stream_ptr())
                _lib.check(rc, "fb_gemm2_swiglu_bwd")
                _lib.count_launch()
        gd = None
        mg = getattr(ctx.params[2], "main_grad", None)
        if mg is not None:
            gemm_tn(dy2, z, out=mg, accumulate=True)
        elif need_d:
            gd = gemm_tn(dy2, z, out_dtype=torch.float32).to(wd.dtype)
        if dgu is None:
            return None, None, None, gd
        dx = None
        if need_x:
            dx = None if ctx.slot is None else ctx.slot.take(T, x2.shape[1], x2.dtype, x2.device)
            if dx is not None and (dx.stride(0) % 8 or dx.data_ptr() % 16):
                dx = None
        dx, gg, gu_ = _gate_up_grads(dgu, x2, wg, wu, ctx.params[:2], (need_x, need_g, need_u), dx)
        return None if dx is None else dx.view(ctx.shape), gg, gu_, gd


def _swiglu_epilogue_ok(x: torch.Tensor, wg: torch.Tensor, wu: torch.Tensor) -> bool:
    return (_kernel_ok(x, wg) and _kernel_ok(x, wu) and wg.shape == wu.shape and wg.shape[0] % 128 == 0 and x.numel() > 0
            and not getattr(wg, "_fp8", False) and not getattr(wu, "_fp8", False) and sac.current() is None
            and _adjacent([wg.detach(), wu.detach()]) and wg.data_ptr() % 16 == 0)


def gate_up_swiglu(x: torch.Tensor, wg: torch.Tensor, wu: torch.Tensor) -> Optional[torch.Tensor]:
    """``silu(x @ Wg.T) * (x @ Wu.T)`` from one product (bf16 on the GPU, adjacent weights, I a multiple of 128, no fp8 weights, no
    selective-checkpointing tape, which counts products), for a down projection that does more than a product: a bias, a hook, a
    forward of its own; ``None`` tells the caller to take the two-step path."""
    return _GateUpSwiGLU.apply(x, wg, wu) if _swiglu_epilogue_ok(x, wg, wu) else None


def gated_mlp(x: torch.Tensor, wg: torch.Tensor, wu: torch.Tensor, wd: torch.Tensor) -> Optional[torch.Tensor]:
    """The whole bias-free SwiGLU MLP under the conditions of ``gate_up_swiglu``; ``None`` where they do not hold."""
    if not (_swiglu_epilogue_ok(x, wg, wu) and wd.dtype is torch.bfloat16 and wd.is_cuda and wd.shape[1] == wg.shape[0] and wd.shape[0] % 8 == 0
            and wd.is_contiguous() and wd.data_ptr() % 16 == 0 and not getattr(wd, "_fp8", False)):
        return None
    return _GatedMLP.apply(x, wg, wu, wd)
