"""sm_100a batched GEMM and chunk-algorithm kernels against PyTorch fp32 oracles (needs a B200: ``pytest -m gpu``)."""
import pytest
import torch
import torch.nn.functional as F

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(autouse=True)
def _status_clean():
    from flame_b200.ops import _lib
    _lib.lib()
    _lib.status_clear()
    yield
    torch.cuda.synchronize()
    assert _lib.status() == 0, f"kernel status word {_lib.status():#x}"


def _meta(lens):
    from flame_b200.ops.varlen import VarlenMeta
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    return VarlenMeta.from_cu_seqlens(cu, sum(lens), torch.device(DEV))


def _bf(*shape, s=0.5):
    return (torch.randn(*shape, device=DEV) * s).to(torch.bfloat16)


def _ref(a, b, a_mn, b_mn):
    af = a.float().transpose(-1, -2) if a_mn else a.float()
    bf = b.float() if b_mn else b.float().transpose(-1, -2)
    return af @ bf


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_bgemm_layouts_on_chunk_views(a_mn, b_mn):
    from flame_b200.ops.bgemm import bgemm
    torch.manual_seed(0)
    NC, H, M, N, K = 19, 3, 64, 256, 128
    # operands are permuted views of token-major storage, as the chunk algorithms pass them
    a = _bf(NC, K if a_mn else M, H, M if a_mn else K).permute(0, 2, 1, 3)
    b = _bf(NC, K if b_mn else N, H, N if b_mn else K).permute(0, 2, 1, 3)
    out = bgemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32)
    assert rel_err(out, _ref(a, b, a_mn, b_mn)) < 1e-5 + 3e-3
    out16 = torch.empty(NC, M, H, N, device=DEV, dtype=torch.bfloat16).permute(0, 2, 1, 3)
    bgemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out16, alpha=0.5)
    assert rel_err(out16, 0.5 * _ref(a, b, a_mn, b_mn)) < 1e-2


def test_bgemm_mask_decay_and_state_step():
    from flame_b200.ops.bgemm import MASK_STRICT, MASK_TRIL, bgemm
    torch.manual_seed(1)
    NC, H, dk, dv = 11, 2, 128, 256
    q, k = _bf(NC, 64, H, dk).permute(0, 2, 1, 3), _bf(NC, 64, H, dk).permute(0, 2, 1, 3)
    d = (-torch.rand(NC, 64, H, device=DEV) * 0.3).cumsum(1).permute(0, 2, 1)
    full = (q.float() @ k.float().transpose(-1, -2)) * (d[..., :, None] - d[..., None, :]).exp()
    assert rel_err(bgemm(q, k, decay=d, mask=MASK_TRIL, out_dtype=torch.float32), full.tril()) < 5e-3
    assert rel_err(bgemm(q, k, decay=d, mask=MASK_STRICT, alpha=0.25), 0.25 * full.tril(-1)) < 1e-2
    # state step through index tables: X[c+1] = gamma_c X[c] - M_c X16[c] + X[c+1]
    M = _bf(NC, H, dk, dk, s=0.05)
    Xf = torch.randn(NC + 1, H, dk, dv, device=DEV)
    X16 = Xf.to(torch.bfloat16)
    gam = torch.rand(NC, H, device=DEV)
    idx = torch.tensor([0, 2, 5, 9], device=DEV, dtype=torch.int32)
    i = idx.long()
    want = Xf.clone()
    want[i + 1] = Xf[i + 1] + gam[i][..., None, None] * Xf[i] - M[i].float() @ X16[i].float()
    bgemm(M, X16, b_mn=True, a_index=idx, b_index=idx, out=Xf, c_index=idx, c_offset=1, accumulate=True, cin=Xf,
          cin_index=idx, gamma=gam, alpha=-1.0, out16=X16, out16_index=idx, out16_offset=1, n_hi=len(idx))
    assert rel_err(Xf, want) < 1e-3
    assert rel_err(X16, want) < 1e-2
    # in-place per-document state: state[d] = gamma_c state[d] - M_c X16[c] + add16[c], bf16 copy to X16[c+1]
    docs = torch.tensor([3, 0, 2, 1], device=DEV, dtype=torch.int32)
    state = torch.randn(4, H, dk, dv, device=DEV)
    add = _bf(NC, H, dk, dv)
    X16 = want.to(torch.bfloat16)
    want_state = state.clone()
    want_state[docs.long()] = gam[i][..., None, None] * state[docs.long()] - M[i].float() @ X16[i].float() + add[i].float()
    want16 = X16.clone()
    want16[i + 1] = want_state[docs.long()].to(torch.bfloat16)
    bgemm(M, X16, b_mn=True, a_index=idx, b_index=idx, out=state, c_index=docs, cin=state, cin_index=docs, gamma=gam,
          alpha=-1.0, add16=add, add16_index=idx, out16=X16, out16_index=idx, out16_offset=1, n_hi=len(idx))
    assert rel_err(state, want_state) < 1e-3
    assert rel_err(X16, want16) < 1e-2


@pytest.mark.parametrize("M,N,K,K2", [(16, 48, 128, 64), (64, 64, 64, 72), (64, 128, 128, 64), (128, 136, 256, 16), (130, 264, 64, 200)])
def test_bgemm_sums_of_products(M, N, K, K2):
    """Several products in one accumulator (added and subtracted, every storage sense), a factor per row, a sum over the heads
    of a group; fp32 accumulation of bf16 operands: 1e-5 in fp32, 2^-8 after rounding to bf16."""
    from flame_b200.ops.bgemm import bgemm
    torch.manual_seed(11)
    hi, G, r = 3, 2, 3
    t = lambda *s: torch.randn(*s, device=DEV).to(torch.bfloat16)  # noqa: E731
    pad = lambda n: (n + 7) // 8 * 8  # noqa: E731
    a, b = t(hi, G * r, M, K), t(hi, G, N, K)                       # b is shared by the heads of a group
    a2, b2 = t(hi, G * r, K2, pad(M))[..., :M], t(hi, G * r, K2, pad(N))[..., :N]
    scale = torch.randn(hi, M, G * r, device=DEV).permute(0, 2, 1)
    bx = b.repeat_interleave(r, 1)
    one, two = a.float() @ bx.float().transpose(-1, -2), a2.float().transpose(-1, -2) @ b2.float()
    Np = pad(N)
    out = torch.empty(hi, G * r, M, Np, device=DEV)[..., :N]
    bgemm(a, b, alpha=0.5, out=out, more=[(a2, b2, True, True, -1)], rowscale=scale)
    assert rel_err(out, 0.5 * (one - two) * scale[..., None]) < 1e-5
    out16 = torch.empty(hi, M, G, Np, device=DEV, dtype=torch.bfloat16)[..., :N].permute(0, 2, 1, 3)
    bgemm(a, b, out=out16, sum_lo=r, more=[(a2, b2, True, True, 1)])
    assert rel_err(out16, (one + two).reshape(hi, G, r, M, N).sum(2)) < 4e-3


@pytest.mark.parametrize("gates", ["mild", "hard"])
@pytest.mark.parametrize("dk,dv,lens", [(64, 64, [1, 64, 65]), (72, 40, [15, 17, 48, 200]), (256, 128, [130, 63])])
def test_gla_edges(dk, dv, lens, gates):
    """Head sizes that are no multiple of the kernels' channel tiles, documents around sub-block and chunk edges, gates so hard
    that a re-based exponent would overflow if any were positive; against the fp32 recurrence (bf16 operands: 2e-2)."""
    from flame_b200.ops import linear_attn as la
    from flame_b200.ops.chunked import gla_tc
    torch.manual_seed(12)
    meta = _meta(lens)
    T, H = sum(lens), 3
    leaf = lambda *s: torch.randn(*s, device=DEV, dtype=torch.bfloat16).requires_grad_(True)  # noqa: E731
    q, k, v, graw = leaf(T, H, dk), leaf(T, H, dk), leaf(T, H, dv), leaf(T, H, dk)
    ins = [q, k, v, graw]
    gate = lambda: F.logsigmoid(graw.float() * 2) / 4 if gates == "mild" else -F.softplus(graw.float()) * 20  # noqa: E731
    ref = _run(lambda c: la.gla_recurrent(c(q), c(k), c(v), gate(), meta), ins, True)
    out = _run(lambda c: gla_tc(c(q), c(k), c(v), gate(), meta), ins, False)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 2e-2


@pytest.mark.parametrize("M,dk,lens", [(8, 64, [1, 16, 17]), (64, 72, [63, 65, 130]), (200, 64, [100, 48])])
def test_gsa_edges(M, dk, lens):
    """Slots around the kernels' thread counts, documents around sub-block and chunk edges; the fused pair of passes and the first
    pass alone (the form context parallelism uses) against the fp32 recurrences."""
    from flame_b200.ops import linear_attn as la
    from flame_b200.ops.chunked import gla_vdecay_tc
    from flame_b200.ops.gla import gsa
    torch.manual_seed(13)
    meta = _meta(lens)
    T, H, dv = sum(lens), 2, 64
    leaf = lambda *s: torch.randn(*s, device=DEV, dtype=torch.bfloat16).requires_grad_(True)  # noqa: E731
    q, k, v, sl, graw = leaf(T, H, dk), leaf(T, H, dk), leaf(T, H, dv), leaf(T, H, M), leaf(T, H, M)
    gate = lambda: F.logsigmoid(graw.float()) / 4  # noqa: E731
    ins = [q, k, v, sl, graw]
    ref = _run(lambda c: la.gsa_recurrent(c(q), c(k), c(v), c(sl), gate(), meta, 0.3), ins, True)
    out = _run(lambda c: gsa(c(q), c(k), c(v), c(sl), gate(), meta, 0.3), ins, False)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 4e-2
    ins = [q, k, sl, graw]
    ref = _run(lambda c: la.gla_recurrent_vdecay(c(q), c(k), c(sl), gate(), meta, 0.3), ins, True)
    out = _run(lambda c: gla_vdecay_tc(c(q), c(k), c(sl), gate(), meta, 0.3), ins, False)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 2e-2


@pytest.mark.parametrize("C", [64, 128])
@pytest.mark.parametrize("H", [1, 3])
@pytest.mark.parametrize("form", ["plain", "gated", "shared"])
def test_chunk_stages_read_nothing_above_the_diagonal(C, H, form):
    """The inverse, the gradient through the scaled inverses and that through the scores, against 64 bits, with NaN above the diagonal
    of the scores and their gradients.  bf16 results: rounded once (2^-8 of the result) after fp32 arithmetic with an exponential
    that is good to 2^-20; sums of C fp32 terms: 2^-16 of the sum of their absolutes covers C 2^-24 and the exponential."""
    from flame_b200.ops import chunk_kernels as ck
    from flame_b200.ops.bgemm import bgemm
    torch.manual_seed(C + H)
    NC = 3
    upper = torch.ones(C, C, dtype=torch.bool, device=DEV).triu(1)
    nan = lambda x, m=upper: x.masked_fill(m, float("nan"))  # noqa: E731
    beta = torch.rand(NC, C, H, device=DEV)
    b = None if form == "plain" else (-torch.rand(NC, C, H, device=DEV) * 0.2).cumsum(1).contiguous()
    rows = lambda x: x.double().permute(0, 2, 1)  # noqa: E731
    br, e = rows(beta), torch.ones(NC, H, C, device=DEV).double() if b is None else rows(b).exp()
    P = (torch.randn(NC, H, C, C, device=DEV) * 0.1).tril(-1)
    dA, dQ, Q = torch.randn(NC, H, C, C, device=DEV), _bf(NC, H, C, C), _bf(NC, H, C, C)
    d = (e.log()[..., :, None] - e.log()[..., None, :]).tril().exp().tril()
    dq, q = dQ.double().tril(), Q.double().tril()

    def near(got, want, size, tol):
        assert ((got.double() - want).abs() <= tol * size + 2.0 ** -8 * want.abs() * (got.dtype == torch.bfloat16)).all()

    if form == "shared":  # attention with a decay, no delta rule
        db = torch.ones(NC, C, H, device=DEV)
        near(ck.scores_bwd(nan(dQ), nan(Q), b, db, 0.5), 0.5 * dq * d, dq.abs(), 2.0 ** -20)
        y = dq * q
        near(rows(db), 1 + y.sum(-1) - y.sum(-2), 1 + y.abs().sum(-1) + y.abs().sum(-2), 2.0 ** -16)
        return
    T, Tu, Tw = ck.delta_inverse(nan(P, upper | torch.eye(C, dtype=torch.bool, device=DEV)) if C == 64 else P, beta, b, bgemm)
    eye = torch.eye(C, dtype=torch.float64, device=DEV)
    want = torch.linalg.solve_triangular(eye + br[..., None] * P.double(), eye.expand_as(P).contiguous(), upper=False, unitriangular=True)
    assert not T.triu(1).any() and (T.double() - want).norm() <= (2.0 ** -8 if C == 64 else 2.0 ** -7) * want.norm()
    dTu, dTw = _bf(NC, H, C, C), None if b is None else _bf(NC, H, C, C)
    w = 0 if b is None else dTw.double() * e[..., None, :]
    dT, dbeta, db = ck.delta_bwd_t(T, dTu, dTw, beta, b, 0.5)
    t, both = T.double(), dTu.double() + w
    size = dTu.double().abs() + (0 if b is None else w.abs())
    near(dT, br[..., None, :] * both, size, 2.0 ** -20)
    near(rows(dbeta), 0.5 * (t * both).sum(-2), (t.abs() * size).sum(-2), 2.0 ** -16)
    if b is not None:
        near(rows(db), 0.5 * br * (t * w).sum(-2), (t * w).abs().sum(-2), 2.0 ** -16)
    strict = dA.double().tril(-1)
    y, y2 = strict * P.double(), dq * q if b is not None else torch.zeros_like(q)
    old, oldb = rows(dbeta), None if b is None else rows(db)
    diag = upper | torch.eye(C, dtype=torch.bool, device=DEV)
    g, gq = ck.delta_bwd_scores(nan(dA, diag), nan(P, diag), nan(dQ), nan(Q), beta, b, 0.5, dbeta, db)
    near(g, br[..., None] * strict * d, strict.abs(), 2.0 ** -20)
    near(rows(dbeta), old + 0.5 * y.sum(-1), old.abs() + y.abs().sum(-1), 2.0 ** -16)
    if b is not None:
        near(gq, dq * d, dq.abs(), 2.0 ** -20)
        z = br[..., None] * y + y2
        near(rows(db), oldb + 0.5 * (z.sum(-1) - z.sum(-2)), oldb.abs() + z.abs().sum(-1) + z.abs().sum(-2), 2.0 ** -16)


@pytest.mark.parametrize("C", [64, 128])
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("H", [1, 3])
def test_delta_inverse(C, gated, H):
    """T = (I + diag(beta) P)^-1 and T scaled by beta and by beta e^b, against the definition in fp64.  Solved in fp32 and rounded to
    bf16 (2^-8 of an entry); at C = 128 the lower-left block comes from products of the rounded diagonal blocks and the scaled
    copies from the rounded T: a few more roundings, 2^-7 in the norm."""
    from flame_b200.ops import chunked
    torch.manual_seed(C + H)
    NC = 5
    P = (torch.randn(NC, H, C, C, device=DEV) * 0.1).tril(-1)
    beta = torch.rand(NC, C, H, device=DEV)
    b = (-torch.rand(NC, C, H, device=DEV) * 0.2).cumsum(1).contiguous() if gated else None
    got = chunked._delta_inverse(P, beta, b)
    br = beta.double().permute(0, 2, 1)
    eye = torch.eye(C, dtype=torch.float64, device=DEV)
    T = torch.linalg.solve_triangular(eye + br[..., None] * P.double(), eye.expand_as(P).contiguous(), upper=False, unitriangular=True)
    want = [T, T * br[..., None, :], T * (br * b.double().permute(0, 2, 1).exp())[..., None, :] if gated else None]
    assert (got[2] is None) == (not gated)
    for g, w in zip(got, want):
        if w is not None:
            assert g.dtype == torch.bfloat16 and not g.triu(1).any()
            if C == 64:
                assert ((g.double() - w).abs() <= 2.0 ** -8 * w.abs() + 1e-5).all()
            assert (g.double() - w).norm() <= (2.0 ** -8 if C == 64 else 2.0 ** -7) * w.norm()


def test_l2norm():
    from flame_b200.ops.chunk_kernels import l2norm
    torch.manual_seed(2)
    x = torch.randn(1000, 6, 256, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    y = l2norm(x)
    xf = x.detach().float().requires_grad_(True)
    yr = xf * torch.rsqrt(xf.pow(2).sum(-1, keepdim=True) + 1e-6)
    assert rel_err(y, yr) < 1e-2
    g = torch.randn_like(y)
    y.backward(g)
    yr.backward(g.float())
    assert rel_err(x.grad, xf.grad) < 2e-2


def _run(fn, inputs, f32):
    for t in inputs:
        t.grad = None
    o = fn((lambda x: x.float()) if f32 else (lambda x: x))
    torch.manual_seed(99)
    (o.float() * torch.randn(o.shape, device=DEV)).sum().backward()
    return [o.detach()] + [t.grad.clone() for t in inputs]


LENS = [300, 77, 129, 64, 1000, 1]


@pytest.mark.parametrize("gated,chunk,dk,dv", [(True, 128, 128, 256), (False, 128, 128, 256), (True, 64, 128, 256),
                                                 (True, 128, 256, 128), (False, 64, 128, 128), (True, 64, 64, 64)])
def test_gated_delta_rule_kernels_match_fp32_chunk_reference(gated, chunk, dk, dv):
    """dk 128 / 256 with dv a multiple of 128 walk the chunk states in the persistent scan kernel (csrc/delta_scan.cu);
    the last case takes the one-launch-per-position path."""
    from flame_b200.ops import linear_attn as la
    from flame_b200.ops.chunked import gated_delta_rule_tc
    torch.manual_seed(3)
    meta = _meta(LENS)
    T, H = sum(LENS), 2
    leaf = lambda *s: torch.randn(*s, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    q, k, v, braw, graw = leaf(T, H, dk), leaf(T, H, dk), leaf(T, H, dv), leaf(T, H), leaf(T, H)
    ins = [q, k, v, braw] + ([graw] if gated else [])

    def make(fn):
        def f(c):
            g = -F.softplus(graw.float()) * 0.3 if gated else None
            return fn(la.l2norm(c(q)), la.l2norm(c(k)), c(v), braw.float().sigmoid(), g, meta)
        return f
    ref = _run(make(la.gated_delta_rule_chunk), ins, True)
    out = _run(make(lambda *a: gated_delta_rule_tc(*a, chunk=chunk)), ins, False)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 3e-2


@pytest.mark.parametrize("dk", [128, 256])
@pytest.mark.parametrize("lens", [[64], [128, 1], [192, 65, 64], [700, 64, 129, 2000]])
def test_delta_scan_kernel_equals_the_per_position_launches(dk, lens, monkeypatch):
    """The states entering the chunks and the adjoints of the states leaving them, from the persistent scan kernel and from one
    batched GEMM per chunk position, for documents of one, two, three and many chunks.  Both keep the state in fp32 and feed its
    bf16 rounding to the tensor core; they add its three terms in another order, so that now and then a state is rounded to
    the neighbouring bf16 value (2^-8 of it): 2^-9 in the norm.  Every chunk is written."""
    from flame_b200.ops import _lib, chunked
    torch.manual_seed(5)
    lay = chunked.ChunkLayout(_meta(lens), 64)
    NC, H, dv = lay.NC, 3, 256
    M = (torch.randn(NC, H, dk, dk, device=DEV) * 0.05 * (128 / dk) ** 0.5).to(torch.bfloat16)
    B = torch.randn(NC, H, dk, dv, device=DEV).to(torch.bfloat16)
    alpha = torch.rand(NC, H, device=DEV) * 0.5 + 0.5
    outs = []
    for scan in ("1", "0"):
        monkeypatch.setenv("FLAME_B200_DELTA_SCAN", scan)
        fill = torch.full((NC + 1, H, dk, dv), float("nan"), dtype=torch.bfloat16, device=DEV)   # (for the allocator to hand out)
        del fill
        before = _lib.launches()
        outs.append([chunked._delta_states(M, B, alpha, lay).double(), chunked._delta_adjoint(M, B, alpha, lay).double()])
        assert scan == "0" or _lib.launches() - before == 2
    _lib.assert_status_ok()
    first, last = lay.first.tolist(), lay.last.tolist()
    for got, want, ends in zip(*outs, (first, last)):
        assert torch.isfinite(got).all() and not got[ends].any() and not want[ends].any()
        assert (got - want).norm() <= 2.0 ** -9 * want.norm().clamp_min(1e-30)


def test_scalar_gla_and_gla_kernels_match_fp32_references():
    from flame_b200.ops import linear_attn as la
    from flame_b200.ops.chunked import gla_tc, scalar_gla_tc
    torch.manual_seed(4)
    meta = _meta(LENS)
    T, H, dk, dv = sum(LENS), 2, 128, 128
    leaf = lambda *s: torch.randn(*s, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    q, k, v, graw, gk = leaf(T, H, dk), leaf(T, H, dk), leaf(T, H, dv), leaf(T, H), leaf(T, H, dk)
    ins = [q, k, v, graw]
    ref = _run(lambda c: la.scalar_gla_chunk(c(q), c(k), c(v), -F.softplus(graw.float()) * 0.3, meta, 0.1), ins, True)
    out = _run(lambda c: scalar_gla_tc(c(q), c(k), c(v), -F.softplus(graw.float()) * 0.3, meta, 0.1), ins, False)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 3e-2
    ins = [q, k, v, gk]
    ref = _run(lambda c: la.gla_chunk(c(q), c(k), c(v), F.logsigmoid(gk.float() * 4), meta), ins, True)
    out = _run(lambda c: gla_tc(c(q), c(k), c(v), F.logsigmoid(gk.float() * 4), meta), ins, False)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 3e-2


def test_selective_scan_kernels_match_recurrence():
    from flame_b200.ops import linear_attn as la
    from flame_b200.ops.scan import selective_scan
    torch.manual_seed(5)
    lens = [70, 1, 64, 130, 17, 300]
    meta = _meta(lens)
    T, Di, N = sum(lens), 96, 16
    u = torch.randn(T, Di, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    draw = torch.randn(T, Di, device=DEV).requires_grad_(True)
    Alog = torch.log(torch.arange(1, N + 1, device=DEV, dtype=torch.float32))[None].repeat(Di, 1).requires_grad_(True)
    B = torch.randn(T, N, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    C = torch.randn(T, N, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    D = torch.randn(Di, device=DEV).requires_grad_(True)
    ins = [u, draw, Alog, B, C, D]

    def run(fn, f32):
        for t in ins:
            t.grad = None
        c = (lambda x: x.float()) if f32 else (lambda x: x)
        y = fn(c(u), F.softplus(draw) * 0.5, -torch.exp(Alog), c(B), c(C), D, meta)
        torch.manual_seed(7)
        (y.float() * torch.randn(y.shape, device=DEV)).sum().backward()
        return [y.detach()] + [t.grad.clone() for t in ins]
    ref = run(la.selective_scan_recurrent, True)
    out = run(selective_scan, False)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 2e-2


@pytest.mark.parametrize("Di,lens", [(2, [1]), (70, [15, 16, 17]), (129, [31, 33, 1, 48]), (130, [63, 64, 65, 2]), (192, [200, 127, 49])])
@pytest.mark.parametrize("gate", [False, True])
def test_selective_scan_edges(Di, lens, gate):
    """Channel counts and documents around the blocks' edges, operands as strided columns of a projection, with and without
    the layer's softplus and gate, against the token-by-token recurrence in fp64.  Operands and results are bf16 (2^-9 of
    rounding each, sums over 16 states and up to 300 steps of same-sized terms): 1e-2."""
    from flame_b200.ops.scan import mamba_scan_gate, selective_scan
    torch.manual_seed(6)
    meta = _meta(lens)
    T, N, R = sum(lens), 16, 3
    wide = lambda n: torch.randn(T, n, device=DEV, dtype=torch.bfloat16).requires_grad_(True)  # noqa: E731
    uz, ssm, raw = wide(2 * Di), wide(R + 2 * N), wide(Di)
    Alog = torch.log(torch.rand(Di, N, device=DEV) * 8 + 0.1).requires_grad_(True)
    D = torch.randn(Di, device=DEV).requires_grad_(True)
    ins = [uz, ssm, raw, Alog, D]
    dy = torch.randn(T, Di, device=DEV, dtype=torch.bfloat16)

    def grads(y):
        return [y.detach()] + list(torch.autograd.grad(y, ins, dy.to(y.dtype), retain_graph=True))
    A = -torch.exp(Alog)
    cols = lambda c: (c(uz)[:, :Di], c(ssm)[:, R:R + N], c(ssm)[:, R + N:], c(uz)[:, Di:])  # noqa: E731
    u, B, C, z = cols(lambda t: t)
    if gate:
        out = grads(mamba_scan_gate(u, raw, A, B, C, D, z, meta))
    else:
        out = grads(selective_scan(u, F.softplus(raw.float()), A, B, C, D, meta) + 0 * z)
    u, B, C, z = cols(lambda t: t.double())
    h, rows = None, []
    dl = F.softplus(raw.double())
    starts = set(meta.cu_cpu().tolist())
    for t in range(T):
        h = torch.zeros(Di, N, device=DEV, dtype=torch.float64) if t in starts else h
        h = h * (dl[t][:, None] * A.double()).exp() + (dl[t] * u[t])[:, None] * B[t][None]
        rows.append((h * C[t][None]).sum(-1) + D.double() * u[t])
    y = torch.stack(rows)
    ref = grads(y * F.silu(z) if gate else y + 0 * z)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 1e-2


def test_selective_scan_gate_and_softplus_far_out():
    """Arguments where the sigmoids and the softplus saturate, underflow or vanish: finite results that match fp64 to 2^-7 of the largest value of
    their kind (bf16 results of single steps)."""
    from flame_b200.ops.scan import mamba_scan_gate
    torch.manual_seed(8)
    T, Di = 40, 130
    meta = _meta([T])
    far = torch.tensor([-300., -100., -88., -40., -10., -1e-3, 0., 1e-3, 10., 40., 88., 100., 300.], device=DEV)
    pick = lambda: far[torch.randint(len(far), (T, Di), device=DEV)].to(torch.bfloat16).requires_grad_(True)  # noqa: E731
    raw, z = pick(), pick()
    u, B, C = (torch.randn(T, n, device=DEV, dtype=torch.bfloat16).requires_grad_(True) for n in (Di, 16, 16))
    A, D = (-torch.rand(Di, 16, device=DEV)).requires_grad_(True), torch.randn(Di, device=DEV).requires_grad_(True)
    ins, dy = [u, raw, B, C, z, A, D], torch.randn(T, Di, device=DEV, dtype=torch.bfloat16)
    y = mamba_scan_gate(u, raw, A, B, C, D, z, meta)
    got = [y.detach()] + list(torch.autograd.grad(y, ins, dy))
    ud, rd, Bd, Cd, zd, Ad, Dd = ref_in = [t.detach().double().requires_grad_(True) for t in ins]
    h, rows, dl = torch.zeros(Di, 16, device=DEV, dtype=torch.float64), [], F.softplus(rd)
    for t in range(T):
        h = h * (dl[t][:, None] * Ad).exp() + (dl[t] * ud[t])[:, None] * Bd[t][None]
        rows.append((h * Cd[t][None]).sum(-1) + Dd * ud[t])
    yr = torch.stack(rows) * F.silu(zd)
    for a, b in zip(got, [yr.detach()] + list(torch.autograd.grad(yr, ref_in, dy.double()))):
        assert torch.isfinite(a).all()
        assert float((a.double() - b).abs().max()) < 2 ** -7 * float(b.abs().max())


@pytest.mark.parametrize("gate", [False, True])
def test_selective_scan_without_a_backward_keeps_one_state_a_chunk(gate):
    """Same output with gradients off, in the memory of the output, one fp32 state and one sum of steps per chunk (and 4 MB),
    also where a parameter would want a gradient."""
    from flame_b200.ops.scan import mamba_scan_gate, selective_scan
    torch.manual_seed(3)
    lens = [1000, 64, 2999, 33]
    meta, T, Di = _meta(lens), sum(lens), 1100
    u, raw, z = (_bf(T, Di) for _ in range(3))
    B, C = _bf(T, 16), _bf(T, 16)
    A, D = -torch.rand(Di, 16, device=DEV), torch.randn(Di, device=DEV).requires_grad_(True)
    delta = F.softplus(raw.float())
    fn = (lambda: mamba_scan_gate(u, raw, A, B, C, D, z, meta)) if gate else (lambda: selective_scan(u, delta, A, B, C, D, meta))
    want = fn().detach()
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    with torch.no_grad():
        got = fn()
    used = torch.cuda.max_memory_allocated() - before
    assert torch.equal(got, want)
    chunks, padded = sum((n + 63) // 64 for n in lens), (Di + 127) // 128 * 128
    assert used <= 2 * T * Di + 4 * chunks * padded * 17 + (4 << 20)


def test_gsa_kernels_match_fp32_chunk_reference():
    from flame_b200.ops import linear_attn as la
    from flame_b200.ops.gla import gsa
    torch.manual_seed(6)
    meta = _meta(LENS)
    T, H, dk, M, dv = sum(LENS), 2, 128, 64, 128
    leaf = lambda *s: torch.randn(*s, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    q, k, v, sl, graw = leaf(T, H, dk), leaf(T, H, dk), leaf(T, H, dv), leaf(T, H, M), leaf(T, H, M)
    ins = [q, k, v, sl, graw]
    ref = _run(lambda c: la.gsa_chunk(c(q), c(k), c(v), c(sl), F.logsigmoid(graw.float()) / 8, meta), ins, True)
    out = _run(lambda c: gsa(c(q), c(k), c(v), c(sl), F.logsigmoid(graw.float()) / 8, meta), ins, False)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 4e-2


def test_value_decay_with_scale_zero():
    """A scale of 0 (a read-out switched off) is a number like any other: zeros and a uniform softmax, zero gradients behind them."""
    from flame_b200.ops.chunked import gla_vdecay_tc
    from flame_b200.ops.gla import gsa
    torch.manual_seed(11)
    meta, T = _meta([77, 64]), 141
    q, k, v = (_bf(T, 2, 64).requires_grad_(True) for _ in range(3))
    g = (-torch.rand(T, 2, 64, device=DEV)).requires_grad_(True)
    o = gla_vdecay_tc(q, k, v, g, meta, 0.0)
    for t in (o.detach(), *torch.autograd.grad(o, [q, k, v, g], torch.randn_like(o))):
        assert torch.equal(t, torch.zeros_like(t))
    s = torch.rand(T, 2, 64, device=DEV).requires_grad_(True)
    o = gsa(q, k, v, s, g, meta, scale=0.0)
    dq, dk, ds = torch.autograd.grad(o, [q, k, s], torch.randn_like(o))
    assert torch.equal(dq, torch.zeros_like(dq)) and torch.equal(dk, torch.zeros_like(dk)) and bool(torch.isfinite(ds).all()) and ds.abs().max() > 0


def test_gsa_slot_gradients_are_added_in_fp32():
    """Both passes read the slots in bf16; for slots in fp32 their gradient is the fp32 sum of the passes' two bf16 gradients, so
    most of its entries are no bf16 values, and one pass' share of it is."""
    from flame_b200.ops.chunked import _TwoReaders
    from flame_b200.ops.gla import gsa
    torch.manual_seed(7)
    meta, T = _meta([300, 77]), 377
    q, k, v = (_bf(T, 2, 64, s=1.0) for _ in range(3))
    s, g = torch.rand(T, 2, 32, device=DEV).requires_grad_(True), -torch.rand(T, 2, 32, device=DEV) * 0.1
    o = gsa(q, k, v, s, g, meta)
    ds, = torch.autograd.grad(o, s, torch.randn_like(o))
    assert ds.dtype == torch.float32 and (ds == ds.bfloat16().float()).float().mean() < 0.9
    for n in (1, 7, 8, 9, 1000, 2048, 2051):
        x = torch.rand(n, device=DEV).requires_grad_(True)
        a, b = _TwoReaders.apply(x, torch.bfloat16)
        assert torch.equal(a, x.bfloat16()) and torch.equal(b, a)
        da, db = _bf(n), _bf(n + 1, s=1e-3)[1:]
        dx, = torch.autograd.grad([a, b], x, [da, db], retain_graph=True)
        assert torch.equal(dx, da.float() + db.float())
        dx, = torch.autograd.grad(b, x, db)
        assert torch.equal(dx, db.float())


def test_mamba2_ssd_grouped_heads_match_recurrence():
    from flame_b200.ops import linear_attn as la
    from flame_b200.ops.scan import mamba2_ssd
    torch.manual_seed(8)
    lens = [70, 1, 64, 130, 17, 200]
    meta = _meta(lens)
    T, H, P, N, G = sum(lens), 8, 64, 128, 2
    leaf = lambda *s: torch.randn(*s, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    x, dtraw, B, C = leaf(T, H, P), leaf(T, H), leaf(T, G, N), leaf(T, G, N)
    A = -torch.rand(H, device=DEV) * 2 - 0.5
    D = torch.randn(H, device=DEV)
    ins = [x, dtraw, B, C]
    ref = _run(lambda c: la.mamba2_ssd_recurrent(c(x), F.softplus(dtraw.float()) * 0.3, A, c(B) * 0.2, c(C) * 0.2, D, meta), ins, True)
    out = _run(lambda c: mamba2_ssd(c(x), F.softplus(dtraw.float()) * 0.3, A, c(B) * 0.2, c(C) * 0.2, D, meta), ins, False)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 3e-2


@pytest.mark.parametrize("M", [16, 40, 64, 72, 128, 200])
@pytest.mark.parametrize("N", [8, 24, 64, 72, 128, 136])
def test_bgemm_result_boxes(M, N):
    """Results that leave by TMA, at the edges of the boxes (32 rows, 64 or 32 columns), in padded and token-major storage whose
    neighbours stay untouched; against fp64.  Sums of K = 72 products of bf16 values in fp32: bf16 rounding of the result (2^-9
    relative) and of the addend's sum, plus 72 fp32 roundings of the absolute sum."""
    from flame_b200.ops.bgemm import MASK_STRICT, MASK_TRIL, bgemm
    torch.manual_seed(M * 1000 + N)
    dev = torch.device("cuda", 0)
    hi, lo, K = 5, 3, 72
    a, b = torch.randn(hi, lo, M, K, device=dev).bfloat16(), torch.randn(hi, lo, N, K, device=dev).bfloat16()
    scale = torch.rand(hi, lo, M, device=dev) + 0.5
    full = torch.einsum("hlmk,hlnk->hlmn", a.double(), b.double())
    size = torch.einsum("hlmk,hlnk->hlmn", a.double().abs(), b.double().abs())
    pad = (N + 7) // 8 * 8 + 8

    def check(got, want, rounding):
        assert ((got.double() - want).abs() <= rounding * want.abs() + 2.0 ** -17 * size + 1e-30).all()

    for token_major in (False, True):
        for dtype in (torch.bfloat16, torch.float32):
            shape = (hi + 1, M + 1, lo, pad) if token_major else (hi + 1, lo, M + 1, pad)
            store = torch.full(shape, 7.0, dtype=dtype, device=dev)
            view = store.permute(0, 2, 1, 3) if token_major else store
            out = view[1:, :, :M, :N]
            eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
            bgemm(a, b, out=out, alpha=0.5, rowscale=scale)
            want = 0.5 * full * scale.double()[..., None]
            check(out, want, eps)
            if dtype == torch.float32:
                bgemm(a, b, out=out, accumulate=True)
                check(out, want + full, eps)
            else:
                add = torch.randn(hi, lo, M, pad, device=dev).bfloat16()[..., :N]
                bgemm(a, b, out=out, add16=add)
                check(out, full + add.double(), eps)
                before = out.double()
                bgemm(a, b, out=out, add16=out)   # in place
                check(out, full + before, eps)
            if M == N:
                for mode, want in ((MASK_TRIL, full.tril()), (MASK_STRICT, full.tril(-1))):
                    bgemm(a, b, out=out, mask=mode)
                    check(out, want, eps)
            mask = torch.ones(view.shape, dtype=torch.bool, device=dev)
            mask[1:, :, :M, :N] = False
            assert (view[mask] == 7.0).all()


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("rows,cols,Ha,Hb,per_row", [(64, 64, 2, 2, True), (128, 64, 1, 6, False), (128, 192, 3, 3, True), (64, 320, 2, 1, False),
                                                     (32, 64, 2, 2, True)])
def test_decay_states_in_one_kernel(rows, cols, Ha, Hb, per_row, reverse):
    """Increments and states of documents of one to nine chunks against the loop in fp64, heads shared on either side, operands as strided
    blocks, one that lies between vectors, and a size that goes through product and scan.  fp32 sums of 64 products a chunk, a decay each
    chunk, one rounding of the state (2^-9); the increments of (32, 64) going backwards are rounded too."""
    from flame_b200.ops.chunked import ChunkLayout, _decay_states
    torch.manual_seed(rows + cols)
    lens, H = [1, 64, 65, 570], max(Ha, Hb)
    lay = ChunkLayout(_meta(lens))
    alpha = torch.rand(lay.NC, H, rows, device=DEV) if per_row else torch.rand(lay.NC, H, device=DEV)
    wide = torch.randn(lay.NC, 64, Ha, rows + 8, device=DEV, dtype=torch.bfloat16)
    a = wide[..., 8:].permute(0, 2, 1, 3)
    odd = torch.randn(lay.NC * 64 * Hb * cols + 1, device=DEV, dtype=torch.bfloat16)
    for b in (odd[:-1].view(lay.NC, 64, Hb, cols).permute(0, 2, 1, 3), odd[1:].view(lay.NC, Hb, 64, cols))[:1 if rows == 32 else 2]:
        got = _decay_states(lay, alpha, a, b, reverse)
        x = torch.einsum("nhtr,nhtc->nhrc", a.double().repeat_interleave(H // Ha, 1), b.double().repeat_interleave(H // Hb, 1))
        want, c = torch.zeros(lay.NC, H, rows, cols, dtype=torch.float64, device=DEV), 0
        al = alpha.double()[..., None] if per_row else alpha.double()[..., None, None]
        for n in lens:
            k = (n + 63) // 64
            s = torch.zeros(H, rows, cols, dtype=torch.float64, device=DEV)
            for i in (range(c + k - 1, c - 1, -1) if reverse else range(c, c + k)):
                want[i] = s
                s = al[i] * s + x[i]
            c += k
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + (0.2 if reverse and rows == 32 else 1e-4)).all()
        if reverse:  # the decay's gradient on the way: fp32 sums of products of two bf16 states
            S = torch.randn(lay.NC, H, rows, cols, device=DEV, dtype=torch.bfloat16)
            again, dot = _decay_states(lay, alpha, a, b, reverse, S)
            terms = got.double() * S.double()
            dims = (-1,) if per_row else (-1, -2)
            assert torch.equal(again, got) and dot.shape == alpha.shape
            assert ((dot.double() - terms.sum(dims)).abs() <= 2.0 ** -18 * terms.abs().sum(dims)).all()


@pytest.mark.parametrize("lens", [[3900], [70, 3900, 1], [65] * 60])
def test_decay_states_both_ways_of_forming_them(lens, monkeypatch):
    """A long document, which the rule leaves to product and scan, and many short ones, which it gives to the one kernel, each formed in both
    ways against the loop in fp64: states rounded once (2^-8) after fp32 sums of at most 3,900 terms (1e-3), where the increments are
    rounded too (product and scan backwards) by as much again, each at its own size; the decay's gradient: sums of products of two bf16 states."""
    from flame_b200.ops import chunked
    torch.manual_seed(5)
    H, R, W = 2, 64, 128
    lay = chunked.ChunkLayout(_meta(lens))
    alpha = torch.rand(lay.NC, H, R, device=DEV)
    a, b = _bf(lay.NC, H, 64, R), _bf(lay.NC, H, 64, W)
    S = _bf(lay.NC, H, R, W)
    assert [chunked._walk_pays(lay, H * R * W, g) for g in (False, True)] == [len(lens) == 60] * 2
    x = a.double().transpose(-1, -2) @ b.double()
    one_kernel, other = ((0.0, 1.0, 1.0),) * 2, ((1.0, 0.0, 0.0),) * 2
    for reverse in (False, True):
        want, size, c = torch.zeros_like(x), torch.zeros_like(x), 0
        for n in lens:
            k, s, z = (n + 63) // 64, torch.zeros_like(x[0]), torch.zeros_like(x[0])
            for i in (range(c + k - 1, c - 1, -1) if reverse else range(c, c + k)):
                want[i], size[i] = s, z
                s, z = alpha[i].double()[..., None] * s + x[i], alpha[i].double()[..., None] * z + x[i].abs()
            c += k
        for rule in (one_kernel, other):
            monkeypatch.setattr(chunked, "WALK_US", rule)
            got = chunked._decay_states(lay, alpha, a, b, reverse)
            rounded = 2.0 ** -8 * size if rule is other and reverse else 0
            assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + rounded + 1e-3).all()
            again, dot = chunked._decay_states(lay, alpha, a, b, reverse, S)
            terms = got.double() * S.double()
            assert torch.equal(again, got) and ((dot.double() - terms.sum(-1)).abs() <= 2.0 ** -18 * terms.abs().sum(-1)).all()


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("x16", [False, True])
@pytest.mark.parametrize("rows,cols,per_row", [(3, 12, True), (4, 8, False), (16, 72, True)])
def test_state_scan_widths(rows, cols, per_row, x16, reverse):
    """Chunk-state recurrence with 16-byte and with 8-byte accesses, documents of one to nine chunks, against the loop in fp64:
    fp32 accumulation (a few 2^-24 per step) and one rounding of the state to bf16 (2^-9)."""
    from flame_b200.ops.chunked import ChunkLayout, _state_scan
    torch.manual_seed(rows * cols)
    lens, H = [1, 64, 65, 570], 2
    lay = ChunkLayout(_meta(lens))
    X = torch.randn(lay.NC, H, rows, cols, device=DEV).to(torch.bfloat16 if x16 else torch.float32)
    alpha = torch.rand(lay.NC, H, rows, device=DEV) if per_row else torch.rand(lay.NC, H, device=DEV)
    got = _state_scan(lay, alpha, X, torch.bfloat16, reverse=reverse)
    want, c = torch.zeros(lay.NC, H, rows, cols, dtype=torch.float64, device=DEV), 0
    a = alpha.double()[..., None] if per_row else alpha.double()[..., None, None]
    for n in lens:
        k = (n + 63) // 64
        s = torch.zeros(H, rows, cols, dtype=torch.float64, device=DEV)
        for i in (range(c + k - 1, c - 1, -1) if reverse else range(c, c + k)):
            want[i] = s
            s = a[i] * s + X[i].double()
        c += k
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()


def _shifted(t, offset):
    """The same values in a contiguous tensor that starts ``offset`` elements into its storage."""
    base = torch.empty(t.numel() + offset, dtype=t.dtype, device=t.device)
    return base[offset:].view(t.shape).copy_(t)


@pytest.mark.parametrize("offset", [1, 2, 4])
@pytest.mark.parametrize("name", ["gla", "gsa", "vdecay", "grouped", "gated", "plain_delta"])
def test_contiguous_operands_at_any_storage_offset(name, offset):
    """Whole chunks are handed on as they lie, so an operand (or the output's gradient) may be contiguous and yet start off a
    16-byte boundary: it is moved before a kernel loads it in vectors, and the result is the aligned call's bit for bit (the
    gated delta rule's decay gradient: up to the order of the 64 x 8 partial sums of a chunk that a shared-memory atomic adds)."""
    from flame_b200.ops import chunked
    from flame_b200.ops.gla import gsa
    torch.manual_seed(offset)
    meta, T, H = _meta([128, 64]), 192, 2
    u = lambda *s: torch.randn(*s, device=DEV)  # noqa: E731
    q, k, v = (u(T, 1 if name == "grouped" and i < 2 else H, 64).bfloat16() for i in range(3))
    per_head, per_key = -torch.rand(T, H, device=DEV) * 0.1, -torch.rand(T, H, 64, device=DEV) * 0.1
    ins, fn = {
        "gla": ([q, k, v, per_key], lambda q, k, v, g: chunked.gla_tc(q, k, v, g, meta)),
        "gsa": ([q, k, v, torch.rand(T, H, 64, device=DEV), per_key], lambda q, k, v, s, g: gsa(q, k, v, s, g, meta)),
        "vdecay": ([q, k, v, per_key], lambda q, k, v, g: chunked.gla_vdecay_tc(q, k, v, g, meta, 0.5)),
        "grouped": ([q, k, v, per_head], lambda q, k, v, g: chunked.scalar_gla_tc(q, k, v, g, meta, 0.5)),
        "gated": ([q * 0.1, k * 0.1, v, torch.rand(T, H, device=DEV), per_head], lambda q, k, v, b, g: chunked.gated_delta_rule_tc(q, k, v, b, g, meta)),
        "plain_delta": ([q * 0.1, k * 0.1, v, torch.rand(T, H, device=DEV)], lambda q, k, v, b: chunked.gated_delta_rule_tc(q, k, v, b, None, meta)),
    }[name]
    dy = u(T, H, 64)
    res = []
    for move in (lambda t: t, lambda t: _shifted(t, offset)):
        args = [move(t).requires_grad_(True) for t in ins]
        y = fn(*args)
        res.append([y.detach(), *torch.autograd.grad(y, args, move(dy.to(y.dtype)))])
    for i, (a, b) in enumerate(zip(*res)):
        if name == "gated" and i == 5:
            assert (a - b).abs().max() <= 512 * 2.0 ** -24 * a.abs().max()
        else:
            assert torch.equal(a, b), i


@pytest.mark.parametrize("dk,dv,H", [(128, 128, 2), (64, 72, 1), (40, 64, 3), (136, 256, 1)])
@pytest.mark.parametrize("lens", [[1], [64, 128], [15, 17, 63, 65, 1, 200], [300, 16, 33]])
def test_gla_reads_and_writes_packed_tokens(dk, dv, H, lens):
    """q, k and the gate's argument read as column blocks of one matrix, their gradients written there, against the form with separate
    operands and the gate formed outside.  Both form the same fp32 gates and products; what may differ is a bf16 rounding of a
    re-ordered sum: 5e-3."""
    from flame_b200.ops.chunked import gla_raw_gate, gla_tc
    from flame_b200.ops.gates import logsigmoid_gate
    from flame_b200.ops.slots import reshaped, split_columns
    torch.manual_seed(dk + len(lens))
    meta, T = _meta(lens), sum(lens)
    sizes = (H * dk, H * dk, H * dv, 8)
    wide0, raw0 = _bf(T, sum(sizes)), _bf(T, H, dk, s=3.0)
    dy, res = _bf(T, H, dv), []
    for new in (True, False):
        wide, raw = wide0.clone().requires_grad_(True), raw0.clone().requires_grad_(True)
        if new:
            q, k, v, _ = split_columns(wide, sizes)
            q, k, v = reshaped(q, T, H, dk), reshaped(k, T, H, dk), reshaped(v, T, H, dv)
            o, lay = gla_raw_gate(q, k, v, raw, 16, meta)
            o = lay.unpack(o)
        else:
            q, k, v, _ = (t.contiguous() for t in wide.split(sizes, 1))
            o = gla_tc(q.view(T, H, dk), k.view(T, H, dk), v.view(T, H, dv), logsigmoid_gate(raw, 16), meta)
        o.backward(dy)
        res.append((o.detach(), wide.grad, raw.grad))
    assert (res[0][1][:, -8:] == 0).all()
    for a, b in zip(*res):
        assert rel_err(a, b) < 5e-3


@pytest.mark.parametrize("rows,cols,wide", [(1, 8, 8), (33, 264, 272), (5000, 512, 512), (70000, 40, 48)])
def test_column_sums(rows, cols, wide):
    """fp32 column sums of a bf16 matrix, also a block of a wider one, against fp64: n 2^-24 relative to the terms, 1e-4."""
    from flame_b200.ops.linear import _column_sums
    x = _bf(rows, wide)[:, :cols]
    assert rel_err(_column_sums(x), x.double().sum(0)) < 1e-4


@pytest.mark.parametrize("lens", [[1], [64, 128], [15, 17, 63, 65, 1, 200]])
@pytest.mark.parametrize("sizes", [(8,), (24, 8, 64), (512, 512, 512)])
def test_silu_into_and_out_of_chunk_rows(lens, sizes):
    """SiLU of column blocks into the chunk layout, and out of it, against fp64: bf16 results rounded once (2^-8); zeros in the padding
    both ways, whatever gradient comes from there."""
    from flame_b200.ops.activations import silu_blocks_to_chunks, silu_out_of_chunks
    from flame_b200.ops.chunked import ChunkLayout
    torch.manual_seed(len(lens))
    T, lay, n = sum(lens), ChunkLayout.of(_meta(lens), 64), sum(sizes)
    wide = _bf(T, n + 16, s=3.0).requires_grad_(True)
    ys = silu_blocks_to_chunks(wide[:, 8:8 + n], sizes, lay)
    dys = [_bf(lay.Tp, m) for m in sizes]
    pad = lay.inv_i32 < 0
    torch.autograd.backward(ys, [d.masked_fill(pad[:, None], 5e3) for d in dys])
    xr = wide.detach()[:, 8:8 + n].double().requires_grad_(True)
    want = F.silu(xr)
    want.backward(torch.cat(dys, 1)[lay.rows].double())
    assert rel_err(torch.cat(ys, 1)[lay.rows], want) < 4e-3 and rel_err(wide.grad[:, 8:8 + n], xr.grad) < 4e-3
    assert all(float(y[pad].abs().sum()) == 0 for y in ys)
    o = _bf(lay.Tp, sizes[0], s=3.0).requires_grad_(True)
    y, dy = silu_out_of_chunks(o.view(lay.NC, 64, -1), lay), _bf(T, sizes[0])
    y.backward(dy)
    orr = o.detach()[lay.rows].double().requires_grad_(True)
    F.silu(orr).backward(dy.double())
    assert rel_err(y, F.silu(orr)) < 4e-3 and rel_err(o.grad[lay.rows], orr.grad) < 4e-3 and float(o.grad[pad].abs().sum()) == 0


@pytest.mark.parametrize("slots", [False, True])
@pytest.mark.parametrize("lens", [[1], [64, 128], [15, 17, 63, 65, 1, 200]])
def test_logsigmoid_gate_of_a_block_in_chunk_rows(lens, slots):
    """The gate of a column block, in the chunk layout: bit for bit what the contiguous form gives, packed; the gradient too."""
    from flame_b200.ops.chunked import ChunkLayout
    from flame_b200.ops.gates import logsigmoid_gate
    T, lay = sum(lens), ChunkLayout.of(_meta(lens), 64)
    wide, out = _bf(T, 40, s=3.0), []
    ds = [torch.randn(lay.NC, 64, 2, 8, device=DEV) for _ in range(1 + slots)]
    for new in (True, False):
        w = wide.clone().requires_grad_(True)
        x = w[:, 16:32].view(T, 2, 8)
        if new:
            g = logsigmoid_gate(x, 8, slots, lay)
        else:
            g = logsigmoid_gate(x.contiguous(), 8, slots)
            g = tuple(lay.pack(t) for t in g) if slots else lay.pack(g)
        g = g if slots else (g,)
        torch.autograd.backward(g, ds)
        out.append((*g, w.grad))
    assert all(torch.equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("P", [64, 128])
@pytest.mark.parametrize("lens", [[1], [64, 128], [15, 17, 63, 65, 1, 200]])
def test_mamba2_elementwise_kernels_in_chunk_rows(lens, P):
    """What stands around the SSD core, its operands in padded rows (the padding's values are zero, as the convolution leaves them): bit for
    bit what the same kernels give per token, sums over the tokens in fp32 to 1e-5; the gradient of y is zero in the padding."""
    from flame_b200.ops.chunked import ChunkLayout
    from flame_b200.ops.gates import mamba2_post, mamba2_pre
    torch.manual_seed(P)
    T, H, lay = sum(lens), 3, ChunkLayout.of(_meta(lens), 64)
    x0, y0, z0, dt0 = _bf(T, H * P), _bf(T, H, P), _bf(T, H * P, s=2.0), _bf(T, H, s=2.0)
    par = [torch.randn(H, device=DEV) for _ in range(3)]
    dxv, dg, dout = _bf(T, H, P), torch.randn(T, H, device=DEV), _bf(T, H * P)
    pack = lambda t: torch.zeros(lay.Tp, *t.shape[1:], dtype=t.dtype, device=DEV).index_copy(0, lay.rows, t)  # noqa: E731
    res = []
    for padded in (True, False):
        f = pack if padded else (lambda t: t)
        pick = (lambda t: t[lay.rows]) if padded else (lambda t: t)
        x, y = f(x0).requires_grad_(True), f(y0).requires_grad_(True)
        z, dt, A, bias, D = (t.clone().requires_grad_(True) for t in (z0, dt0, *par))
        xv, dts, g = mamba2_pre(x, dt, bias, A, H, P, lay if padded else None)
        out = mamba2_post(y, x, z, D, H, P, lay if padded else None)
        gx = torch.autograd.grad([xv, g], [x, dt, bias, A], [f(dxv), f(dg)])
        gy = torch.autograd.grad([out], [y, x, z, D], [dout])
        if padded:
            pad = lay.inv_i32 < 0
            assert all(float(t[pad].abs().sum()) == 0 for t in (xv, dts, g, gy[0]))
        res.append(([pick(xv), pick(dts), pick(g), out, pick(gx[0]), gx[1], pick(gy[0]), pick(gy[1]), gy[2]], [gx[2], gx[3], gy[3]]))
    assert all(torch.equal(a, b) for a, b in zip(res[0][0], res[1][0]))
    assert all(rel_err(a, b) < 1e-5 for a, b in zip(res[0][1], res[1][1]))


@pytest.mark.parametrize("P", [64, 256])
@pytest.mark.parametrize("lens", [[1], [128], [15, 17, 63, 65, 1, 200]])
def test_mamba2_skip_gradient_in_place(lens, P):
    """x as a column block read by the value and by the skip connection: its gradient, added up in the kernel and written into the block's
    columns, against the two gradients of separate readers (each rounded to bf16 and so their sum: 3 half ulps); the rest bit for bit."""
    from flame_b200.ops.chunked import ChunkLayout
    from flame_b200.ops.gates import mamba2_post, mamba2_pre, mamba2_pre_skip
    from flame_b200.ops.slots import split_columns
    torch.manual_seed(P)
    T, H, lay = sum(lens), 3, ChunkLayout.of(_meta(lens), 64)
    for rows, lay_ in ((T, None), (lay.Tp, lay)):
        w0, y0, z0, dt0 = _bf(rows, H * P + 24), _bf(rows, H, P), _bf(T, H * P, s=2.0), _bf(T, H, s=2.0)
        par = [torch.randn(H, device=DEV) for _ in range(3)]
        dxv, dg, dout, db = _bf(rows, H, P), torch.randn(rows, H, device=DEV), _bf(T, H * P), _bf(rows, 24)
        res = []
        for together in (True, False):
            w, y, z, dt, A, bias, D = (t.clone().requires_grad_(True) for t in (w0, y0, z0, dt0, *par))
            if together:
                x, b = split_columns(w, (H * P, 24))
                xv, _, g, xs = mamba2_pre_skip(x, dt, bias, A, H, P, lay_)
            else:
                x, b = w[:, :H * P], w[:, H * P:]
                xs = x
                xv, _, g = mamba2_pre(x, dt, bias, A, H, P, lay_)
            out = mamba2_post(y, xs, z, D, H, P, lay_)
            gr = torch.autograd.grad([xv, g, out, b], [w, y, z, dt, bias, A, D], [dxv, dg, dout, db])
            real = slice(None) if lay_ is None else lay.rows
            res.append((gr[0][real].float(), [out, *gr[1:]]))
        assert all(torch.equal(a, b) for a, b in zip(res[0][1], res[1][1]))
        (a, _), (b, _) = res
        assert torch.equal(a[:, H * P:], b[:, H * P:])
        # terms of either sign: each rounding is relative to a term, bounded here by the larger of the terms' sizes
        assert float((a - b).abs().max()) <= 3 * 2.0 ** -8 * float(max(a.abs().max(), b.abs().max())) and rel_err(a, b) < 3 * 2.0 ** -8


def test_gla_gate_formed_in_the_kernel():
    """log(sigmoid(x)) / 16 of the preparation kernel (the first row of a chunk holds one token's gate) against fp64: the exponential is
    off by 2^-22, the other operations round to 2^-24 each, 2^-21 together, also where the gate is nearly zero."""
    from flame_b200.ops import chunk_kernels
    from flame_b200.ops.chunked import ChunkLayout
    T, H, dk = 300, 2, 64
    lay = ChunkLayout.of(_meta([1] * T), 64)
    x = torch.cat([torch.linspace(-60, 60, T * H * dk - 2, device=DEV), torch.tensor([float("-inf"), 0.0], device=DEV)]).bfloat16().view(T, H, dk)
    b = chunk_kernels.gla_prep(x, x, x, 1.0, lay, 16.0)[0][:, 0]
    want = F.logsigmoid(x.double()) / 16
    assert b[-1, -1, -2] == float("-inf")
    ok = want.abs() < float("inf")
    assert ((b.double() - want).abs()[ok] <= 2.0 ** -21 * want.abs()[ok]).all()


def test_silu_rows_round_as_often_as_torch():
    """Every bf16 argument in [-80, 80]: no more results off the correctly rounded one than torch's fp32 chain leaves, both ways."""
    from flame_b200.ops.activations import silu_out_of_chunks
    from flame_b200.ops.chunked import ChunkLayout
    x = torch.arange(1 << 16, device=DEV, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    x = x[(x.abs() <= 80) & (x.abs() >= 2.0 ** -60)]
    x = x[:len(x) // 64 * 64].view(-1, 64)
    lay, off = ChunkLayout.of(_meta([x.shape[0]]), 64), []
    xr = x.double().requires_grad_(True)
    want = F.silu(xr)
    want.sum().backward()
    for new in (True, False):
        xi = torch.zeros(lay.Tp if new else len(x), 64, device=DEV, dtype=x.dtype).index_copy(0, torch.arange(len(x), device=DEV), x).requires_grad_(True)
        y = silu_out_of_chunks(xi.view(lay.NC, 64, 64), lay) if new else F.silu(xi)
        y.sum().backward()
        off.append([int((a != b.to(a.dtype)).sum()) for a, b in ((y, want), (xi.grad[:len(x)], xr.grad))])
    assert off[0][0] <= off[1][0] and off[0][1] <= off[1][1], off


@pytest.mark.parametrize("add", [False, True])
@pytest.mark.parametrize("lens", [[1], [15, 17, 63, 65, 1, 200]])
def test_mamba2_gradients_of_the_padding_are_zero(lens, add):
    """What the backward hands on for padded rows is seen by tensor hooks and gradient statistics: zeros, not what stood in the memory (free
    blocks of its size are filled with NaN first)."""
    from flame_b200.ops.chunked import ChunkLayout
    from flame_b200.ops.gates import mamba2_post, mamba2_pre_skip
    T, H, P, lay = sum(lens), 3, 64, ChunkLayout.of(_meta(lens), 64)
    pad = lay.inv_i32 < 0
    x = _bf(lay.Tp, H * P).masked_fill(pad[:, None], 0).requires_grad_(True)
    y, z, dt = _bf(lay.Tp, H, P).requires_grad_(True), _bf(T, H * P), _bf(T, H)
    par = [torch.randn(H, device=DEV) for _ in range(3)]
    xv, _, g, xs = mamba2_pre_skip(x, dt, par[0], par[1], H, P, lay)
    out = mamba2_post(y, xs.detach().requires_grad_(True) if not add else xs, z, par[2], H, P, lay)
    dirty = [torch.full((lay.Tp, H * P), float("nan"), device=DEV, dtype=torch.bfloat16) for _ in range(8)]
    del dirty
    gx, gy = torch.autograd.grad([xv, g, out], [x, y], [torch.ones_like(xv), torch.ones_like(g), torch.ones_like(out)])
    for t in (gx, gy):
        assert torch.isfinite(t).all() and float(t[pad].abs().sum()) == 0
    xl = xs.detach().requires_grad_(True)
    dirty = [torch.full((lay.Tp, H * P), float("nan"), device=DEV, dtype=torch.bfloat16) for _ in range(8)]
    del dirty
    mamba2_post(y, xl, z, par[2], H, P, lay).backward(torch.ones_like(out))
    assert torch.isfinite(xl.grad).all() and float(xl.grad[pad].abs().sum()) == 0


@pytest.mark.parametrize("sizes,fits", [((8, 16), True), ((8,), False), ((16, 16), False)])
def test_silu_blocks_are_all_of_the_columns(sizes, fits):
    """Blocks that leave columns over (whose gradient nobody would write) or reach past them are not taken."""
    from flame_b200.ops.activations import silu_blocks_to_chunks
    from flame_b200.ops.chunked import ChunkLayout
    assert (silu_blocks_to_chunks(_bf(70, 24), sizes, ChunkLayout.of(_meta([70]), 64)) is not None) == fits


@pytest.mark.parametrize("raw", [False, True])
@pytest.mark.parametrize("lens", [[1], [64, 128], [15, 17, 63, 65, 1, 200], [300, 16, 33]])
def test_gla_backward_writes_its_tokens_alone(lens, raw):
    """The three gradients as column blocks of wider matrices with a chunk's worth of rows behind the last token: the blocks hold what
    matrices of their own do, and everything around them is what it was."""
    from flame_b200.ops import chunk_kernels
    from flame_b200.ops.chunked import ChunkLayout
    torch.manual_seed(len(lens))
    T, H, dk, lay = sum(lens), 2, 72, ChunkLayout.of(_meta(lens), 64)
    NC, n = lay.NC, H * dk
    q, k, g = _bf(T, H, dk), _bf(T, H, dk), _bf(T, H, dk, s=3.0)
    b = chunk_kernels.gla_prep(q, k, g, 0.1, lay, 16.0)[0]
    ins = (q, k, b, _bf(NC, H, 64, 64), _bf(NC, 64, H, dk), _bf(NC, 64, H, dk), _bf(NC * 3, 16, H, dk), _bf(NC * 3, 48, H, dk),
           torch.randn(NC, H, dk, device=DEV))
    want = chunk_kernels.gla_bwd(*ins, 0.1, lay, g if raw else None, 16.0)
    store = [torch.full((T + 64, n + 16), 7.0, dtype=t.dtype, device=DEV) for t in want]
    blocks = [s[:T, 8:8 + n].view(T, H, dk) for s in store]
    chunk_kernels.gla_bwd(*ins, 0.1, lay, g if raw else None, 16.0, blocks)
    for s, block, w in zip(store, blocks, want):
        assert torch.equal(block, w)
        block.fill_(7.0)
        assert (s == 7.0).all()


@pytest.mark.parametrize("G,N,lead", [(1, 128, 512), (2, 64, 512), (1, 64, 516), (2, 40, 512)])
def test_shared_queries_and_keys_as_column_blocks(G, N, lead):
    """q and k read as blocks of one matrix, and their gradients written into one, equal whole tensors bit for bit: also blocks that do
    not start on 16 bytes (copied), a state size of the general path, a second run of a retained graph, and through saved-tensor hooks."""
    from flame_b200.ops.chunked import ChunkLayout, grouped_scalar_gla_chunks
    from flame_b200.ops.slots import reshaped, split_columns
    torch.manual_seed(G + N)
    lay = ChunkLayout.of(_meta([130, 1, 64]), 64)
    H, P, rows = 4, 64, lay.Tp
    x = _bf(rows, lead + 2 * G * N, s=0.3).requires_grad_(True)
    v, g = _bf(rows, H, P), -torch.rand(rows, H, device=DEV) * 0.1
    do = _bf(lay.NC, 64, H, P)

    def grads(blocks, hooks=False):
        first, k, q = split_columns(x, (lead, G * N, G * N)) if blocks else (t.contiguous() for t in x.split((lead, G * N, G * N), 1))
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.to(DEV)) if hooks else torch.enable_grad():
            o = grouped_scalar_gla_chunks(reshaped(q, rows, G, N), reshaped(k, rows, G, N), v, g, lay)
        out = [torch.autograd.grad((o, first), x, (do, torch.ones_like(first)), retain_graph=True)[0] for _ in range(2)]
        return [o.detach(), *out]

    want = grads(False)
    for got in (grads(True), grads(True, hooks=True)):
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("shape", [(1, 5), (15, 16, 40), (17, 33), (518, 16, 96), (0, 64)])
def test_sums_of_partials(shape):
    """fp32 partials added up in a fixed order, against 64 bits: as many roundings as terms of a thread and groups (2^-24 each)."""
    from flame_b200.ops.chunk_kernels import _sum_parts
    torch.manual_seed(3)
    x = torch.randn(shape, device=DEV)
    bound = (shape[0] / 16 + 17) * 2.0 ** -24 * x.double().abs().sum(0)
    assert ((_sum_parts(x).double() - x.double().sum(0)).abs() <= bound).all()
