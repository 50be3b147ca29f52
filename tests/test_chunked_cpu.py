"""The batched-GEMM chunk algorithms (gated delta rule, scalar-gated and per-channel-gated linear attention) against
their token-by-token definitions, forward and backward, on the CPU reference path of ``ops.bgemm`` (fp32)."""
import pytest
import torch
import torch.nn.functional as F

from conftest import rel_err
from flame_b200.ops import linear_attn as la
from flame_b200.ops.bgemm import MASK_TRIL, bgemm, bmm
from flame_b200.ops.chunked import ChunkLayout, gated_delta_rule_tc, gla_tc, scalar_gla_tc
from flame_b200.ops.varlen import VarlenMeta


def _meta(lens):
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    return VarlenMeta.from_cu_seqlens(cu, sum(lens))


LENS = [70, 1, 64, 130, 17]


def _leaf(*shape):
    return torch.randn(*shape).requires_grad_(True)


def _run(fn, inputs):
    for t in inputs:
        t.grad = None
    o = fn()
    torch.manual_seed(99)
    (o * torch.randn_like(o)).sum().backward()
    return [o.detach()] + [t.grad.clone() for t in inputs]


def test_chunk_layout_pack_unpack_roundtrip():
    meta = _meta(LENS)
    lay = ChunkLayout.of(meta)
    assert lay.NC == sum((n + 63) // 64 for n in LENS)
    x = torch.randn(sum(LENS), 3, 5)
    p = lay.pack(x)
    assert p.shape == (lay.NC, 64, 3, 5)
    assert torch.equal(lay.unpack(p), x)
    assert p.abs().sum().item() == pytest.approx(x.abs().sum().item(), rel=1e-5)  # padding rows are zero
    # chunk positions: every listed chunk has its successor in the same document
    first = set(lay.first.tolist())
    for s, idx in enumerate(lay.steps):
        for c in idx.tolist():
            assert (c + 1) not in first


def test_bgemm_reference_layouts_and_bmm_gradients():
    torch.manual_seed(0)
    a = torch.randn(3, 2, 8, 5, requires_grad=True)       # [hi, lo, M, K]
    bt = torch.randn(3, 2, 5, 7, requires_grad=True)      # [hi, lo, K, N]  (mn storage)
    out = bmm(a, bt, b_mn=True, alpha=0.5)
    ref = 0.5 * a @ bt
    assert rel_err(out, ref) < 1e-6
    g = torch.randn_like(out)
    ga, gb = torch.autograd.grad(out, (a, bt), g)
    ra, rb = torch.autograd.grad(ref, (a, bt), g)
    assert rel_err(ga, ra) < 1e-6 and rel_err(gb, rb) < 1e-6
    # masked, decayed scores
    q, k = torch.randn(2, 2, 6, 4), torch.randn(2, 2, 6, 4)
    d = -torch.rand(2, 2, 6).cumsum(-1)
    s = bgemm(q, k, decay=d, mask=MASK_TRIL)
    full = (q @ k.transpose(-1, -2)) * (d[..., :, None] - d[..., None, :]).exp()
    assert rel_err(s, full.tril()) < 1e-6


@pytest.mark.parametrize("gated,chunk", [(True, 128), (False, 128), (True, 64)])
def test_gated_delta_rule_tc_matches_recurrence(gated, chunk):
    torch.manual_seed(2)
    meta = _meta(LENS)
    T, H, K, V = sum(LENS), 2, 16, 24
    q, k, v, braw, graw = _leaf(T, H, K), _leaf(T, H, K), _leaf(T, H, V), _leaf(T, H), _leaf(T, H)
    ins = [q, k, v, braw] + ([graw] if gated else [])

    def make(fn):
        def f():
            g = -F.softplus(graw) if gated else None
            return fn(la.l2norm(q), la.l2norm(k), v, braw.sigmoid(), g, meta)
        return f
    ref = _run(make(la.gated_delta_rule_recurrent), ins)
    out = _run(make(lambda *a: gated_delta_rule_tc(*a, chunk=chunk)), ins)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 1e-4


@pytest.mark.parametrize("G,H,scale,chunk", [(1, 4, 1.0, 64), (2, 6, 0.3, 64), (2, 4, 0.5, 128), (3, 3, 1.0, 64)])
def test_scalar_gla_grouped_heads_match_expanded_heads(G, H, scale, chunk):
    """Queries and keys shared by groups of heads against the same ones repeated per head: output and every gradient (fp32
    sums in another order: 1e-5)."""
    torch.manual_seed(3)
    meta = _meta(LENS)
    T, dk, dv = sum(LENS), 16, 8
    q, k, v, graw = _leaf(T, G, dk), _leaf(T, G, dk), _leaf(T, H, dv), _leaf(T, H)
    ins = [q, k, v, graw]
    ref = _run(lambda: scalar_gla_tc(q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1), v, -F.softplus(graw), meta, scale, chunk), ins)
    out = _run(lambda: scalar_gla_tc(q, k, v, -F.softplus(graw), meta, scale, chunk), ins)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 1e-5


def test_scalar_gla_tc_matches_chunk_reference():
    torch.manual_seed(3)
    meta = _meta(LENS)
    T, H, K, V = sum(LENS), 3, 16, 8
    q, k, v, graw = _leaf(T, H, K), _leaf(T, H, K), _leaf(T, H, V), _leaf(T, H)
    ins = [q, k, v, graw]
    ref = _run(lambda: la.scalar_gla_chunk(q, k, v, -F.softplus(graw), meta, 0.3), ins)
    out = _run(lambda: scalar_gla_tc(q, k, v, -F.softplus(graw), meta, 0.3), ins)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 1e-4


def test_gla_tc_matches_recurrence_with_strong_gates():
    torch.manual_seed(4)
    meta = _meta(LENS)
    T, H, K, V = sum(LENS), 2, 16, 24
    q, k, v, graw = _leaf(T, H, K), _leaf(T, H, K), _leaf(T, H, V), _leaf(T, H, K)
    ins = [q, k, v, graw]
    ref = _run(lambda: la.gla_recurrent(q, k, v, F.logsigmoid(graw * 8), meta), ins)   # decays down to e^-20 per step
    out = _run(lambda: gla_tc(q, k, v, F.logsigmoid(graw * 8), meta), ins)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 1e-4
    assert all(torch.isfinite(t).all() for t in out)


def test_gla_vdecay_tc_and_gsa_match_recurrence():
    from flame_b200.ops.chunked import gla_vdecay_tc
    from flame_b200.ops.gla import gsa
    torch.manual_seed(5)
    meta = _meta(LENS)
    T, H, K, M = sum(LENS), 2, 16, 8
    q, k, s, graw = _leaf(T, H, K), _leaf(T, H, K), _leaf(T, H, M), _leaf(T, H, M)
    ins = [q, k, s, graw]
    ref = _run(lambda: la.gla_recurrent_vdecay(q, k, s, F.logsigmoid(graw * 4), meta, 0.25), ins)
    out = _run(lambda: gla_vdecay_tc(q, k, s, F.logsigmoid(graw * 4), meta, 0.25), ins)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 1e-4
    v = _leaf(T, H, 12)
    ins = [q, k, v, s, graw]
    ref = _run(lambda: la.gsa_recurrent(q, k, v, s, F.logsigmoid(graw) / 8, meta), ins)
    out = _run(lambda: gsa(q, k, v, s, F.logsigmoid(graw) / 8, meta), ins)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 1e-4


def test_mamba2_ssd_grouped_matches_recurrence():
    from flame_b200.ops.scan import mamba2_ssd
    torch.manual_seed(6)
    meta = _meta(LENS)
    T, H, P, N, G = sum(LENS), 4, 8, 16, 2
    x, dtraw, B, C = _leaf(T, H, P), _leaf(T, H), _leaf(T, G, N), _leaf(T, G, N)
    A = -torch.rand(H) * 2 - 0.5
    D = torch.randn(H)
    ins = [x, dtraw, B, C]
    ref = _run(lambda: la.mamba2_ssd_recurrent(x, F.softplus(dtraw), A, B, C, D, meta), ins)
    out = _run(lambda: mamba2_ssd(x, F.softplus(dtraw), A, B, C, D, meta), ins)
    for a, b in zip(out, ref):
        assert rel_err(a, b) < 1e-4


def test_chunk_layout_arrays_match_a_per_token_construction():
    """The array-built layout (rows, inverse map, first / last chunks, per-position lists) against the obvious loops."""
    from flame_b200.ops.chunked import ChunkLayout
    lens = [1, 63, 64, 65, 130, 7]
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    meta = VarlenMeta.from_cu_seqlens(cu, sum(lens), torch.device("cpu"))
    lay = ChunkLayout(meta, 64)
    rows, first, last, c0 = [], [], [], 0
    steps = {}
    for d, n in enumerate(lens):
        nc = (n + 63) // 64
        rows += list(range(c0 * 64, c0 * 64 + n))
        first.append(c0)
        last.append(c0 + nc - 1)
        for s_ in range(nc - 1):
            steps.setdefault(s_, []).append((c0 + s_, d))
        c0 += nc
    assert lay.NC == c0 and lay.T == sum(lens) and lay.Tp == c0 * 64 and not lay.aligned
    assert lay.rows.tolist() == rows and lay.first.tolist() == first and lay.last.tolist() == last
    inv = [-1] * (c0 * 64)
    for t_, r in enumerate(rows):
        inv[r] = t_
    assert lay.inv_i32.tolist() == inv
    assert [s.tolist() for s in lay.steps] == [[c for c, _ in steps[k]] for k in sorted(steps)]
    assert [d.tolist() for d in lay.step_docs] == [[d for _, d in steps[k]] for k in sorted(steps)]
    x = torch.randn(sum(lens), 3, requires_grad=True)
    packed = lay.pack(x)
    assert packed.shape == (c0, 64, 3)
    assert torch.equal(lay.unpack(packed), x)
    assert float(packed.detach().reshape(-1, 3)[[i for i, v in enumerate(inv) if v < 0]].abs().sum()) == 0.0
    packed.square().sum().backward()
    assert torch.allclose(x.grad, 2 * x.detach())


def test_column_split_writes_one_gradient_matrix():
    from flame_b200.ops.gates import split_columns
    x = torch.randn(5, 9, requires_grad=True)
    a, b, c = split_columns(x, (2, 4, 3))
    (a.sum() * 2 + (c * c).sum()).backward()      # the middle block gets no gradient at all
    ref = torch.zeros(5, 9)
    ref[:, :2] = 2
    ref[:, 6:] = 2 * x.detach()[:, 6:]
    assert torch.equal(x.grad, ref)


@pytest.mark.parametrize("dev", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_grouped_score_gradient_is_rounded_once(dev, monkeypatch):
    """The operand of dq and dk is ``scale dQ e^{b_i - b_j}`` rounded to bf16 once: within half a step (2^-8) of its value, plus the
    exponential's 32-bit error (exponents up to 7: 2^-20 of it)."""
    from flame_b200.ops import chunked
    torch.manual_seed(0)
    cu = torch.tensor([0, 128], dtype=torch.int32)
    meta, scale = VarlenMeta.from_cu_seqlens(cu, 128, torch.device(dev)), 0.3
    leaf = lambda *s: torch.randn(*s, device=dev).bfloat16().requires_grad_(True)  # noqa: E731
    q, k, v, g = leaf(128, 1, 64), leaf(128, 1, 64), leaf(128, 4, 64), -torch.rand(128, 4, device=dev) * 0.1
    calls = []

    def spy(a, b, **kw):
        r = bgemm(a, b, **kw)
        calls.append((kw, r))
        return r
    monkeypatch.setattr(chunked, "bgemm", spy)
    o = scalar_gla_tc(q, k, v, g, meta, scale, chunk=64)
    calls.clear()
    torch.autograd.grad(o, [q, k], torch.randn_like(o))
    dQ = next(r for kw, r in calls if kw.get("mask") == MASK_TRIL).double()
    used = [kw["more"][0][0].double() for kw, _ in calls if kw.get("sum_lo", 1) > 1]
    b = g.view(2, 64, 4).double().cumsum(1).permute(0, 2, 1)
    want = scale * dQ * (b[..., :, None] - b[..., None, :]).exp().tril()
    assert len(used) == 2 and used[0].dtype == torch.float64
    for gq in used:
        assert ((gq - want).abs() <= (2.0 ** -8 + 2.0 ** -19) * want.abs()).all()


_MOST = {"gla": "v", "gsa": "v", "vdecay": "qk"}   # what these can do without (their other gradients come from one kernel)


@pytest.mark.parametrize("dev,name", [("cpu", n) for n in ("grouped", "gated", "plain_delta")] + [
    pytest.param("cuda", n, marks=pytest.mark.gpu) for n in ("grouped", "gated", "plain_delta", "gla", "gsa", "vdecay")])
def test_only_the_gradients_that_are_asked_for_are_formed(dev, name, monkeypatch):
    """Every single gradient by itself is the one of the whole backward (the same sums; on the GPU the gated rule's decay up to
    the order of shared-memory atomics) with fewer products and launches, and the operands that stand still get none."""
    from flame_b200.ops import _lib, chunked
    from flame_b200.ops.gla import gsa
    torch.manual_seed(1)
    lens = [128, 70, 1]
    T, H, d = sum(lens), 2, 64
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    meta = VarlenMeta.from_cu_seqlens(cu, T, torch.device(dev))
    dt = torch.bfloat16 if dev == "cuda" else torch.float32
    u = lambda *s: torch.randn(*s, device=dev).to(dt)  # noqa: E731
    rate = lambda *s: -torch.rand(*s, device=dev) * 0.1  # noqa: E731
    q, k = (u(T, 1 if name == "grouped" else H, d) * 0.2 for _ in range(2))
    named, fn = {
        "grouped": (dict(q=q, k=k, v=u(T, H, d), g=rate(T, H)), lambda q, k, v, g: scalar_gla_tc(q, k, v, g, meta, 0.5)),
        "gated": (dict(q=q, k=k, v=u(T, H, d), b=torch.rand(T, H, device=dev), g=rate(T, H)),
                  lambda q, k, v, b, g: gated_delta_rule_tc(q, k, v, b, g, meta)),
        "plain_delta": (dict(q=q, k=k, v=u(T, H, d), b=torch.rand(T, H, device=dev)), lambda q, k, v, b: gated_delta_rule_tc(q, k, v, b, None, meta)),
        "gla": (dict(q=q, k=k, v=u(T, H, d), g=rate(T, H, d)), lambda q, k, v, g: gla_tc(q, k, v, g, meta)),
        "gsa": (dict(q=q, k=k, v=u(T, H, d), s=torch.rand(T, H, d, device=dev), g=rate(T, H, d)), lambda q, k, v, s, g: gsa(q, k, v, s, g, meta)),
        "vdecay": (dict(q=q, k=k, v=u(T, H, d), g=rate(T, H, d)), lambda q, k, v, g: chunked.gla_vdecay_tc(q, k, v, g, meta, 0.5)),
    }[name]
    dy = u(T, H, d)
    calls = []
    monkeypatch.setattr(chunked, "bgemm", lambda *a, **kw: calls.append(1) or bgemm(*a, **kw))

    def run(wanted):
        args = {n: t.clone().requires_grad_(n in wanted) for n, t in named.items()}
        y = fn(**args)
        calls.clear()
        before = _lib.launches()
        grads = torch.autograd.grad(y, [args[n] for n in wanted], dy.to(y.dtype))
        return dict(zip(wanted, grads)), (len(calls), _lib.launches() - before)
    whole, most = run(list(named))
    for n in named:
        got, work = run([n])
        if dev == "cuda" and name == "gated" and n == "g":
            assert (got[n] - whole[n]).abs().max() <= 512 * 2.0 ** -24 * whole[n].abs().max()
        else:
            assert torch.equal(got[n], whole[n]), n
        if n in _MOST.get(name, n):
            assert work[0] < most[0] and (dev == "cpu" or work[1] < most[1]), (n, work, most)
    still = [n for n in named if n not in "qk"]
    got, work = run(still)
    assert work[0] < most[0] or name in _MOST


@pytest.mark.parametrize("lens", [[64, 128], LENS])
def test_mamba2_elementwise_reference_in_chunk_rows(lens):
    """Where the kernels do not apply, operands in the padded rows of a layout give the same numbers as packed ones, zeros in the padding;
    x's gradient too.  The same fp32 operations on the same rows: equal (the parameters' gradients are sums over the tokens: 1e-5)."""
    from flame_b200.ops.gates import mamba2_post, mamba2_pre_skip
    torch.manual_seed(0)
    T, H, P, lay = sum(lens), 2, 4, ChunkLayout.of(_meta(lens), 64)
    x0, y0, z0, dt0 = torch.randn(T, H * P), torch.randn(T, H, P), torch.randn(T, H * P), torch.randn(T, H)
    par, res = [torch.randn(H) for _ in range(3)], []
    for padded in (True, False):
        f = (lambda t: lay.pack(t).flatten(0, 1).clone()) if padded else torch.clone
        pick = (lambda t: t[lay.rows]) if padded else (lambda t: t)
        x, y = f(x0).requires_grad_(True), f(y0).requires_grad_(True)
        z, dt, bias, A, D = (t.clone().requires_grad_(True) for t in (z0, dt0, *par))
        xv, dts, g, xs = mamba2_pre_skip(x, dt, bias, A, H, P, lay if padded else None)
        out = mamba2_post(y, xs, z, D, H, P, lay if padded else None)
        if padded:
            assert xv.shape[0] == dts.shape[0] == g.shape[0] == lay.Tp
            assert all(float(t[lay.inv_i32 < 0].abs().sum()) == 0 for t in (xv, dts, g))
        total = (pick(xv) * x0.view(T, H, P)).sum() + (pick(g) * dt0).sum() + (out * z0).sum()
        res.append([pick(xv), pick(dts), pick(g), out] + [pick(t) if i < 2 else t for i, t in enumerate(torch.autograd.grad(total, [x, y, z, dt, bias, A, D]))])
    for a, b in zip(*res):
        assert rel_err(a, b) < 1e-5
