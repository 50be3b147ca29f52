"""Numerics of every CUDA kernel against a plain PyTorch fp32 reference of the same op (run on a B200)."""
import math

import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(autouse=True)
def _status():
    from flame_b200.ops import _lib
    _lib.status_clear()
    yield
    _lib.assert_status_ok()


def _meta(lens):
    from flame_b200.ops.varlen import VarlenMeta
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    return VarlenMeta.from_cu_seqlens(cu, sum(lens), torch.device(DEV))


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (304, 520, 200), (1024, 1024, 1024), (4096, 2816, 1024)])
def test_gemm_three_layouts(M, N, K):
    from flame_b200.ops import gemm
    torch.manual_seed(0)
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(N, K, device=DEV, dtype=torch.bfloat16)
    ref = a.float() @ b.float().t()
    assert rel_err(gemm.gemm_nt(a, b, splits=1), ref) < 5e-3
    bt, at = b.t().contiguous(), a.t().contiguous()
    assert rel_err(gemm.gemm_nn(a, bt, splits=1), ref) < 5e-3
    assert rel_err(gemm.gemm_tn(at, bt, splits=1), ref) < 5e-3
    assert rel_err(gemm.gemm_nt(a, b, out_dtype=torch.float32, splits=1), ref) < 1e-5


def test_gemm_split_k_and_accumulate():
    from flame_b200.ops import gemm
    torch.manual_seed(1)
    dy = torch.randn(8192, 1024, device=DEV, dtype=torch.bfloat16)
    x = torch.randn(8192, 512, device=DEV, dtype=torch.bfloat16)
    ref = dy.float().t() @ x.float()
    assert rel_err(gemm.gemm_tn(dy, x, out_dtype=torch.float32), ref) < 1e-5
    acc = torch.ones(1024, 512, device=DEV)
    gemm.gemm_tn(dy, x, out=acc, accumulate=True, splits=4)
    assert rel_err(acc, ref + 1) < 1e-5
    # bitwise repeatable (fixed reduction order)
    o1 = gemm.gemm_tn(dy, x, out_dtype=torch.float32, splits=4)
    o2 = gemm.gemm_tn(dy, x, out_dtype=torch.float32, splits=4)
    assert torch.equal(o1, o2)


@pytest.mark.parametrize("M,N,K", [(136, 72, 5000), (1000, 520, 9000), (256, 256, 2048), (2040, 2312, 8200), (5640, 1024, 4096)])
def test_gemm_tiles_cut_along_k(M, N, K):
    """Tiles of the last round in pieces of K: few tiles and many, ragged in every dimension, all output forms, also where the result's rows
    or start rule out tensor copies (then nothing is cut).  fp32 results: the accumulator takes 16 products a step and cuts off below its last place, on average half
    of it, always in the same direction: K / 16 steps of 2^-24.  bf16 results: 2^-8."""
    from flame_b200.ops import _lib, gemm
    if (M, N) != (5640, 1024):
        assert _lib.lib().fb_gemm_cut_bytes(M, N, K) > 0
    tol = K / 16 * 2 ** -24
    torch.manual_seed(2)
    at = torch.randn(K, M, device=DEV, dtype=torch.bfloat16)
    bt = torch.randn(K, N, device=DEV, dtype=torch.bfloat16)
    a, b = at.t().contiguous(), bt.t().contiguous()
    ref = a.float() @ b.float().t()
    for fn, x, y in ((gemm.gemm_nt, a, b), (gemm.gemm_nn, a, bt), (gemm.gemm_tn, at, bt)):
        assert rel_err(fn(x, y), ref) < 2 ** -8
        out = fn(x, y, out_dtype=torch.float32)
        assert rel_err(out, ref) < tol
        assert torch.equal(out, fn(x, y, out_dtype=torch.float32))
        assert rel_err(fn(x, y, out_dtype=torch.float32, alpha=0.5), 0.5 * ref) < tol
        wide = torch.ones(M, N + 9, device=DEV)
        for lo, hi in ((4, 4 + N), (1, 1 + N)):     # rows of 4 (N + 9) bytes: no tensor copies
            fn(x, y, out=wide[:, lo:hi], accumulate=True)
        assert rel_err(wide[:, 5:N], (ref[:, 1:N - 4] + 1) + ref[:, 4:N - 1]) < tol
        assert torch.equal(wide[:, [0, N + 5]], torch.ones(M, 2, device=DEV))
        wide = torch.ones(M, N + 8, device=DEV)     # a column block
        fn(x, y, out=wide[:, 4:4 + N], accumulate=True)
        assert rel_err(wide[:, 4:4 + N], ref + 1) < tol
        assert torch.equal(wide[:, [0, 3, N + 4, N + 7]], torch.ones(M, 4, device=DEV))


@pytest.mark.parametrize("variant", [1, 2])
@pytest.mark.parametrize("splits", [1, 4])
def test_gemm_results_that_start_between_vectors(variant, splits):
    """Results whose rows are whole vectors apart (or lie back to back) but start between vectors: every output form, with a bias too, in
    both kernels and after a split along K, equals the result on a boundary bit for bit and leaves its neighbours alone."""
    from flame_b200.ops import _lib, gemm
    torch.manual_seed(6)
    M, N, K = 136, 296, 1024
    at, bt = (torch.randn(K, n, device=DEV, dtype=torch.bfloat16) for n in (M, N))
    bias = torch.randn(N, device=DEV).to(torch.bfloat16)
    a, b = at.t().contiguous(), bt.t().contiguous()
    old = _lib.lib().fb_gemm_set_variant(variant)
    try:
        forms = [(torch.float32, dict(accumulate=True)), (torch.float32, {}), (torch.bfloat16, {}), (torch.bfloat16, dict(bias=bias))]
        for dtype, more in forms[:4 if splits == 1 else 3]:
            want = torch.ones(M, N, device=DEV, dtype=dtype)
            gemm.gemm_nt(a, b, out=want, splits=splits, **more)
            for start in (1, 2, 3, 4, 5):
                for pitch in (N, N + 8) if splits == 1 else (N,):
                    store = torch.ones(M * pitch + 16, device=DEV, dtype=dtype)
                    out = store[start:start + M * pitch].view(M, pitch)[:, :N]
                    gemm.gemm_nt(a, b, out=out, splits=splits, **more)
                    assert torch.equal(out, want)
                    out.fill_(1)
                    assert (store == 1).all()
                    if not more.get("bias") is None:
                        continue
                    gemm.gemm_tn(at, bt, out=out, **more)   # the library's own choice of a split
                    assert rel_err(out, want) < 2 ** -8
    finally:
        _lib.lib().fb_gemm_set_variant(old)


@pytest.mark.parametrize("N,dtype,start,pitch", [(70, torch.float32, 0, 70), (68, torch.bfloat16, 0, 68), (72, torch.float32, 2, 72),
                                                 (72, torch.float32, 0, 77), (72, torch.bfloat16, 3, 80)])
def test_gemm_results_without_tensor_copies_are_split_or_whole(N, dtype, start, pitch):
    """Few tiles and a long K into results that no tensor copy can write: where the rows lie back to back the sum is split over the whole K
    as the library's model says (equal to that split asked for, bit for bit), else it is whole: one launch, no scratch."""
    from flame_b200.ops import _lib, gemm
    M, K = 136, 5000
    torch.manual_seed(9)
    a, b = torch.randn(K, M, device=DEV, dtype=torch.bfloat16), torch.randn(K, 80, device=DEV, dtype=torch.bfloat16)[:, :N]
    assert _lib.lib().fb_gemm_cut_bytes(M, N, K) > 0
    split = int(_lib.lib().fb_gemm_pick_splits(M, N, K)) if pitch == N else 1
    assert (split > 1) == (pitch == N)
    got, want = (torch.zeros(M * pitch + 8, device=DEV, dtype=dtype)[start:start + M * pitch].view(M, pitch)[:, :N] for _ in range(2))
    gemm.gemm_tn(a, b, out=want, splits=split)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before, held = _lib.launches(), torch.cuda.memory_allocated()
    gemm.gemm_tn(a, b, out=got)
    assert _lib.launches() - before == (2 if split > 1 else 1)
    assert split > 1 or torch.cuda.max_memory_allocated() == held
    assert torch.equal(got, want)


def test_gemm_scratch_belongs_to_one_product():
    """Products in pieces share no scratch: threads on one stream, each between whose two launches another's may come, and a captured
    product that is replayed after a larger one on its stream, with the memory in between handed to others.  All bits as alone."""
    import threading
    from flame_b200.ops import _lib, gemm
    M, N, K = 136, 72, 5000
    assert _lib.lib().fb_gemm_cut_bytes(M, N, K) > 0 and _lib.lib().fb_gemm_cut_bytes(2040, 2312, 8200) > _lib.lib().fb_gemm_cut_bytes(M, N, K)
    torch.manual_seed(4)
    mk = lambda *s: torch.randn(*s, device=DEV, dtype=torch.bfloat16)  # noqa: E731
    pairs = [(mk(M, K), mk(N, K)) for _ in range(4)]
    want = [gemm.gemm_nt(a, b, out_dtype=torch.float32) for a, b in pairs]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        for _ in range(50):
            if not torch.equal(gemm.gemm_nt(*pairs[i], out_dtype=torch.float32), want[i]):
                bad.append(i)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        gemm.gemm_nt(*pairs[0], out_dtype=torch.float32)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            out = gemm.gemm_nt(*pairs[0], out_dtype=torch.float32)
        gemm.gemm_nt(mk(2040, 8200), mk(2312, 8200))
        others = [torch.full((1 << 18,), 7.0, device=DEV) for _ in range(64)]
        graph.replay()
    s.synchronize()
    assert torch.equal(out, want[0]) and all(bool((o == 7).all()) for o in others)


@pytest.mark.parametrize("lens,H,Hkv,Dh,window", [([128], 1, 1, 64, 0), ([300, 77, 129], 2, 1, 64, 0),
                                                   ([1000, 24, 512], 4, 4, 64, 0), ([640], 2, 2, 64, 200),
                                                   ([300, 200], 2, 1, 128, 0), ([300, 200], 2, 2, 128, 100),
                                                   ([64], 1, 1, 128, 0), ([1000, 24, 513, 1], 8, 2, 128, 0),
                                                   ([2048, 333], 4, 1, 128, 512), ([4096], 2, 2, 128, 0)])
def test_attention_forward_backward(lens, H, Hkv, Dh, window):
    from flame_b200.ops.attention import attention, attention_reference
    torch.manual_seed(2)
    meta = _meta(lens)
    T = sum(lens)
    q = torch.randn(T, H, Dh, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    k = torch.randn(T, Hkv, Dh, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    v = torch.randn(T, Hkv, Dh, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    o = attention(q, k, v, meta, None, window)
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    oref = attention_reference(qf, kf, vf, meta, 1 / math.sqrt(Dh), window)
    assert rel_err(o, oref) < 1e-2
    # both head dims run backward kernels of this library (head dim 128: the transposed-score kernel)
    do = torch.randn_like(o)
    o.backward(do)
    oref.backward(do.float())
    assert rel_err(q.grad, qf.grad) < 2e-2
    assert rel_err(k.grad, kf.grad) < 2e-2
    assert rel_err(v.grad, vf.grad) < 2e-2


def test_rmsnorm_residual_and_gated():
    from flame_b200.ops.norm import rms_norm, rms_norm_gated, rms_norm_reference
    torch.manual_seed(3)
    T, D = 777, 1024
    x = torch.randn(T, D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    r = torch.randn(T, D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(D, device=DEV) * 0.1 + 1).to(torch.bfloat16).requires_grad_(True)
    y, res = rms_norm(x, w, 1e-6, r, True)
    xf, rf, wf = (t.detach().float().requires_grad_(True) for t in (x, r, w))
    yr, resr = rms_norm_reference(xf, wf, 1e-6, rf, True)
    assert rel_err(y, yr) < 1e-2 and rel_err(res, resr) < 1e-2
    g1, g2 = torch.randn_like(y), torch.randn_like(res)
    (y.float() * g1.float()).sum().backward(retain_graph=True)
    torch.autograd.backward([res], [g2])
    (yr * g1.float()).sum().backward(retain_graph=True)
    torch.autograd.backward([resr], [g2.float()])
    assert rel_err(x.grad, xf.grad) < 2e-2 and rel_err(r.grad, rf.grad) < 2e-2 and rel_err(w.grad, wf.grad) < 2e-2
    # gated, per-head
    o = torch.randn(T, 4, 256, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    g = torch.randn(T, 4, 256, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    w2 = torch.ones(256, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    out = rms_norm_gated(o, g, w2, 1e-5, "swish")
    of, gf, w2f = (t.detach().float().requires_grad_(True) for t in (o, g, w2))
    outr = rms_norm_reference(of, w2f, 1e-5, gate=gf, activation="swish")
    assert rel_err(out, outr) < 1e-2
    dout = torch.randn_like(out)
    out.backward(dout)
    outr.backward(dout.float())
    assert rel_err(o.grad, of.grad) < 2e-2 and rel_err(g.grad, gf.grad) < 2e-2 and rel_err(w2.grad, w2f.grad) < 2e-2


@pytest.mark.parametrize("D", [256, 264, 320, 512, 520])
@pytest.mark.parametrize("rows,gate", [(1, None), (5, "swish"), (777, "sigmoid"), (4803, "swish")])
def test_rmsnorm_backward_of_rows_side_by_side(D, rows, gate):
    """Widths around those at which a row's lanes change, and numbers of rows that end inside a trip, against 64 bits.  dx and dgate:
    three fp32 roundings and a row sum of D terms (2^-20 of the row's largest), rounded to bf16 (2^-8); dw: a sum over the rows."""
    from flame_b200.ops.norm import rms_norm, rms_norm_gated
    torch.manual_seed(D + rows)
    mk = lambda *s: torch.randn(*s, device=DEV).to(torch.bfloat16).requires_grad_(True)  # noqa: E731
    x, g, w = mk(rows, D), mk(rows, D), mk(D)
    dy = torch.randn(rows, D, device=DEV).to(torch.bfloat16)
    ins = (x, w) if gate is None else (x, w, g)
    y = rms_norm(x, w, 1e-5) if gate is None else rms_norm_gated(x, g, w, 1e-5, gate)
    got = torch.autograd.grad(y, ins, dy)
    xd, gd, wd = (t.detach().double().requires_grad_(True) for t in (x, g, w))
    rstd = torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5)
    act = {None: 1.0, "swish": gd * gd.sigmoid(), "sigmoid": gd.sigmoid()}[gate]
    want = torch.autograd.grad(xd * rstd * wd * act, (xd, wd) if gate is None else (xd, wd, gd), dy.double())
    for a, r, i in zip(got, want, ins):
        big = r.abs().amax(-1, keepdim=True) if r.dim() == 2 else (dy.double() * xd * rstd * act).abs().sum(0).detach()
        assert ((a.double() - r).abs() <= 2.0 ** -8 * r.abs() + 2.0 ** -18 * big).all(), i.shape


@pytest.mark.parametrize("D", [64, 128, 256, 320, 768, 1024, 2048, 2056])
@pytest.mark.parametrize("rows,form", [(1, "residual"), (9, "residual"), (4803, "residual"), (4803, "plain"), (4803, "swish")])
def test_rmsnorm_backward_with_the_next_rows_on_their_way(D, rows, form):
    """Every width class, with the gradient of a residual and without, with a gate, and numbers of rows that end inside a trip; bounds as in
    the test above."""
    from flame_b200.ops.norm import rms_norm, rms_norm_gated
    torch.manual_seed(D + rows)
    mk = lambda *s: torch.randn(*s, device=DEV).to(torch.bfloat16).requires_grad_(True)  # noqa: E731
    x, r, g, w = mk(rows, D), mk(rows, D), mk(rows, D), mk(D)
    dy, dz = (torch.randn(rows, D, device=DEV).to(torch.bfloat16) for _ in range(2))
    xd, gd, wd = (t.detach().double().requires_grad_(True) for t in (x, g, w))
    act = gd * gd.sigmoid() if form == "swish" else 1.0
    if form == "residual":
        y, z = rms_norm(x, w, 1e-5, r, True)
        got = torch.autograd.grad((y, z), (x, w), (dy, dz))
        xd = z.detach().double().requires_grad_(True)     # the sum as it was rounded
    elif form == "plain":
        got = torch.autograd.grad(rms_norm(x, w, 1e-5), (x, w), dy)
    else:
        got = torch.autograd.grad(rms_norm_gated(x, g, w, 1e-5, form), (x, w, g), dy)
    rstd = torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5)
    want = list(torch.autograd.grad(xd * rstd * wd * act, (xd, wd, gd) if form == "swish" else (xd, wd), dy.double()))
    size = [v.abs().amax(-1, keepdim=True) for v in want]
    size[1] = (dy.double() * xd * rstd * act).abs().sum(0).detach()
    if form == "residual":
        want[0] = want[0] + dz.double()
        size[0] = size[0] + dz.double().abs()
    for a, b, big in zip(got, want, size):
        assert ((a.double() - b).abs() <= 2.0 ** -8 * b.abs() + 2.0 ** -18 * big).all(), b.shape


@pytest.mark.parametrize("D", [56, 64, 128, 136, 256])
@pytest.mark.parametrize("extra", [-1, 0, 5])
def test_rmsnorm_backward_of_plain_rows_around_four_per_trip(D, extra):
    """Short rows without gate and residual around the 2^24 elements from which a trip takes four of them; dx as in the tests above, dw: a sum of
    all rows in fp32, at most 500 terms one after the other in a thread and as many partial sums (2^-24 of the sum of absolutes each)."""
    from flame_b200.ops.norm import rms_norm
    torch.manual_seed(D)
    rows = -(-(1 << 24) // D) + extra
    x, w = (torch.randn(*s, device=DEV).to(torch.bfloat16).requires_grad_(True) for s in ((rows, D), (D,)))
    dy = torch.randn(rows, D, device=DEV).to(torch.bfloat16)
    dx, dw = torch.autograd.grad(rms_norm(x, w, 1e-5), (x, w), dy)
    v, g = x.detach().double(), dy.double()
    rstd = torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-5)
    gw = g * w.detach().double()
    want = rstd * (gw - v * rstd * (gw * v * rstd).mean(-1, keepdim=True))
    assert ((dx.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * want.abs().amax(-1, keepdim=True)).all()
    terms = g * v * rstd
    assert ((dw.double() - terms.sum(0)).abs() <= 2.0 ** -8 * terms.sum(0).abs() + 1000 * 2.0 ** -24 * terms.abs().sum(0)).all()


@pytest.mark.parametrize("D", [264, 512, 520, 1024, 1032, 2048, 2056])
@pytest.mark.parametrize("rows,form", [(1, "plain"), (9, "sum"), (777, "prenorm"), (777, "swish"), (777, "sigmoid"), (777, "bare")])
def test_rmsnorm_forward_of_rows_in_registers(D, rows, form):
    """Widths around what a lane holds, with a residual (the sum kept, or not), a gate and without a weight, against 64 bits: a sum of D
    squares and four roundings in fp32 (2^-18), rounded to bf16 (2^-8); the kept sum is the rounded one."""
    from flame_b200.ops.norm import rms_norm, rms_norm_gated
    torch.manual_seed(D + rows)
    x, r, w = (torch.randn(*s, device=DEV).to(torch.bfloat16) for s in ((rows, D), (rows, D), (D,)))
    v = x.double()
    if form == "prenorm":
        y, z = rms_norm(x, w, 1e-5, r, True)
        assert torch.equal(z, x + r)
        v = z.double()
    elif form == "sum":
        y, v = rms_norm(x, w, 1e-5, r), None
        both = [x.double() + r.double(), (x + r).double()]   # whether the sum is rounded is the operator's choice
    elif form in ("swish", "sigmoid"):
        y = rms_norm_gated(x, r, w, 1e-5, form)
    else:
        y = rms_norm(x, None if form == "bare" else w, 1e-5)
    act = {"swish": r.double() * r.double().sigmoid(), "sigmoid": r.double().sigmoid()}.get(form, 1.0)
    near = []
    for v in both if form == "sum" else [v]:
        want = v * torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-5) * (1.0 if form == "bare" else w.double()) * act
        near.append(bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * want.abs().amax(-1, keepdim=True)).all()))
    assert any(near)


@pytest.mark.parametrize("D", [640, 768, 776, 1272, 1280, 1288])
@pytest.mark.parametrize("form", ["plain", "sum", "prenorm", "swish", "sigmoid"])
def test_rmsnorm_forward_of_rows_that_fill_their_vectors(D, form):
    """Widths around those at which a lane takes three or five vectors instead of four or eight; bounds as in the test above."""
    test_rmsnorm_forward_of_rows_in_registers(D, 777, form)


@pytest.mark.parametrize("H", [1, 3, 4, 5, 9])
@pytest.mark.parametrize("Dh,rot", [(64, 64), (128, 128), (64, 32), (48, 16)])
@pytest.mark.parametrize("many", [False, True])
def test_rope_heads_of_one_thread(H, Dh, rot, many):
    """Numbers of heads around what a thread takes, partial rotation, both directions, in place in a wider matrix, beside it and from fp32,
    against 64 bits: two products and a sum (2^-22 of the larger operand), rounded to bf16 (2^-8)."""
    from flame_b200.ops.rope import rope_from_fp32_, rope_inplace_, rope_rotated
    torch.manual_seed(H + Dh + rot)
    T = 333 + many * (600000 * 16 // (H * rot))   # beyond this a thread takes several heads
    pos = torch.randint(0, 500, (T,), device=DEV, dtype=torch.int32)
    ang = torch.rand(500, rot // 2, device=DEV) * 6
    cos, sin = ang.cos(), ang.sin()
    wide = torch.randn(T, (H + 2) * Dh, device=DEV).to(torch.bfloat16)
    x = wide[:, Dh:(H + 1) * Dh].view(T, H, Dh)
    src, before = x.clone(), wide.clone()

    def check(y, src, sign):
        a, b = src[..., :rot // 2].double(), src[..., rot // 2:rot].double()
        c, s = cos[pos.long(), None].double(), sign * sin[pos.long(), None].double()
        want, size = torch.cat([a * c - b * s, a * s + b * c], -1), torch.maximum(a.abs(), b.abs()).repeat(1, 1, 2)
        assert ((y[..., :rot].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -22 * size).all()

    check(rope_rotated(x, pos, cos, sin), src, 1)
    assert torch.equal(wide, before)
    rope_inplace_(x, pos, cos, sin, conj=True)
    check(x, src, -1)
    assert torch.equal(x[..., rot:], src[..., rot:])
    assert torch.equal(wide[:, :Dh], before[:, :Dh]) and torch.equal(wide[:, (H + 1) * Dh:], before[:, (H + 1) * Dh:])
    if rot == Dh:
        f = torch.randn(T, H, Dh, device=DEV)
        rope_from_fp32_(f, x, pos, cos, sin, conj=True)
        check(x, f, -1)


@pytest.mark.parametrize("op", ["swiglu", "gate_up", "embedding", "attention64", "attention128", "qkv_attention", "stickbreaking", "qkv_stickbreaking"])
def test_gradients_that_start_between_vectors(op):
    """A whole gradient that begins off a 16-byte boundary gives what one on a boundary gives (attention adds dq up in no fixed order)."""
    from flame_b200.ops.activations import swiglu
    from flame_b200.ops.attention import attention
    from flame_b200.ops.attn_block import qkv_attention
    from flame_b200.ops.embedding import embedding
    from flame_b200.ops.linear import gate_up_swiglu
    from flame_b200.ops.stickbreaking import sb_attention, sb_qkv_attention
    torch.manual_seed(2)
    T, H, meta = 200, 2, _meta([77, 123])
    leaf = lambda *s: torch.randn(*s, device=DEV).to(torch.bfloat16).requires_grad_(True)  # noqa: E731
    D = 128 if op == "attention128" else 64
    w = leaf(2 * 128, 64)
    ins, run = {
        "swiglu": ([leaf(T, 256)], swiglu),
        "gate_up": ([leaf(T, 64)], lambda x: gate_up_swiglu(x, w.detach()[:128], w.detach()[128:])),
        "embedding": ([leaf(50, 64)], lambda t: embedding(torch.arange(T, device=DEV) % 50, t)),
        "qkv_attention": ([leaf(T, 3 * H * 64)], lambda x: qkv_attention(x, meta, H, H, 64)),
        "stickbreaking": ([leaf(T, H, 64) for _ in range(3)], lambda q, k, v: sb_attention(q, k, v, meta)[0]),
        "qkv_stickbreaking": ([leaf(T, 3 * H * 64)], lambda x: sb_qkv_attention(x, meta, H, 64)),
    }.get(op, ([leaf(T, H, D) for _ in range(3)], lambda q, k, v: attention(q, k, v, meta)))
    y = run(*ins)
    y = y[0] if isinstance(y, tuple) else y
    dy = torch.randn(y.shape, device=DEV).to(torch.bfloat16)
    odd = torch.empty(y.numel() + 3, device=DEV, dtype=torch.bfloat16)[3:].view(y.shape).copy_(dy)
    assert odd.data_ptr() % 16
    want = torch.autograd.grad(y, ins, dy, retain_graph=True)
    for a, b in zip(torch.autograd.grad(y, ins, odd), want):
        assert rel_err(a, b) < (2 ** -9 if "att" in op or "stick" in op else 1e-9)


def test_activations_and_rotations_between_vectors():
    """Whole operands that begin off a 16-byte boundary."""
    from flame_b200.ops.activations import swiglu
    from flame_b200.ops.rope import rope_inplace_, rope_rotated
    torch.manual_seed(2)
    x = torch.randn(200, 256, device=DEV).to(torch.bfloat16)
    odd = torch.empty(x.numel() + 3, device=DEV, dtype=torch.bfloat16)[3:].view(x.shape).copy_(x)
    assert torch.equal(swiglu(odd), swiglu(x))
    pos = torch.arange(200, device=DEV, dtype=torch.int32)
    ang = torch.rand(200, 32, device=DEV)
    want = rope_rotated(x.view(200, 4, 64), pos, ang.cos(), ang.sin())
    assert rel_err(rope_rotated(odd.view(200, 4, 64), pos, ang.cos(), ang.sin()), want) < 2 ** -8
    rope_inplace_(odd.view(200, 4, 64), pos, ang.cos(), ang.sin())
    assert rel_err(odd.view(200, 4, 64), want) < 2 ** -8


def test_swiglu_rope_embedding():
    from flame_b200.ops.activations import swiglu, swiglu_reference
    from flame_b200.ops.embedding import embedding
    from flame_b200.ops.rope import apply_rope, rope_reference, rope_tables
    torch.manual_seed(4)
    gu = torch.randn(513, 2 * 2816, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    a = swiglu(gu)
    guf = gu.detach().float().requires_grad_(True)
    ar = swiglu_reference(guf)
    assert rel_err(a, ar) < 1e-2
    da = torch.randn_like(a)
    a.backward(da)
    ar.backward(da.float())
    assert rel_err(gu.grad, guf.grad) < 2e-2
    meta = _meta([100, 300, 113])
    cos, sin = rope_tables(64, 512, 10000.0, torch.device(DEV))
    x = torch.randn(513, 4, 64, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    y = apply_rope(x, meta.position_ids, cos, sin)
    yr = rope_reference(x.detach().float(), meta.position_ids, cos, sin)
    assert rel_err(y, yr) < 1e-2
    dy = torch.randn_like(y)
    y.backward(dy)
    assert rel_err(x.grad, rope_reference(dy.float(), meta.position_ids, cos, sin, conj=True)) < 1e-2
    w = torch.randn(1000, 256, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    ids = torch.randint(0, 1000, (3, 700), device=DEV)
    e = embedding(ids, w)
    assert torch.equal(e, w.detach()[ids])
    de = torch.randn_like(e)
    e.backward(de)
    ref = torch.zeros(1000, 256, device=DEV).index_add_(0, ids.reshape(-1), de.reshape(-1, 256).float())
    assert rel_err(w.grad, ref) < 1e-2


@pytest.mark.parametrize("lens,H", [([128], 1), ([300, 77, 129, 1], 2), ([1000, 24, 512], 3), ([4096], 2), ([4096, 2500], 1)])
def test_stickbreaking_attention_forward_backward(lens, H):
    from flame_b200.ops.linear_attn import stickbreaking_reference
    from flame_b200.ops.stickbreaking import sb_attention
    torch.manual_seed(9)
    meta = _meta(lens)
    T, Dh = sum(lens), 64
    q = torch.randn(T, H, Dh, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    k = torch.randn(T, H, Dh, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    v = torch.randn(T, H, Dh, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    o, rem = sb_attention(q, k, v, meta)
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    oref, remref = stickbreaking_reference(qf, kf, vf, meta)
    assert rel_err(o, oref) < 1e-2
    assert (rem - remref).abs().max().item() < 2e-2
    do = torch.randn_like(o)
    drem = torch.randn_like(rem) * 0.3
    torch.autograd.backward([o, rem], [do, drem])
    torch.autograd.backward([oref, remref], [do.float(), drem])
    # dl = dA - sigma * prefix: the prefix is a difference against do . o, which the kernels carry to fp32 accuracy (a
    # two-term bf16 split of the output), so the error no longer grows with the row length (rows of 4096 included)
    assert rel_err(q.grad, qf.grad) < 3e-2
    assert rel_err(k.grad, kf.grad) < 3e-2
    assert rel_err(v.grad, vf.grad) < 3e-2


@pytest.mark.parametrize("size", [1.0, 6.0])
def test_stickbreaking_attention_at_tile_edges_and_far_out(size):
    """Documents around the 64-key and 128-query tiles against fp64, with logits of some units and of some forty (neighbours beyond 2^60 : 1,
    where the weights are 0 or 1): outputs and value gradients of bf16 weights and operands, 1e-2; gradients
    through the logits, small differences of their sums, 3e-2 where the weights are not saturated, and finite."""
    from flame_b200.ops.linear_attn import stickbreaking_reference
    from flame_b200.ops.stickbreaking import sb_attention
    torch.manual_seed(11)
    lens, H = [1, 2, 63, 64, 65, 127, 128, 129, 191, 192, 193, 320], 2
    meta, T = _meta(lens), sum(lens)
    q, k, v = ((torch.randn(T, H, 64, device=DEV) * (size if i < 2 else 1)).bfloat16().requires_grad_(True) for i in range(3))
    do, drem = torch.randn(T, H, 64, device=DEV).bfloat16(), None
    o, rem = sb_attention(q, k, v, meta)
    qd, kd, vd = (t.detach().double().requires_grad_(True) for t in (q, k, v))
    od, remd = stickbreaking_reference(qd, kd, vd, meta)
    drem = torch.randn_like(rem) * 0.3
    torch.autograd.backward([o, rem], [do, drem])
    torch.autograd.backward([od, remd], [do.double(), drem.double()])
    assert rel_err(o, od) < 1e-2 and rel_err(v.grad, vd.grad) < 1e-2 and (rem - remd).abs().max().item() < 1e-5
    for a, b in ((q, qd), (k, kd)):
        assert torch.isfinite(a.grad).all() and (size > 1 or rel_err(a.grad, b.grad) < 3e-2)


@pytest.mark.parametrize("nats", [1.0, 30.0, 41.0, 43.0, 55.0, 69.0])
def test_stickbreaking_remainder_beside_dominating_keys(nats):
    """What one or two keys of large logits leave of a row, relative to itself: the exponent's argument is rounded twice (100 2^-24), the
    rest are a handful of fp32 roundings, 2^-17 together.  The two are neighbours that share a reciprocal, or are not; a logit counts up to 2^100 : 1."""
    from flame_b200.ops.stickbreaking import sb_attention
    n, H = 12, 2
    q, k = torch.zeros(n, H, 64, device=DEV), torch.zeros(n, H, 64, device=DEV)
    q[:, :, 0], k[3, 0, 0], k[2 if nats < 40 else 5, 1, 0] = 16.0, nats / 2, -nats / 2   # logits +-nats, the others 0
    k[6, :, 0] = nats / 2 if nats < 40 else 0.0
    q, k, v = q.bfloat16(), k.bfloat16(), torch.randn(n, H, 64, device=DEV).bfloat16()
    o, rem = sb_attention(q, k, v, _meta([n]))
    logits = torch.einsum("ihd,jhd->hij", q.double(), k.double()) / 8
    stay = torch.nn.functional.logsigmoid(-logits).masked_fill(torch.ones(n, n, device=DEV, dtype=torch.bool).triu(), 0.0)
    want = stay.sum(-1).exp()
    rem = rem if rem.shape == want.shape else rem.t()
    assert want.min() > 1e-36
    assert ((rem.double() - want).abs() <= 2.0 ** -17 * want).all()


@pytest.mark.parametrize("left,right", [(42.0, 42.0), (16.0, 69.0), (69.0, 16.0), (60.0, 25.5), (69.0, 69.0), (80.0, 80.0), (5.0, 69.0)])
@pytest.mark.parametrize("at", [4, 5])
def test_stickbreaking_remainder_beside_two_dominating_neighbours(left, right, at):
    """Two large logits next to one another, at either place in a pair of keys: what they leave of a row, relative to itself down to 2^-124 (bound of
    the test above, twice), below 2^-123 where it is less; the weights of the keys around them likewise."""
    from flame_b200.ops.stickbreaking import sb_attention
    n = 10
    q, k, v = (torch.zeros(n, 1, 64, device=DEV) for _ in range(3))
    q[:, 0, 0], k[at, 0, 0], k[at + 1, 0, 0] = 16.0, left / 2, right / 2
    v[:, 0, :n] = torch.eye(n, device=DEV)     # outputs are the weights
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    o, rem = sb_attention(q, k, v, _meta([n]))
    rem = rem.reshape(n)
    logits = q[:, 0].double() @ k[:, 0].double().t() / 8
    logits = logits.clamp(max=100 * 0.6931471805599453)
    mask = torch.ones(n, n, device=DEV, dtype=torch.bool).triu()
    stay = torch.nn.functional.logsigmoid(-logits).masked_fill(mask, 0.0)
    want = stay.sum(-1).exp()
    att = ((torch.nn.functional.logsigmoid(logits) + stay.flip(-1).cumsum(-1).flip(-1) - stay).exp()).masked_fill(mask, 0.0)
    small = want < 2.0 ** -124
    assert ((rem.double() - want).abs() <= 2.0 ** -16 * want)[~small].all() and (rem[small] < 2.0 ** -123).all()
    got = o[:, 0, :n].double()
    assert ((got - att).abs() <= 2.0 ** -8 * att + 2.0 ** -123).all()


def test_short_conv_forward_backward():
    from flame_b200.ops import linear_attn as la
    from flame_b200.ops.conv import short_conv
    torch.manual_seed(8)
    meta = _meta([5, 300, 2, 1, 260])
    T, D, W = 568, 256, 4
    x = torch.randn(T, D, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(D, 1, W, device=DEV) * 0.5).to(torch.bfloat16).requires_grad_(True)
    b = torch.randn(D, device=DEV).to(torch.bfloat16).requires_grad_(True)
    for act, bias in (("silu", b), (None, None)):
        y = short_conv(x, w, bias, meta, act)
        xf, wf = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
        bf = bias.detach().float().requires_grad_(True) if bias is not None else None
        yr = la.short_conv(xf, wf, bf, meta, act)
        assert rel_err(y, yr) < 1e-2
        dy = torch.randn_like(y)
        grads = torch.autograd.grad(y, [x, w] + ([bias] if bias is not None else []), dy)
        refs = torch.autograd.grad(yr, [xf, wf] + ([bf] if bf is not None else []), dy.float())
        for g, r in zip(grads, refs):
            assert rel_err(g, r) < 2e-2


@pytest.mark.parametrize("D", [8, 40, 64, 96, 128, 192, 256, 264, 512, 1000, 2048, 2304, 4096, 7040])
@pytest.mark.parametrize("rows,form", [(1, "plain"), (37, "residual"), (37, "gate"), (700, "plain"), (5000, "residual")])
def test_rms_norm_every_row_length(D, rows, form):
    """Row lengths around the forms of the kernels (lanes of a warp, warps of a block), row counts that leave the last block ragged;
    bf16 results (2^-9) of fp32 arithmetic, weight gradients summed over the rows in fp32 and rounded once: 5e-3."""
    from flame_b200.ops.norm import rms_norm, rms_norm_gated
    torch.manual_seed(14)
    leaf = lambda *s: torch.randn(*s, device=DEV, dtype=torch.bfloat16).requires_grad_(True)  # noqa: E731
    x, o, w = leaf(rows, D), leaf(rows, D), leaf(D)
    dy, dr = torch.randn_like(x), torch.randn_like(x)
    xd, od, wd = (t.detach().double().requires_grad_(True) for t in (x, o, w))
    if form == "residual":
        out = list(rms_norm(x, w, 1e-6, o, True))
        r = (x.detach() + o.detach()).double().requires_grad_(True)   # the sum is stored in bf16 before it is normalised
        ref = [r * torch.rsqrt(r.pow(2).mean(-1, keepdim=True) + 1e-6) * wd, r]
        got = torch.autograd.grad(out, [x, w], [dy, dr])
        want = torch.autograd.grad(ref, [r, wd], [dy.double(), dr.double()])
    else:
        gate = o if form == "gate" else None
        out = [rms_norm_gated(x, o, w, 1e-6) if form == "gate" else rms_norm(x, w, 1e-6)]
        y = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * wd
        ref = [y * torch.nn.functional.silu(od) if gate is not None else y]
        got = torch.autograd.grad(out, [x, w] + ([o] if gate is not None else []), dy)
        want = torch.autograd.grad(ref, [xd, wd] + ([od] if gate is not None else []), dy.double())
    for a, b in zip(out + list(got), ref + list(want)):
        assert rel_err(a, b) < 5e-3


@pytest.mark.parametrize("D,lens", [(8, [1]), (136, [2, 3, 1, 4]), (120, [7, 57, 1]), (264, [64, 63, 65, 130]), (128, [4500, 3])])
@pytest.mark.parametrize("silu", [True, False])
def test_short_conv_width_four_edges(D, lens, silu):
    """Rows and channels around the block's tiles, documents shorter than the taps, a strided input, against fp64; bf16
    results of up to four taps (2^-9 each way), weight gradients summed in fp32 and rounded to bf16: 5e-3."""
    from flame_b200.ops.conv import short_conv
    torch.manual_seed(9)
    meta = _meta(lens)
    T = sum(lens)
    wide = torch.randn(T, 2 * D, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    w = (torch.randn(D, 1, 4, device=DEV) * 0.5).to(torch.bfloat16).requires_grad_(True)
    b = torch.randn(D, device=DEV).to(torch.bfloat16).requires_grad_(True)
    dy = torch.randn(T, D, device=DEV, dtype=torch.bfloat16)
    act = "silu" if silu else None
    y = short_conv(wide[:, D:], w, b, meta, act)
    out = [y] + list(torch.autograd.grad(y, [wide, w, b], dy))
    f = [t.detach().double().requires_grad_(True) for t in (wide, w, b)]
    x, pos = f[0][:, D:], meta.position_ids.long()
    yr = f[2].expand(T, D)
    for j in range(min(4, T)):
        shifted = torch.cat([x.new_zeros(j, D), x[:T - j]])
        yr = yr + torch.where((pos >= j)[:, None], shifted, torch.zeros_like(x)) * f[1][:, 0, 3 - j]
    yr = torch.nn.functional.silu(yr) if silu else yr
    ref = [yr] + list(torch.autograd.grad(yr, f, dy.double()))
    for a, r in zip(out, ref):
        assert rel_err(a, r) < 5e-3


@pytest.mark.parametrize("W", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("cols", [(0, 64), (16, 64), (3, 52)])
def test_short_conv_of_one_row(W, cols):
    """One token out of a wider matrix: torch calls such a row contiguous whatever its stride.  Against fp64, 5e-3 as above."""
    from flame_b200.ops import linear_attn as la
    from flame_b200.ops.conv import short_conv
    torch.manual_seed(W)
    (c, width), D, meta = cols, 32, _meta([1])
    wide = torch.randn(1, width, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    w, b = (torch.randn(*n, device=DEV, dtype=torch.bfloat16).requires_grad_(True) for n in ((D, 1, W), (D,)))
    dy = torch.randn(1, width, device=DEV, dtype=torch.bfloat16)[:, c:c + D]
    ins = [wide, w, b]
    y = short_conv(wide[:, c:c + D], w, b, meta, "silu")
    out = [y] + list(torch.autograd.grad(y, ins, dy))
    f = [t.detach().double().requires_grad_(True) for t in ins]
    yr = la.short_conv(f[0][:, c:c + D], f[1], f[2], meta, "silu")
    for a, r in zip(out, [yr] + list(torch.autograd.grad(yr, f, dy.double()))):
        assert rel_err(a, r) < 5e-3


@pytest.mark.parametrize("V", [8, 1000, 8192, 8200, 16384, 16392, 32000, 32768, 32776])
def test_cross_entropy_row_lengths(V):
    """Vocabularies around what a CTA holds in registers (and beyond, where it walks the row); ignored rows, a row with -inf
    entries, a large common offset; loss in fp32 (1e-5), gradients rounded to bf16 (2^-8)."""
    from flame_b200.ops.cross_entropy import cross_entropy
    torch.manual_seed(15)
    rows = 9
    base = (torch.randn(rows, V, device=DEV) * 3).to(torch.bfloat16)
    base[3] += 200.0
    base[4, ::2] = float("-inf")
    lab = torch.randint(0, V, (rows,), device=DEV)
    lab[1] = -100
    lab[4] = lab[4] // 2 * 2 + 1
    ref_in = base.double().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(ref_in, lab)
    (want,) = torch.autograd.grad(ref, ref_in)
    leaf = base.clone().requires_grad_(True)
    loss = cross_entropy(leaf * 1.0, lab)
    (got,) = torch.autograd.grad(loss, leaf)
    assert abs(loss.item() - ref.item()) < 1e-5 * abs(ref.item()) + 1e-6
    assert rel_err(got, want) < 4e-3


@pytest.mark.parametrize("V", [1024, 1032, 2048, 2056, 4096, 4104, 12296])
def test_cross_entropy_by_threads_of_a_row(V):
    """Rows around the lengths at which a row's CTA changes its threads or vectors, against 64 bits entry by entry: three roundings of
    fp32 and two exponentials (2^-18), and bf16 twice, in the gradient and in its product with the loss's gradient (2^-7).  A row with
    its target in the first and one in the last vector, an ignored row with a target inside, a row of NaN, one with +inf."""
    from flame_b200.ops.cross_entropy import cross_entropy
    torch.manual_seed(V)
    rows = 303
    base = (torch.randn(rows, V, device=DEV) * 4).to(torch.bfloat16)
    lab = torch.randint(0, V, (rows,), device=DEV)
    lab[0], lab[1], lab[2] = 0, V - 1, 5
    lab[lab == 5] = 6
    lab[2] = 5
    base[3, 7] = float("-inf")
    ref_in = base.double().requires_grad_(True)
    (want,) = torch.autograd.grad(torch.nn.functional.cross_entropy(ref_in, lab, ignore_index=5), ref_in)
    leaf = base.clone().requires_grad_(True)
    loss = cross_entropy(leaf * 1.0, lab, ignore_index=5)
    (got,) = torch.autograd.grad(loss, leaf, torch.tensor(0.75, device=DEV))
    size = want.abs() + (lab[:, None] == torch.arange(V, device=DEV)) / rows  # (p - 1: the difference keeps the error of p and 1)
    assert ((got.double() - 0.75 * want).abs() <= 2.0 ** -7 * 0.75 * want.abs() + 2.0 ** -18 * size).all()
    base[4, 9], base[5, V - 1] = float("nan"), float("inf")
    leaf = base.clone().requires_grad_(True)
    loss = cross_entropy(leaf * 1.0, lab, ignore_index=5)
    (bad,) = torch.autograd.grad(loss, leaf)
    assert loss.isnan() and bad[4].isnan().all() and bad[5, V - 1].isnan()
    rest = torch.arange(rows, device=DEV) > 5
    assert torch.equal((bad[rest].float() * 0.75).to(torch.bfloat16), got[rest])


@pytest.mark.parametrize("V", [1000, 4096, 32000])
@pytest.mark.parametrize("spread", [1.0, 20.0, 100.0])
def test_cross_entropy_exponentials_far_below_the_maximum(V, spread):
    """Logits down to 100 below the row's largest, loss and gradient against 64 bits.  __expf(y) is documented to be good to 2 + 1.173 |y| units
    in the last place (2^-23); a gradient is that of its entry and that of the sum (of entries near the maximum, and V roundings),
    two products, and bf16 twice (2^-7)."""
    from flame_b200.ops.cross_entropy import cross_entropy
    torch.manual_seed(V)
    rows = 67
    base = (-torch.rand(rows, V, device=DEV) * spread).to(torch.bfloat16)
    base[:, 3] = 0.0
    base[1] = -100.0
    base[1, 8] = 0.0
    lab = torch.randint(0, V, (rows,), device=DEV)
    lab[2] = 3
    ref = base.double().requires_grad_(True)
    want_loss = torch.nn.functional.cross_entropy(ref, lab, reduction="none")
    leaf = base.clone().requires_grad_(True)
    loss = cross_entropy(leaf * 1.0, lab)
    (got,) = torch.autograd.grad(loss, leaf)
    (want,) = torch.autograd.grad(want_loss.mean(), ref)
    loss, want_loss = loss.item(), want_loss.mean().item()
    y = ref.detach() - ref.detach().amax(1, keepdim=True)
    p = y.exp() / y.exp().sum(1, keepdim=True)
    of_exp = (2 + 1.173 * y.abs()) * 2.0 ** -23
    of_sum = (p * of_exp).sum(1, keepdim=True) + 2.0 ** -18   # at most 64 entries one after the other in a thread, then shuffles
    bound = 2.0 ** -7 * want.abs() + (p * (of_exp + of_sum + 2.0 ** -22) + 2.0 ** -23 * (lab[:, None] == torch.arange(V, device=DEV))) / rows
    assert ((got.double() - want).abs() <= bound + 1.2e-38).all()
    assert abs(loss - want_loss) <= of_sum.max().item() + 2.0 ** -21 * want_loss


@pytest.mark.parametrize("n", [1, 7, 8, 4096, 100003])
def test_gradient_of_the_loss_as_a_factor(n):
    """The product with the scalar in device memory equals that of two bf16 tensors bit for bit; other forms take the tensors'."""
    from flame_b200.ops.cross_entropy import _times
    torch.manual_seed(n)
    g, s = torch.randn(n, device=DEV).to(torch.bfloat16), torch.tensor(0.3, device=DEV)
    want = g * s.to(torch.bfloat16)
    with torch.no_grad():
        assert torch.equal(_times(g, s), want)
        odd = torch.empty(n + 1, dtype=torch.bfloat16, device=DEV)[1:].copy_(g)
        assert torch.equal(_times(odd, s), want)
        both = torch.vmap(lambda f: _times(g, f))(torch.stack([s, -s]))
        assert torch.equal(both[0], want) and torch.equal(both[1], -want)
    f = s.clone().requires_grad_(True)
    (d,) = torch.autograd.grad(_times(g, f).float().sum(), f)
    assert d is not None


def test_embedding_backward_runs_of_ids():
    """Runs of one id longer than a warp, ids outside the table (another rank's vocabulary slice), against index_add in fp64."""
    from flame_b200.ops.embedding import embedding
    torch.manual_seed(16)
    V, D = 50, 136
    ids = torch.cat([torch.full((100,), 7), torch.randint(0, V, (333,)), torch.full((64,), 49), torch.tensor([-3, V, V + 9, 0])]).to(DEV)
    ids = ids[torch.randperm(ids.numel(), device=DEV)]
    w = torch.randn(V, D, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    y = embedding(ids, w)
    dy = torch.randn_like(y)
    (dw,) = torch.autograd.grad(y, w, dy)
    keep = (ids >= 0) & (ids < V)
    ref = torch.zeros(V, D, device=DEV, dtype=torch.float64).index_add_(0, ids[keep], dy[keep].double())
    assert rel_err(dw, ref) < 4e-3
    assert torch.equal(y[~keep], torch.zeros_like(y[~keep]))


@pytest.mark.parametrize("H,Hkv,window", [(3, 3, 0), (4, 2, 100)])
def test_fused_qkv_attention_head_dim_128(H, Hkv, window):
    """Rotary attention of head dim 128 on the fused projection buffer against the definition on its slices, in fp32; ragged
    documents (bf16 operands: 2e-2)."""
    from flame_b200.ops.attention import attention_reference
    from flame_b200.ops.attn_block import qkv_attention
    from flame_b200.ops.rope import rope_reference, rope_tables
    torch.manual_seed(17)
    meta = _meta([300, 1, 77])
    T, Dh = 378, 128
    qkv = torch.randn(T, (H + 2 * Hkv) * Dh, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    rope = rope_tables(Dh, 512, 10000.0, torch.device(DEV))
    do = torch.randn(T, H * Dh, device=DEV, dtype=torch.bfloat16)
    o = qkv_attention(qkv, meta, H, Hkv, Dh, rope=rope, window=window)
    (got,) = torch.autograd.grad(o, qkv, do)
    f = qkv.detach().float().requires_grad_(True)
    q, k, v = f[:, :H * Dh].view(T, H, Dh), f[:, H * Dh:(H + Hkv) * Dh].view(T, Hkv, Dh), f[:, (H + Hkv) * Dh:].view(T, Hkv, Dh)
    q, k = rope_reference(q, meta.position_ids, *rope), rope_reference(k, meta.position_ids, *rope)
    ref = attention_reference(q, k, v, meta, Dh ** -0.5, window).reshape(T, H * Dh)
    (want,) = torch.autograd.grad(ref, f, do.float())
    assert rel_err(o, ref) < 2e-2 and rel_err(got, want) < 2e-2


@pytest.mark.parametrize("Dh", [64, 128])
@pytest.mark.parametrize("offset", [0, 3])
def test_fused_qkv_attention_leaves_its_input_alone(Dh, offset):
    """Two calls on one buffer (at any storage offset) give one result and keep the buffer; giving the buffer away changes neither
    result nor gradient: the same kernels on the same rotated values, so bit for bit (but for dq's fp32 sums: their order)."""
    from flame_b200.ops.attn_block import qkv_attention
    from flame_b200.ops.rope import rope_tables
    torch.manual_seed(18)
    meta, T, H, Hkv = _meta([200, 1, 77]), 278, 4, 2
    n = (H + 2 * Hkv) * Dh
    leaf = torch.empty(T * n + offset, device=DEV, dtype=torch.bfloat16).normal_()[offset:].view(T, n).requires_grad_(True)
    before = leaf.detach().clone()
    rope = rope_tables(Dh, 512, 10000.0, torch.device(DEV))
    do = torch.randn(T, H * Dh, device=DEV, dtype=torch.bfloat16)
    got = []
    for buf, own in ((leaf, False), (leaf, False), (leaf * 1.0, True)):
        o = qkv_attention(buf, meta, H, Hkv, Dh, rope=rope, own=own)
        got.append((o.detach(), *torch.autograd.grad(o, leaf, do)))
    assert torch.equal(leaf.detach(), before)
    for o, g in got[1:]:
        assert torch.equal(o, got[0][0])
        assert (g - got[0][1]).abs().max() <= 2.0 ** -8 * got[0][1].abs().max()


def test_fused_linear_cross_entropy_and_cross_entropy():
    from flame_b200.ops.cross_entropy import cross_entropy, fused_linear_cross_entropy
    torch.manual_seed(5)
    T, D, V = 3000, 256, 32000
    x = (torch.randn(T, D, device=DEV) * 0.5).to(torch.bfloat16).requires_grad_(True)
    w = (torch.randn(V, D, device=DEV) * 0.05).to(torch.bfloat16).requires_grad_(True)
    lab = torch.randint(0, V, (T,), device=DEV)
    lab[::7] = -100
    loss = fused_linear_cross_entropy(x, w, lab, chunk=1024)
    xf, wf = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(xf @ wf.t(), lab, ignore_index=-100)
    assert abs(loss.item() - ref.item()) / ref.item() < 5e-3
    loss.backward()
    ref.backward()
    assert rel_err(x.grad, xf.grad) < 3e-2 and rel_err(w.grad, wf.grad) < 3e-2
    logits = (xf.detach() @ wf.detach().t()).to(torch.bfloat16).requires_grad_(True)
    lf = logits.detach().float().requires_grad_(True)
    l2 = cross_entropy(logits.clone().requires_grad_(True), lab)
    r2 = torch.nn.functional.cross_entropy(lf, lab, ignore_index=-100)
    assert abs(l2.item() - r2.item()) / r2.item() < 5e-3


def test_adamw_matches_torch_and_skips_nan():
    from flame_b200.ops import optim as O
    torch.manual_seed(6)
    n = 100003
    p0 = torch.randn(n, device=DEV)
    g = torch.randn(n, device=DEV) * 3
    p, m, v = p0.clone(), torch.zeros(n, device=DEV), torch.zeros(n, device=DEV)
    lowp = torch.empty(n, device=DEV, dtype=torch.bfloat16)
    ctrl = torch.zeros(O.CTRL_SIZE, device=DEV)
    ref = torch.nn.Parameter(p0.clone())
    opt = torch.optim.AdamW([ref], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    for _ in range(3):
        O.sumsq_accumulate(g, ctrl[0:1], accumulate=False)
        O.adamw_step(p, m, v, g, lowp, ctrl, 1e-2, 0.9, 0.95, 1e-8, 0.1, 1.0, True)
        O.adamw_finalize(ctrl, 1.0, True)
        ref.grad = g.clone()
        torch.nn.utils.clip_grad_norm_([ref], 1.0)
        opt.step()
    assert rel_err(p, ref.detach()) < 1e-5
    assert rel_err(lowp, ref.detach()) < 1e-2
    assert int(ctrl[O.CTRL_STEP]) == 3
    before = p.clone()
    ctrl[0] = float("nan")
    O.adamw_step(p, m, v, g, lowp, ctrl, 1e-2, 0.9, 0.95, 1e-8, 0.1, 1.0, True)
    O.adamw_finalize(ctrl, 1.0, True)
    assert torch.equal(p, before) and int(ctrl[O.CTRL_SKIPPED]) == 1 and int(ctrl[O.CTRL_STEP]) == 3


def test_transformer_block_matches_reference_path():
    """The whole model on kernels vs the same weights through the PyTorch reference ops (fp32)."""
    import os
    from flame_b200.models import ModelConfig, build_model
    cfg = ModelConfig("transformer", hidden_size=256, num_hidden_layers=2, num_heads=4, vocab_size=1024,
                      max_position_embeddings=4096)
    torch.manual_seed(7)
    m32 = build_model(cfg, device=DEV, dtype=torch.float32, seed=3)
    mbf = build_model(cfg, device=DEV, dtype=torch.bfloat16, init=False)
    mbf.load_state_dict({k: v.to(torch.bfloat16) for k, v in m32.state_dict().items()})
    ids = torch.randint(3, 1024, (1, 1500), device=DEV)
    cu = torch.tensor([0, 600, 601, 1500], dtype=torch.int32)
    a = m32(input_ids=ids, labels=ids, cu_seqlens=cu).loss
    b = mbf(input_ids=ids, labels=ids, cu_seqlens=cu).loss
    assert abs(a.item() - b.item()) / a.item() < 2e-2
    a.backward()
    b.backward()
    ga = m32.model.layers[0].attn.q_proj.weight.grad
    gb = mbf.model.layers[0].attn.q_proj.weight.grad
    assert rel_err(gb, ga) < 8e-2


def test_smoke_entry():
    import __graft_entry__ as ge
    ge.smoke()


def test_operator_level_selective_checkpointing_on_the_kernel_path():
    """``selective op``: the recomputation replays the kept GEMM / attention outputs; same loss and gradients as no AC."""
    from flame_b200.models import ModelConfig, build_model
    from flame_b200.parallel import OptimConfig, ParallelDims, ShardedEngine
    from flame_b200.parallel.parallelize import apply_activation_checkpointing
    cfg = ModelConfig("transformer", hidden_size=256, num_hidden_layers=2, num_heads=4, vocab_size=512)
    ids = torch.randint(3, 512, (1, 384), device=DEV, generator=torch.Generator(DEV).manual_seed(3))
    meta = _meta([100, 128, 96, 60])
    grads, losses = [], []
    for option in (None, "op"):
        model = build_model(cfg, device="meta", dtype=torch.bfloat16, init=False)
        if option:
            apply_activation_checkpointing(model, "selective", option)
        eng = ShardedEngine(model, ParallelDims(world_size=1), torch.device(DEV), torch.bfloat16, OptimConfig())
        eng.init_weights(0)
        model.train()
        eng.zero_grad()
        n0 = _lib_launches()
        loss = model(input_ids=ids, labels=ids, meta=meta).loss
        loss.backward()
        losses.append(float(loss))
        launches = _lib_launches() - n0
        losses.append(launches)
        for u in eng.units:
            eng._fold_autograd_grads(u)      # gradients that came back through autograd join the flat fp32 buffer
        grads.append(eng.grad_all.clone())
    assert losses[0] == losses[2]
    assert rel_err(grads[1], grads[0]) < 2e-3
    assert losses[3] > losses[1]             # the recomputation did launch kernels (norms, the 2nd and 4th products, ...)
    # fewer launches than a full recomputation would add: the kept products and the attention are not run again
    assert losses[3] - losses[1] < losses[1]


def _lib_launches():
    from flame_b200.ops import _lib
    return _lib.launches()


@pytest.mark.parametrize("opts", [dict(label_smoothing=0.1), dict(logit_scale=0.5, lse_square_scale=1e-3),
                                  dict(logit_softcapping=20.0, label_smoothing=0.05, lse_square_scale=1e-4)])
def test_cross_entropy_options_match_the_written_out_loss(opts):
    """Label smoothing, logit scale, z-loss and soft-capping (fla/modules/fused_cross_entropy.py:374-400) in the CE kernel
    and through the chunked linear + CE head, against the fp32 formula."""
    from flame_b200.ops.cross_entropy import CEOptions, cross_entropy, cross_entropy_reference, fused_linear_cross_entropy
    torch.manual_seed(6)
    T, D, V = 777, 128, 4096
    x = (torch.randn(T, D, device=DEV) * 0.7).to(torch.bfloat16).requires_grad_(True)
    w = (torch.randn(V, D, device=DEV) * 0.2).to(torch.bfloat16).requires_grad_(True)
    lab = torch.randint(0, V, (T,), device=DEV)
    lab[::13] = -100
    opt = CEOptions(**opts)
    xf, wf = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    ref = cross_entropy_reference(xf @ wf.t(), lab, -100, opt)
    ref.backward()
    loss = fused_linear_cross_entropy(x, w, lab, chunk=256, **opts)
    loss.backward()
    assert abs(loss.item() - ref.item()) < 2e-2 * abs(ref.item())
    assert rel_err(x.grad, xf.grad) < 3e-2 and rel_err(w.grad, wf.grad) < 3e-2
    logits = (xf.detach() @ wf.detach().t()).to(torch.bfloat16).requires_grad_(True)
    lf = logits.detach().float().requires_grad_(True)
    cross_entropy_reference(lf, lab, -100, opt).backward()
    out = cross_entropy(logits.clone().detach().requires_grad_(True), lab, **opts)
    lg2 = logits.detach().clone().requires_grad_(True)
    out = cross_entropy(lg2, lab, **opts)
    out.backward()
    assert abs(out.item() - cross_entropy_reference(lf.detach(), lab, -100, opt).item()) < 1e-2 * abs(out.item())
    assert rel_err(lg2.grad, lf.grad) < 3e-2


def test_gate_up_projection_with_swiglu_epilogue():
    """The fused gate | up GEMM with the activation in its epilogue against the GEMM followed by the SwiGLU kernel."""
    from flame_b200.ops.activations import swiglu
    from flame_b200.ops.linear import gate_up_swiglu, linear_fused
    torch.manual_seed(12)
    T, K, I = 1000, 512, 1408   # T not a multiple of the tile, I = 11 x 128
    flat = (torch.randn(2 * I * K, device=DEV) * 0.05).to(torch.bfloat16)
    wg = flat[: I * K].view(I, K).requires_grad_(True)
    wu = flat[I * K:].view(I, K).requires_grad_(True)
    x = torch.randn(T, K, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    z = gate_up_swiglu(x, wg, wu)
    assert z is not None and z.shape == (T, I)
    ref = swiglu(linear_fused(x.detach(), [wg.detach(), wu.detach()]))
    assert rel_err(z, ref) < 2e-3
    dz = torch.randn_like(z)
    z.backward(dz)
    xf, gf, uf = (t.detach().float().requires_grad_(True) for t in (x, wg, wu))
    zr = torch.nn.functional.silu(xf @ gf.t()) * (xf @ uf.t())
    zr.backward(dz.float())
    assert rel_err(x.grad, xf.grad) < 2e-2 and rel_err(wg.grad, gf.grad) < 2e-2 and rel_err(wu.grad, uf.grad) < 2e-2


@pytest.mark.parametrize("T,K,I,grads", [(1, 64, 128, "autograd"), (255, 64, 384, "adjacent"), (257, 72, 128, "apart"), (1000, 512, 1408, "adjacent"),
                                         (20000, 128, 256, "autograd"), (300, 64, 384, "hooks"), (300, 64, 384, "frozen")])
def test_gated_mlp_in_one_node(T, K, I, grads):
    """Both activations in the products' epilogues against 64 bits, over partial tiles in rows and columns, several rounds of tiles, and
    every way the weights' gradients go.  Operands and results of bf16, sums of up to 1,408 terms: each output within a few 2^-8 of
    itself."""
    from flame_b200.ops import linear as ops
    torch.manual_seed(13)
    flat = (torch.randn(3 * I * K, device=DEV) * K ** -0.5).to(torch.bfloat16)
    ws = [torch.nn.Parameter(flat[i * I * K:(i + 1) * I * K].view(*((I, K) if i < 2 else (K, I)))) for i in range(3)]
    if grads in ("adjacent", "apart"):
        acc = torch.ones(3, 2 * I * K, device=DEV)
        for i, w in enumerate(ws):
            w.main_grad = (acc.view(-1)[i * I * K:(i + 1) * I * K] if grads == "adjacent" else acc[i, :I * K]).view(w.shape)
    if grads == "frozen":
        ws[0].requires_grad_(False), ws[2].requires_grad_(False)
    x = torch.randn(T, 2 * K, device=DEV, dtype=torch.bfloat16)[:, K:].requires_grad_(True)   # rows apart
    dy = torch.randn(T, K + 3, device=DEV, dtype=torch.bfloat16)[:, 3:]                       # rows that start between vectors
    pack = (lambda t: t.clone()) if grads == "hooks" else (lambda t: t)
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        y = ops.gated_mlp(x, *ws)
    y.backward(dy)
    xr, *wr = (t.detach().double().requires_grad_(True) for t in (x, *ws))
    yr = (torch.nn.functional.silu(xr @ wr[0].t()) * (xr @ wr[1].t())) @ wr[2].t()
    yr.backward(dy.double())
    assert rel_err(y, yr) < 1e-2 and rel_err(x.grad, xr.grad) < 1.5e-2
    for i, (w, r) in enumerate(zip(ws, wr)):
        if not w.requires_grad:
            assert w.grad is None
            continue
        assert rel_err(w.main_grad - 1 if hasattr(w, "main_grad") else w.grad, r.grad) < 1.5e-2
    if grads == "apart":
        assert torch.equal(acc[:, I * K:], torch.ones(3, I * K, device=DEV))


@pytest.mark.parametrize("how", ["hook", "bias"])
def test_mlp_whose_down_projection_is_a_call_of_its_own(how):
    """A hook on the down projection is called, a bias of its own is added, and all else equals the MLP in one node bit for bit."""
    from flame_b200.models.modules import GatedMLP
    from flame_b200.ops import linear as ops
    torch.manual_seed(3)
    D, I, T = 64, 256, 300
    flat = (torch.randn(3 * I * D, device=DEV) * 0.1).to(torch.bfloat16)
    mlp = GatedMLP(D, I)
    for i, m in enumerate((mlp.gate_proj, mlp.up_proj, mlp.down_proj)):
        m.weight = torch.nn.Parameter(flat[i * I * D:(i + 1) * I * D].view(m.weight.shape))
    x, dy = (torch.randn(T, D, device=DEV).to(torch.bfloat16).requires_grad_(i == 0) for i in range(2))
    ins = [x, mlp.gate_proj.weight, mlp.up_proj.weight, mlp.down_proj.weight]
    assert ops.gated_mlp(*ins) is not None
    want = mlp(x)
    grads = torch.autograd.grad(want, ins, dy)
    seen = []
    if how == "hook":
        mlp.down_proj.register_forward_hook(lambda m, i, o: seen.append(i[0].shape))
    else:
        mlp.down_proj.bias = torch.nn.Parameter(torch.ones(D, device=DEV, dtype=torch.bfloat16))
    got = mlp(x)
    again = torch.autograd.grad(got, ins, dy)
    assert seen == [(T, I)] * (how == "hook")
    assert torch.equal(got, want) if how == "hook" else rel_err(got, want.float() + 1) < 2 ** -8
    assert all(torch.equal(a, b) for a, b in zip(again, grads))


@pytest.mark.parametrize("grads", ["autograd", "main_grad"])
@pytest.mark.parametrize("reentrant", [False, True])
def test_mlp_in_one_node_under_activation_checkpointing(grads, reentrant):
    """Recomputed in the backward pass, where the saved weights are other tensors than the parameters: output and gradients, which go to
    main_grad or to autograd, equal those without, bit for bit."""
    from torch.utils.checkpoint import checkpoint
    from flame_b200.ops import linear as ops
    torch.manual_seed(4)
    D, I, T = 64, 256, 300
    flat = (torch.randn(3 * I * D, device=DEV) * 0.1).to(torch.bfloat16)
    x, dy = (torch.randn(T, D, device=DEV).to(torch.bfloat16) for _ in range(2))

    def run(fn):
        ws = [torch.nn.Parameter(flat[i * I * D:(i + 1) * I * D].view((I, D) if i < 2 else (D, I))) for i in range(3)]
        acc = torch.zeros(3 * I * D, device=DEV)
        if grads == "main_grad":
            for i, w in enumerate(ws):
                w.main_grad = acc[i * I * D:(i + 1) * I * D].view(w.shape)
        leaf = x.clone().requires_grad_(True)
        y = fn(lambda t: ops.gated_mlp(t, *ws), leaf)
        y.backward(dy)
        assert all((w.grad is None) == (grads == "main_grad") for w in ws)
        return [y.detach(), leaf.grad, acc] + [w.grad for w in ws if w.grad is not None]

    want = run(lambda f, t: f(t))
    assert want[2].any() == (grads == "main_grad")
    assert all(torch.equal(a, b) for a, b in zip(run(lambda f, t: checkpoint(f, t, use_reentrant=reentrant)), want))


@pytest.mark.parametrize("covered", [True, False])
def test_mlp_in_one_node_whose_weights_are_still_to_be_gathered(covered):
    """The unit's weights lie in a shard (of a world of one) and their place holds NaN: the first product of the forward pass that reads them
    fetches them on its way, and so does the backward's; a gather that does not cover the weight is flushed before.  All bits as with
    the weights in place, and no gather is left behind."""
    import numpy as np
    from flame_b200.ops import gemm, linear as ops
    torch.manual_seed(5)
    D, I, T, shift = 256, 384, 700, 14
    n = 3 * I * D
    shard = (torch.randn(n, device=DEV) * 0.1).to(torch.bfloat16)
    assert n * 2 % (1 << shift) == 0
    flat = shard.clone()
    ws = [torch.nn.Parameter(flat[i * I * D:(i + 1) * I * D].view((I, D) if i < 2 else (D, I))) for i in range(3)]
    x, dy = (torch.randn(T, D, device=DEV).to(torch.bfloat16).requires_grad_(i == 0) for i in range(2))
    want = ops.gated_mlp(x, *ws)
    grads = torch.autograd.grad(want, [x, *ws], dy)
    flags, flushed = torch.zeros((n * 2 >> shift) + 1, dtype=torch.int32, device=DEV), []

    def pend(epoch, lo, hi):
        flat.data.fill_(float("nan"))

        def flush():
            flat.data.copy_(shard)
            p.done = True
            gemm.set_pending_gather(None)
            flushed.append(epoch)
        p = gemm.PendingGather(None, flat.data_ptr(), lo, hi, np.array([shard.data_ptr()], dtype=np.uint64), 1, 0, n * 2, shift, flags, epoch, flush)
        gemm.set_pending_gather(p)
        return p

    try:
        first = pend(1, 0, n * 2 if covered else I * D * 2)                       # not covered: ends before the up projection
        got = ops.gated_mlp(x, *ws)
        assert first.done and torch.equal(got, want) and flushed == ([] if covered else [1])
        second = pend(2, 0 if covered else n * 2 - 16, n * 2)                     # not covered: begins inside the down projection
        again = torch.autograd.grad(got, [x, *ws], dy)
        assert second.done and all(torch.equal(a, b) for a, b in zip(again, grads)) and flushed == ([] if covered else [1, 2])
        assert torch.equal(flat, shard)
    finally:
        gemm.set_pending_gather(None)


@pytest.mark.gpu
@pytest.mark.parametrize("with_lb", [False, True])
def test_hgrn2_gate_kernels_match_the_elementwise_chain(with_lb):
    """fla/layers/hgrn2.py:160-190 as one kernel each way, against the fp32 PyTorch expressions."""
    from flame_b200.ops.gates import hgrn2_gates, hgrn2_gates_reference
    torch.manual_seed(3)
    T, D = 1000, 512
    dev = torch.device("cuda")
    q_raw = (torch.randn(T, D, device=dev) * 2).bfloat16().requires_grad_(True)
    f_raw = (torch.randn(T, D, device=dev) * 3).bfloat16().requires_grad_(True)
    lb = (torch.rand(D, device=dev) * 0.5 + 0.01).requires_grad_(True) if with_lb else None
    q, k, g = hgrn2_gates(q_raw, f_raw, lb)
    wq, wk, wg = torch.randn_like(q), torch.randn_like(k), torch.randn_like(g)
    ((q.float() * wq.float()).sum() + (k.float() * wk.float()).sum() + (g * wg).sum()).backward()
    got = [q_raw.grad.float(), f_raw.grad.float()] + ([lb.grad.float()] if with_lb else [])
    q32 = q_raw.detach().float().requires_grad_(True)
    f32 = f_raw.detach().float().requires_grad_(True)
    lb32 = lb.detach().clone().requires_grad_(True) if with_lb else None
    qr, kr, gr = hgrn2_gates_reference(q32, f32, lb32)
    ((qr * wq.float()).sum() + (kr * wk.float()).sum() + (gr * wg).sum()).backward()
    want = [q32.grad, f32.grad] + ([lb32.grad] if with_lb else [])
    assert torch.allclose(q.float(), qr, atol=2e-2, rtol=2e-2)
    assert torch.allclose(k.float(), kr, atol=1e-2, rtol=2e-2)
    assert torch.allclose(g, gr, atol=1e-4, rtol=1e-4)
    for a, b in zip(got, want):
        err = (a - b).abs().max() / b.abs().max().clamp_min(1e-6)
        assert err < 2e-2, err


@pytest.mark.gpu
def test_mamba2_glue_kernels_match_the_elementwise_chain():
    """fla/layers/mamba2.py:241-331: softplus(dt + bias), x dt, the log decay, the D skip and the silu(z) gate as two
    kernels each way, on strided column views of the projection output like the layer uses them."""
    from flame_b200.ops import gates
    torch.manual_seed(5)
    T, H, P, N = 777, 4, 64, 32
    dev = torch.device("cuda")
    Di, conv_dim = H * P, H * P + 2 * N
    big = (torch.randn(T, Di + conv_dim + H, device=dev) * 1.5).bfloat16().requires_grad_(True)
    conv_out = torch.randn(T, conv_dim, device=dev).bfloat16().requires_grad_(True)
    dt_bias = torch.randn(H, device=dev).requires_grad_(True)
    A_log = torch.rand(H, device=dev).requires_grad_(True)
    D = torch.randn(H, device=dev).requires_grad_(True)
    y_in = torch.randn(T, H, P, device=dev).bfloat16().requires_grad_(True)
    w1, w2, w3, w4 = (torch.randn(T, H, P, device=dev), torch.randn(T, H, device=dev), torch.randn(T, H, device=dev),
                      torch.randn(T, Di, device=dev))

    def run(use_kernel):
        for t in (big, conv_out, dt_bias, A_log, D, y_in):
            t.grad = None
        z, _, dt_raw = gates.split_columns(big, (Di, conv_dim, H))
        xs, _, _ = gates.split_columns(conv_out, (Di, N, N))
        pre = gates.mamba2_pre if use_kernel else gates.mamba2_pre_reference
        post = gates.mamba2_post if use_kernel else gates.mamba2_post_reference
        xv, dt, g = pre(xs, dt_raw, dt_bias, A_log, H, P)
        out = post(y_in, xs, z, D, H, P)
        loss = (xv.float() * w1).sum() + (dt * w2).sum() + (g * w3).sum() + (out.float() * w4).sum()
        loss.backward()
        return ([xv.float(), dt, g, out.float()],
                [t.grad.float().clone() for t in (big, conv_out, dt_bias, A_log, D, y_in)])

    outs_k, grads_k = run(True)
    outs_r, grads_r = run(False)
    for a, b in zip(outs_k, outs_r):
        assert rel_err(a, b) < 1e-2
    for a, b in zip(grads_k, grads_r):
        assert rel_err(a, b) < 2e-2, rel_err(a, b)


@pytest.mark.parametrize("with_slots", [False, True])
@pytest.mark.parametrize("shape", [(1, 8), (3, 5, 8), (77, 4, 64)])
def test_logsigmoid_gate(shape, with_slots):
    """One pass against torch in fp64: the results are fp32 (a few ulp of __expf and log1pf; 1 - exp(g) loses none to
    cancellation), the gradient is rounded to bf16 once (2^-9 relative)."""
    from flame_b200.ops.gates import logsigmoid_gate
    torch.manual_seed(0)
    x = (torch.randn(*shape, device="cuda") * 6).bfloat16()
    x.view(-1)[:4] = torch.tensor([60.0, -60.0, 0.0, -1e4])
    x.requires_grad_(True)
    xr = x.detach().double().requires_grad_(True)
    got = logsigmoid_gate(x, 16.0, with_slots)
    want = torch.nn.functional.logsigmoid(xr) / 16.0
    got = got if with_slots else (got,)
    wants = (want, 1 - want.exp()) if with_slots else (want,)
    grads = [torch.randn_like(g) for g in got]
    for g, w in zip(got, wants):
        assert g.dtype == torch.float32 and ((g.double() - w).abs() <= 2e-6 * w.abs() + 1e-9).all()
    dx, = torch.autograd.grad(got, x, grads)
    dw, = torch.autograd.grad(wants, xr, [g.double() for g in grads])
    scale = sum(g.double().abs() for g in grads) / 16 * torch.sigmoid(-xr.detach())
    assert ((dx.double() - dw).abs() <= 2.0 ** -8 * dw.abs() + 1e-5 * scale + 1e-9).all()


@pytest.mark.parametrize("with_bias", [False, True])
@pytest.mark.parametrize("M", [1, 31, 128, 200, 520])
@pytest.mark.parametrize("N", [8, 40, 64, 72, 256, 264])
def test_gemm_result_boxes(M, N, with_bias):
    """bf16 results at the edges of the boxes that leave by TMA (32 rows x 64 columns; tiles of 256 and of 128 rows), in storage
    whose neighbours stay untouched; fp32 sums of K = 72 products and one bf16 rounding (2^-9 relative)."""
    from flame_b200.ops.gemm import gemm_nt
    torch.manual_seed(M * 1000 + N)
    K = 72
    a, b = torch.randn(M, K, device=DEV).bfloat16(), torch.randn(N, K, device=DEV).bfloat16()
    bias = torch.randn(N + 1, device=DEV).bfloat16()
    want = 0.5 * (a.double() @ b.double().t())
    size = a.double().abs() @ b.double().abs().t()
    for offset in (0, 1) if with_bias else (0,):   # an unaligned bias takes scalar loads
        bb = bias[offset:offset + N] if with_bias else None
        store = torch.full((M + 2, (N + 7) // 8 * 8 + 8), 7.0, dtype=torch.bfloat16, device=DEV)
        gemm_nt(a, b, out=store[1:M + 1, :N], alpha=0.5, bias=bb)
        ref = want + bb.double() if with_bias else want
        got = store[1:M + 1, :N].double()
        assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -17 * size + 1e-30).all()
        store[1:M + 1, :N] = 7.0
        assert (store == 7.0).all()


@pytest.mark.parametrize("activation", ["silu", None])
@pytest.mark.parametrize("T,D", [(1, 8), (67, 72), (1333, 2048), (2500, 4096)])
def test_short_conv_strips(T, D, activation):
    """Width 4, strips of one and of several 64-row tiles, ragged ends, documents shorter than the taps; against torch in fp32.
    Outputs and dx are rounded to bf16 once (2^-9); dw and db sum T products in fp32 and are rounded once."""
    from flame_b200.ops.conv import short_conv
    torch.manual_seed(T + D)
    lens, left = [], T
    for n in [1, 2, 3, 70, 1] + [509] * 9:
        lens.append(min(n, left))
        left -= lens[-1]
        if left == 0:
            break
    meta = _meta(lens)
    x, dy = torch.randn(T, D, device=DEV).bfloat16().requires_grad_(True), torch.randn(T, D, device=DEV).bfloat16()
    w, b = (torch.randn(D, 1, 4, device=DEV) * 0.4).bfloat16().requires_grad_(True), torch.randn(D, device=DEV).bfloat16().requires_grad_(True)
    y = short_conv(x, w, b, meta, activation)
    got = torch.autograd.grad(y, [x, w, b], dy)
    xr, wr, br = (t.detach().double().requires_grad_(True) for t in (x, w, b))
    parts, c = [], 0
    for n in lens:
        z = torch.nn.functional.conv1d(torch.nn.functional.pad(xr[c:c + n].t()[None], (3, 0)), wr, br, groups=D)[0].t()
        parts.append(torch.nn.functional.silu(z) if activation else z)
        c += n
    want_y = torch.cat(parts)
    want = torch.autograd.grad(want_y, [xr, wr, br], dy.double())
    assert rel_err(y, want_y) < 3e-3
    for g, r in zip(got, want):
        assert rel_err(g, r) < 5e-3


def test_short_conv_backward_needs_no_more_partials_than_it_writes():
    """Width 4, 40,000 tokens x 1,024 channels: beside dx the backward holds 37 strips of partial sums (and 4 MB)."""
    from flame_b200.ops.conv import short_conv
    T, D = 40000, 1024
    x = torch.randn(T, D, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    w = torch.randn(D, 1, 4, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    y, dy = short_conv(x, w, None, _meta([T]), "silu"), torch.randn(T, D, device=DEV, dtype=torch.bfloat16)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    torch.autograd.grad(y, [x, w], dy)
    assert torch.cuda.max_memory_allocated() - before <= 2 * T * D + 37 * D * 5 * 4 + (4 << 20)


@pytest.mark.parametrize("chunk", [64, 128])
@pytest.mark.parametrize("lens", [[1], [16, 64, 3], [65, 128, 1, 1, 2], [127, 63, 192], [200, 15, 17, 49], [4097, 5]])
@pytest.mark.parametrize("main", [False, True])
def test_short_convs_in_chunk_rows(lens, chunk, main):
    """Three convolutions of one launch into the padded rows and back, documents that end before, on and behind the tiles of 16 rows and
    the chunks: bit for bit what one convolution each and a gather give (the same sums in the same order per row), weight gradients
    (fp32 sums over other strips, at most 4,102 rows: n 2^-24 sqrt(n) of the terms' size) to 1e-4.  The padding's incoming gradient is
    not looked at."""
    from flame_b200.ops.chunked import ChunkLayout
    from flame_b200.ops.conv import short_conv, short_convs_in_chunks
    torch.manual_seed(len(lens))
    meta, T = _meta(lens), sum(lens)
    lay, widths = ChunkLayout.of(meta, chunk), (72, 8, 136)
    wide = torch.randn(T, sum(widths) + 8, device=DEV).bfloat16()
    ws = [(torch.randn(n, 1, 4, device=DEV) * 0.4).bfloat16() for n in widths]
    bs = [None, torch.randn(8, device=DEV).bfloat16(), torch.randn(136, device=DEV).bfloat16()]
    dys = [torch.randn(lay.Tp, n, device=DEV).bfloat16() for n in widths]
    results = []
    for together in (True, False):
        x = wide.clone().requires_grad_(True)
        params = [p.clone().requires_grad_(True) for p in ws + [b for b in bs if b is not None]]
        if main:
            for p in params:
                p.main_grad = torch.ones(p.shape, device=DEV)
        w, b = params[:3], [None, *params[3:]]
        xs = torch.split(x[:, :sum(widths)], widths, 1)
        if together:
            ys = short_convs_in_chunks(xs, w, b, meta, "silu", chunk)
        else:
            ys = [lay.pack(short_conv(*a, meta, "silu")).reshape(lay.Tp, -1) for a in zip(xs, w, b)]
        pad = (lay.inv_i32 < 0)[:, None]
        torch.autograd.backward(ys, [dy.masked_fill(pad, 7e3 if together else 0) for dy in dys])
        results.append((list(ys), x.grad, [p.main_grad if main else p.grad for p in params]))
    (y1, x1, p1), (y2, x2, p2) = results
    assert all(torch.equal(a, b) for a, b in zip(y1, y2)) and torch.equal(x1, x2)
    for a, b in zip(p1, p2):
        assert rel_err(a, b) < (1e-4 if main else 5e-3)   # rounded to bf16 once without main_grad


@pytest.mark.parametrize("cols,dtype", [(1, torch.float32), (6, torch.float32), (6, torch.bfloat16), (3, torch.bfloat16), (8, torch.float32)])
def test_row_gather_of_few_scalars(cols, dtype):
    """Rows that are whole 16-byte vectors, whole 4-byte words and neither, also out of a wider matrix: exact."""
    from flame_b200.ops.chunked import ChunkLayout
    lens = [5, 64, 700, 1]
    lay = ChunkLayout.of(_meta(lens), 64)
    for x in (torch.randn(sum(lens), cols, device=DEV).to(dtype), torch.randn(sum(lens), cols + 2, device=DEV).to(dtype)[:, 2:]):
        got = lay.pack(x).reshape(lay.Tp, cols)
        want = torch.zeros(lay.Tp, cols, device=DEV, dtype=dtype).index_copy(0, lay.rows, x)
        assert torch.equal(got, want) and torch.equal(lay.unpack(lay.pack(x)), x)


@pytest.mark.parametrize("lens", [[1], [128], [129, 127, 0, 1], [1] * 1023 + [300, 5], [4096] * 3 + [64] * 1500, [270000, 262016, 130, 262017]])
def test_attention_work_list(lens):
    """Prefix sums of the documents' tiles in their order and by falling length (beyond the last bin's 2,047 tiles in any order), over more
    documents than the block has threads: exact."""
    import numpy as np
    from flame_b200.ops.varlen import VarlenMeta
    n = len(lens)
    meta = VarlenMeta.from_cu_seqlens(torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32), sum(lens), torch.device(DEV))
    offs = meta.tile_offsets
    assert offs.shape == (n + 1,)
    whole = torch.as_strided(offs, (3 * n + 2,), (1,)).tolist()
    tiles = [-(-x // 128) for x in lens]
    docs = whole[2 * n + 2:]
    assert whole[:n + 1] == [0] + list(np.cumsum(tiles))
    assert sorted(docs) == list(range(n)) and whole[n + 1:2 * n + 2] == [0] + list(np.cumsum([tiles[d] for d in docs]))
    clipped = [min(tiles[d], 2047) for d in docs]
    assert clipped == sorted(clipped, reverse=True)


@pytest.mark.parametrize("D", [64, 128, 256, 512])
@pytest.mark.parametrize("gate", [None, "dense", "block"])
def test_norm_out_of_chunk_rows(D, gate):
    """A norm that reads the chunk layout, with its gate a column block of a wider matrix: bit for bit what unpacking and a dense gate
    give, gradients too (zeros in the padding); the weight's gradient sums the same rows over other blocks: 5e-3 after rounding to bf16."""
    from flame_b200.ops.chunked import ChunkLayout
    from flame_b200.ops.norm import rms_norm, rms_norm_chunks, rms_norm_gated
    from flame_b200.ops.slots import reshaped, split_columns
    torch.manual_seed(D)
    lens, H = [1, 63, 65, 300, 64, 7], 3
    T, lay = sum(lens), ChunkLayout.of(_meta(lens), 64)
    o0 = torch.randn(lay.NC, 64, H, D, device=DEV).bfloat16()
    wide0, w0, dy = torch.randn(T, 16 + H * D, device=DEV).bfloat16(), torch.randn(D, device=DEV).bfloat16(), torch.randn(T, H, D, device=DEV).bfloat16()
    out = []
    for new in (True, False):
        o, wide, w = (t.clone().requires_grad_(True) for t in (o0, wide0, w0))
        g = None
        if gate is not None:
            g = reshaped(split_columns(wide, (16, H * D))[1], T, H, D) if gate == "block" and new else wide[:, 16:].reshape(T, H, D).contiguous()
        if new:
            y = rms_norm_chunks(o, lay, w, 1e-5, g)
        else:
            y = rms_norm(lay.unpack(o), w, 1e-5) if g is None else rms_norm_gated(lay.unpack(o), g, w, 1e-5)
        y.backward(dy)
        out.append((y.detach(), o.grad, wide.grad, w.grad))
    for a, b in zip(out[0][:3], out[1][:3]):
        assert (a is None and b is None) or torch.equal(a, b)
    assert rel_err(out[0][3], out[1][3]) < 5e-3


@pytest.mark.parametrize("H,bf16,decay,mul", [(6, True, True, 1.0), (1, False, True, 2.0), (16, True, False, 1.0), (128, True, True, 2.0)])
def test_delta_gates(H, bf16, decay, mul):
    """The delta rule's gates in the chunk layout, from column blocks that start between vectors, against fp64: fp32 results of a few
    operations (1e-5), gradients of bf16 values rounded once (5e-3), of the parameters summed over the rows in fp32 (1e-3)."""
    from flame_b200.ops.chunked import ChunkLayout
    from flame_b200.ops.gates import delta_gates, delta_gates_torch
    from flame_b200.ops.slots import split_columns
    torch.manual_seed(H)
    lens = [1, 63, 65, 2000, 64, 7]
    T, lay = sum(lens), ChunkLayout.of(_meta(lens), 64)
    dt = torch.bfloat16 if bf16 else torch.float32
    x = (torch.randn(T, 3 + 2 * H, device=DEV) * 4).bfloat16().requires_grad_(True)
    A, d = (torch.randn(H, device=DEV).to(dt).requires_grad_(True) for _ in range(2))
    _, a, b = split_columns(x, (3, H, H))
    beta, g = delta_gates(b, a if decay else None, A if decay else None, d if decay else None, mul, lay)
    dbeta, dg = torch.randn_like(beta), torch.randn_like(beta)
    ins = [x, A, d] if decay else [x]
    got = torch.autograd.grad([beta, g] if decay else [beta], ins, [dbeta, dg] if decay else [dbeta])
    xr, Ar, dr = (t.detach().double().requires_grad_(True) for t in (x, A, d))
    sp = torch.nn.functional.softplus(xr[:, 3:3 + H] + dr, threshold=100)
    want_b, want_g = mul * torch.sigmoid(xr[:, 3 + H:]), -Ar.exp() * sp
    flat = lambda t: t.reshape(lay.Tp, H)  # noqa: E731
    assert rel_err(flat(beta)[lay.rows], want_b) < 1e-5 and float(flat(beta)[lay.inv_i32 < 0].abs().sum()) == 0
    want = [(flat(dbeta)[lay.rows].double() * want_b).sum()]
    if decay:
        assert rel_err(flat(g)[lay.rows], want_g) < 1e-5 and float(flat(g)[lay.inv_i32 < 0].abs().sum()) == 0
        want.append((flat(dg)[lay.rows].double() * want_g).sum())
        plain = delta_gates_torch(b.detach(), a.detach(), A.detach(), d.detach(), mul)
        assert rel_err(plain[0], want_b) < 1e-5 and rel_err(plain[1], want_g) < 1e-5
    want = torch.autograd.grad(sum(want), [xr, Ar, dr] if decay else [xr])
    for i, (p, q) in enumerate(zip(got, want)):
        assert rel_err(p, q) < (5e-3 if i == 0 or bf16 else 1e-3)


@pytest.mark.parametrize("rows", [1, 300])
@pytest.mark.parametrize("mains", [False, True])
def test_side_by_side_projections_of_odd_sizes(rows, mains):
    """One product for projections of which some start between vectors (64 + 6 + 6 rows), their gradients written side by side; against
    fp64.  bf16 results of 128-term sums (2^-8), weight gradients in fp32 with main_grad."""
    from flame_b200.ops.linear import linear_fused, side_by_side
    from flame_b200.ops.slots import split_columns
    torch.manual_seed(rows)
    flat, grad = torch.randn(76 * 128, device=DEV).bfloat16() * 0.1, torch.ones(76 * 128, device=DEV)
    ws, at = [], 0
    for n in (64, 6, 6):
        w = torch.nn.Parameter(flat[at:at + n * 128].view(n, 128))
        if mains:
            w.main_grad = grad[at:at + n * 128].view(n, 128)
        ws.append(w)
        at += n * 128
    x = torch.randn(rows, 128, device=DEV).bfloat16().requires_grad_(True)
    assert side_by_side(x, ws)
    parts = split_columns(linear_fused(x, ws), (64, 6, 6))
    dys = [torch.randn_like(p) for p in parts]
    torch.autograd.backward(parts, dys)
    xr, wr, dy = x.detach().double(), flat.view(76, 128).double(), torch.cat(dys, 1).double()
    assert rel_err(torch.cat(parts, 1), xr @ wr.T) < 5e-3 and rel_err(x.grad, dy @ wr) < 5e-3
    got = grad.view(76, 128) - 1 if mains else torch.cat([w.grad for w in ws])
    assert rel_err(got, dy.T @ xr) < (1e-4 if mains else 5e-3)


def test_delta_gates_are_as_exact_as_fp32_allows():
    """Against fp64, at decay rates of 1 to 16 and arguments whose fp32 sum is exact: an exponential and a logarithm of at most one ulp each
    (2^-23), a sum and two products or quotients of half of one: 4 x 2^-23 for the decay, 2 x 2^-23 for beta, relative."""
    from flame_b200.ops.chunked import ChunkLayout
    from flame_b200.ops.gates import delta_gates
    from flame_b200.ops.varlen import VarlenMeta
    torch.manual_seed(0)
    T, H = 4096, 16
    lay = ChunkLayout.of(VarlenMeta.from_cu_seqlens(torch.tensor([0, T], dtype=torch.int32), T, torch.device(DEV)), 64)
    b = (torch.randn(T, H, device=DEV) * 8).bfloat16()
    a = (torch.randn(T, H, device=DEV) * 64).round().clamp(-240, 240).div(16).bfloat16()
    A_log, dt = torch.linspace(0, 2.77, H, device=DEV), torch.randint(-32, 32, (H,), device=DEV) / 16.0
    beta, g = delta_gates(b, a, A_log, dt, 2.0, lay)
    wb = 2 * b.double().sigmoid()
    x = a.double() + dt.double()
    wg = -A_log.double().exp() * (x.clamp_min(0) + torch.log1p((-x.abs()).exp()))
    assert ((beta.view(T, H).double() - wb) / wb).abs().max() <= 2 * 2.0 ** -23
    assert ((g.view(T, H).double() - wg) / wg).abs().max() <= 4 * 2.0 ** -23


@pytest.mark.parametrize("kind", ["softmax", "stickbreaking"])
def test_attention_reads_the_work_list_by_its_own_name(kind, monkeypatch):
    """The kernels' work list is a tensor of its whole length: a copy of it serves as well, and nobody asks for the prefix sums that are
    its head (a copy of those would end where the kernels begin to read).  Same list, so the forward is the same bit for bit."""
    from flame_b200.ops.attention import attention
    from flame_b200.ops.stickbreaking import sb_attention
    from flame_b200.ops.varlen import VarlenMeta
    torch.manual_seed(0)
    lens = [129, 1, 300]
    meta, T = _meta(lens), sum(lens)
    assert meta.tile_list.shape == (3 * len(lens) + 2,) and torch.equal(meta.tile_offsets, meta.tile_list[:len(lens) + 1])
    q, k, v = (torch.randn(T, 2, 64, device=DEV).bfloat16().requires_grad_(True) for _ in range(3))
    call = (lambda m: attention(q, k, v, m)) if kind == "softmax" else (lambda m: sb_attention(q, k, v, m)[0])
    want = call(meta)
    other = _meta(lens)
    other._tile_list = meta.tile_list.clone()
    monkeypatch.setattr(VarlenMeta, "tile_offsets", property(lambda self: pytest.fail("prefix sums asked for")))
    got = call(other)
    got.sum().backward()
    assert torch.equal(got, want) and all(torch.isfinite(t.grad).all() for t in (q, k, v))


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_stickbreaking_value_gradient_does_not_see_what_is_not_finite_elsewhere(bad):
    """A value that is not finite spoils the gradients of queries and keys, but the values' gradient is the weights times dO alone:
    as without it, up to the order in which fp32 partial sums are added, which turns the bf16 rounding (2^-8) of less than one entry in
    ten: 1e-3, in that document and in the others."""
    from flame_b200.ops.stickbreaking import sb_attention
    torch.manual_seed(0)
    lens, H = [300, 70, 129], 2
    meta, T = _meta(lens), sum(lens)
    q, k, v, do = (torch.randn(T, H, 64, device=DEV).bfloat16() for _ in range(4))
    grads = []
    for x in (None, bad):
        args = [t.clone() for t in (q, k, v)]
        if x is not None:
            args[2][150, 0, 3] = x
        args = [t.requires_grad_(True) for t in args]
        grads.append(torch.autograd.grad(sb_attention(*args, meta)[0], args, do))
    assert torch.isfinite(grads[1][2]).all() and rel_err(grads[1][2], grads[0][2]) < 1e-3
    for clean, spoilt in zip(grads[0][:2], grads[1][:2]):
        assert rel_err(spoilt[300:], clean[300:]) < 1e-3 and rel_err(spoilt[:, 1], clean[:, 1]) < 1e-3
        assert torch.isfinite(spoilt[:128, 0]).all() if clean is grads[0][0] else True
        assert not torch.isfinite(spoilt[:300, 0]).all()


def test_short_convs_in_chunk_rows_copy_nothing_for_a_new_batch():
    """The layout's maps are all that the host makes for a new batch: the positions of the padded rows come from those of the packed ones,
    on the device, so with the layout there the convolutions wait for no copy."""
    from flame_b200.ops.chunked import ChunkLayout
    from flame_b200.ops.conv import short_convs_in_chunks
    lens = [65, 1, 200]
    x, w = torch.randn(sum(lens), 64, device=DEV).bfloat16(), torch.randn(64, 1, 4, device=DEV).bfloat16()
    meta = _meta(lens)
    ChunkLayout.of(meta, 64)
    torch.cuda.synchronize()
    torch.cuda.set_sync_debug_mode("error")
    try:
        assert short_convs_in_chunks((x,), (w,), (None,), meta, "silu", 64) is not None
    finally:
        torch.cuda.set_sync_debug_mode("default")


@pytest.mark.parametrize("form", ["block", "broadcast"])
def test_side_by_side_projections_of_odd_sizes_take_any_gradient(form):
    """The gradient of one product for projections of 64 + 6 + 6 rows as a block that starts between vectors of wider rows, and as one row for
    all tokens: the same numbers as dense."""
    from flame_b200.ops.linear import linear_fused, side_by_side
    torch.manual_seed(0)
    flat = torch.randn(76 * 128, device=DEV).bfloat16() * 0.1
    ws = [torch.nn.Parameter(flat[a * 128:b * 128].view(b - a, 128)) for a, b in ((0, 64), (64, 70), (70, 76))]
    x = torch.randn(300, 128, device=DEV).bfloat16().requires_grad_(True)
    assert side_by_side(x, ws)
    dy = torch.randn(300, 88, device=DEV).bfloat16()[:, 3:79] if form == "block" else torch.randn(76, device=DEV).bfloat16().expand(300, 76)
    got, want = (torch.autograd.grad(linear_fused(x, ws), [x, *ws], d) for d in (dy, dy.contiguous()))
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("offset", [1, 4])
@pytest.mark.parametrize("form", ["plain", "residual", "gate"])
def test_norm_operands_start_anywhere(form, offset):
    """Contiguous operands (and the gradients that come back) that start between vectors are moved before a kernel loads them: bit for bit
    the aligned call's results."""
    from flame_b200.ops.norm import rms_norm, rms_norm_gated

    def shifted(t):
        return torch.empty(t.numel() + offset, dtype=t.dtype, device=DEV)[offset:].view(t.shape).copy_(t)
    torch.manual_seed(offset)
    x, other, dy, dr = (torch.randn(37, 3, 128, device=DEV).bfloat16() for _ in range(4))
    w, res = torch.rand(128, device=DEV).bfloat16(), []
    for move in (lambda t: t.clone(), shifted):
        args = [move(t).requires_grad_(True) for t in ((x,) if form == "plain" else (x, other))]
        if form == "gate":
            ys = (rms_norm_gated(args[0], args[1], w),)
        else:
            ys = rms_norm(args[0], w, 1e-6, args[1], True) if form == "residual" else (rms_norm(args[0], w),)
        res.append([*ys, *torch.autograd.grad(ys, args, [move(dy), move(dr)][:len(ys)])])
    assert all(torch.equal(a, b) for a, b in zip(*res))
