"""Gradients of column blocks written in place (``ops/slots.py``), and layers whose projections run as one GEMM."""
import copy
import threading

import pytest
import torch

from flame_b200.ops import slots
from flame_b200.ops.slots import split_columns


class _Scale(torch.autograd.Function):
    """A consumer that writes its gradient where it belongs."""

    @staticmethod
    def forward(ctx, x, c):
        ctx.c, ctx.slot = c, slots.of(x)
        return x * c

    @staticmethod
    def backward(ctx, dy):
        if ctx.slot is None:
            return dy * ctx.c, None
        return torch.mul(dy, ctx.c, out=ctx.slot.take(*dy.shape, dy.dtype, dy.device)), None


SIZES = (3, 1, 4)


def _views(x):
    return split_columns(x, SIZES), x.split(SIZES, dim=1)


@pytest.mark.parametrize("rows", [1, 5])
def test_same_gradient_as_slices(rows):
    torch.manual_seed(0)
    x = torch.randn(rows, sum(SIZES), dtype=torch.float64, requires_grad=True)
    (a, b, c), (a2, b2, c2) = _views(x)
    y = _Scale.apply(a, 2.0).square().sum() + _Scale.apply(b, 3.0).sum() + _Scale.apply(b, -1.5).square().sum() + (0.5 * c).cos().sum()
    w = (2.0 * a2).square().sum() + (3.0 * b2).sum() + (1.5 * b2).square().sum() + (0.5 * c2).cos().sum()
    want, = torch.autograd.grad(w, x)
    for _ in range(2):  # a second run of the same graph has a buffer of its own
        got, = torch.autograd.grad(y, x, retain_graph=True)
        torch.testing.assert_close(got, want, rtol=1e-12, atol=1e-12)


def test_unused_block_and_partial_runs():
    torch.manual_seed(0)
    x = torch.randn(4, sum(SIZES), dtype=torch.float64, requires_grad=True)
    a, b, c = split_columns(x, SIZES)
    y = _Scale.apply(a, 2.0).square().sum() + _Scale.apply(c, 3.0).square().sum()
    ga, = torch.autograd.grad(y, a, retain_graph=True)       # stops at the view: keeps its buffer
    kept = ga.clone()
    gx, = torch.autograd.grad(2.0 * y, x, retain_graph=True)  # another run: must not write into the first one's
    torch.testing.assert_close(ga, kept)
    want = torch.cat([8 * x[:, :3], 0 * x[:, 3:4], 18 * x[:, 4:]], 1).detach()
    torch.testing.assert_close(gx, 2 * want, rtol=1e-12, atol=1e-12)


class _ScaleHeads(torch.autograd.Function):
    """A consumer of ``[T, H, d]`` rows (``slots.reshaped``) that writes its gradient where it belongs."""

    @staticmethod
    def forward(ctx, x):
        ctx.slot = slots.of(x)
        return 2.0 * x

    @staticmethod
    def backward(ctx, dy):
        T, H, d = dy.shape
        return ctx.slot.take(T, H * d, dy.dtype, dy.device).view(T, H, d).copy_(2.0 * dy)


@pytest.mark.parametrize("rows", [1, 2])
def test_rows_of_heads(rows):
    """A gradient that comes back through a reshape is still the block of the buffer it was written to; of one row, the reshape
    hands back another stride."""
    x = torch.randn(rows, 12, dtype=torch.float64, requires_grad=True)
    a, b = split_columns(x, (8, 4))
    y = _ScaleHeads.apply(slots.reshaped(a, rows, 2, 4)).square().sum() + _ScaleHeads.apply(slots.reshaped(b, rows, 4, 1)).sum()
    got, = torch.autograd.grad(y, x)
    torch.testing.assert_close(got, torch.cat([8 * x[:, :8], 0 * x[:, 8:] + 2], 1).detach(), rtol=1e-12, atol=1e-12)


def test_another_stream_gets_its_own_matrix(monkeypatch):
    """The shared buffer is written on the stream that allocated it only; the other block's gradient is copied in."""
    holder = slots._Holder(5)
    first, second = slots.Slot(holder, 0, 2), slots.Slot(holder, 2, 3)
    monkeypatch.setattr(torch._C, "_current_graph_task_id", lambda: 7)
    a = first.take(4, 2, torch.float32, torch.device("cpu"))
    holder.stream = 1
    b = second.take(4, 3, torch.float32, torch.device("cpu"))
    assert a.untyped_storage().data_ptr() == holder.buffer.untyped_storage().data_ptr()
    assert b.untyped_storage().data_ptr() != holder.buffer.untyped_storage().data_ptr()


def test_runs_in_two_threads_never_share_a_buffer(monkeypatch):
    """Two backward runs of one graph: the second asks for its columns just when the first has allocated the buffer."""
    run, between, done = threading.local(), threading.Event(), threading.Event()

    class Holder(slots._Holder):
        def __setattr__(self, name, value):
            super().__setattr__(name, value)
            if name == "stream" and getattr(run, "id", 0) == 1 and not between.is_set():
                between.set()
                done.wait(0.5)   # a holder that makes runs take turns lets this time run out

    monkeypatch.setattr(torch._C, "_current_graph_task_id", lambda: run.id)
    holder, got = Holder(5), {}
    one, two = slots.Slot(holder, 0, 2), slots.Slot(holder, 2, 3)

    def first():
        run.id = 1
        got[1] = one.take(4, 2, torch.float32, torch.device("cpu"))

    def second():
        run.id = 2
        between.wait(5)
        got[2] = two.take(4, 3, torch.float32, torch.device("cpu"))
        done.set()
    threads = [threading.Thread(target=f) for f in (first, second)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got[1].untyped_storage().data_ptr() != got[2].untyped_storage().data_ptr()


def test_backward_of_one_graph_in_several_threads():
    torch.manual_seed(0)
    x = torch.randn(64, sum(SIZES), dtype=torch.float64, requires_grad=True)
    a, b, c = split_columns(x, SIZES)
    y = _Scale.apply(a, 2.0).square().sum() + _Scale.apply(b, 3.0).square().sum() + _Scale.apply(c, -1.0).square().sum()
    want, = torch.autograd.grad(y, x, retain_graph=True)
    wrong = []

    def work(i):
        for _ in range(50):
            g, = torch.autograd.grad(i * y, x, retain_graph=True)
            if not torch.equal(g, i * want):
                wrong.append(i)
    threads = [threading.Thread(target=work, args=(2.0 ** i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def _adjacent(layers):
    """The layers' weights as row blocks of one matrix, their gradients too."""
    ws = [l.weight for l in layers]
    n, d = sum(w.shape[0] for w in ws), ws[0].shape[1]
    flat, grad = torch.empty(n, d, dtype=ws[0].dtype, device=ws[0].device), torch.zeros(n, d, device=ws[0].device)
    c = 0
    for w in ws:
        flat[c:c + w.shape[0]].copy_(w.detach())
        w.data, w.main_grad = flat[c:c + w.shape[0]], grad[c:c + w.shape[0]]
        c += w.shape[0]


def test_layers_that_somebody_listens_to_run_by_themselves(monkeypatch):
    """One product stands for three projections only while nobody could tell: hooks on one of them or on all modules, and a
    forward put on an instance, are honoured."""
    from torch.nn.modules import module as nn_module
    from flame_b200.models import modules
    monkeypatch.setattr(modules.linear_ops, "side_by_side", lambda x, ws: True)   # (as the engine lays them out on a GPU)
    x = torch.randn(3, 8)
    layers = [modules.Linear(8, n) for n in SIZES]
    seen = []
    note = lambda m, *a: seen.append(m)  # noqa: E731
    assert modules.side_by_side(layers, x)
    for register in (layers[1].register_forward_hook, layers[1].register_forward_pre_hook, layers[1].register_full_backward_hook,
                     nn_module.register_module_forward_hook, nn_module.register_module_forward_pre_hook,
                     nn_module.register_module_full_backward_hook, nn_module.register_module_full_backward_pre_hook):
        handle = register(note)
        try:
            assert not modules.side_by_side(layers, x), register
        finally:
            handle.remove()
    assert modules.side_by_side(layers, x)
    handle = nn_module.register_module_forward_hook(note)
    try:
        modules.split_projections(x, layers)
    finally:
        handle.remove()
    assert seen == layers
    plain = layers[2].forward
    layers[2].forward = lambda t: 2 * plain(t)
    assert not modules.side_by_side(layers, x)
    torch.testing.assert_close(modules.split_projections(x, layers)[2], 2 * plain(x))


def test_one_view_of_tensors_that_are_not_adjacent_is_refused():
    from flame_b200.ops.linear import _cat_view
    flat = torch.arange(24.0).view(6, 4)
    assert torch.equal(_cat_view([flat[:2], flat[2:5]]), flat[:5])
    with pytest.raises(ValueError):
        _cat_view([flat[:2].clone(), flat[2:5].clone()])


@pytest.mark.gpu
@pytest.mark.parametrize("name,kw", [
    ("Attention", dict(num_heads=4)), ("Attention", dict(num_heads=2, num_kv_heads=1)), ("StickBreakingAttention", dict(num_heads=4)),
    ("GatedLinearAttention", dict(num_heads=2)), ("DeltaNet", dict(num_heads=2)), ("GatedDeltaNet", dict(num_heads=2, head_dim=64)),
    ("GatedSlotAttention", dict(num_heads=2)), ("Mamba", dict(intermediate_size=512, time_step_rank=16)), ("Mamba2", dict(num_heads=8)),
])
def test_layers_under_saved_tensor_hooks(name, kw):
    """What is saved for the backward goes to the host and comes back as copies (the projections' weights too, which then lie
    apart): the same numbers go through the same kernels, so the input's gradient is the same (fp32 sums of attention's dq by
    atomics: 2^-8 of the largest entry)."""
    from flame_b200.models import layers as layers_mod
    from flame_b200.ops.varlen import VarlenMeta
    torch.manual_seed(0)
    dev = torch.device("cuda", 0)
    D, cu = 256, (0, 1, 66, 131)
    m = getattr(layers_mod, name)(D, **kw)
    for p in m.parameters():
        torch.nn.init.normal_(p, std=0.05) if p.dim() > 1 else torch.nn.init.uniform_(p, 0.5, 1.0)
    m = m.to(dev)
    for n, p in m.named_parameters():
        if n not in ("A_log", "dt_bias", "D"):
            p.data = p.data.bfloat16()
    if hasattr(m, "q_proj"):
        _adjacent([m.q_proj, m.k_proj, m.v_proj])
        for layer in (m.q_proj, m.k_proj, m.v_proj):
            del layer.weight.main_grad
    meta = VarlenMeta.from_cu_seqlens(torch.tensor(cu, dtype=torch.int32, device=dev))
    x, dy = torch.randn(cu[-1], D, device=dev).bfloat16().requires_grad_(True), torch.randn(cu[-1], D, device=dev).bfloat16()
    want = torch.autograd.grad(m(x, meta), [x, *m.parameters()], dy)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.to(dev)):
        y = m(x, meta)
    for a, b in zip(torch.autograd.grad(y, [x, *m.parameters()], dy), want):
        assert (a.double() - b.double()).abs().max() <= 2.0 ** -8 * b.double().abs().max()


@pytest.mark.gpu
@pytest.mark.parametrize("name,kw", [
    ("GatedLinearAttention", dict(num_heads=2)),
    ("GatedLinearAttention", dict(num_heads=2, use_short_conv=True)),
    ("DeltaNet", dict(num_heads=2)),
    ("DeltaNet", dict(num_heads=2, use_short_conv=False)),
    ("GatedDeltaNet", dict(num_heads=2, head_dim=64)),
    ("GatedSlotAttention", dict(num_heads=2)),
    ("GatedSlotAttention", dict(num_heads=2, use_short_conv=True)),
    ("GatedSlotAttention", dict(num_heads=2, feature_map="relu")),
])
@pytest.mark.parametrize("cu", [(0, 1), (0, 128), (0, 1, 66, 131)])
def test_layer_with_adjacent_projections(name, kw, cu):
    """One GEMM for adjacent projections or one each: bf16 rounding of the same sums (the input's gradient is rounded once
    instead of three times), so both lie within a few bf16 steps (2^-8 of the largest entry) of one another."""
    from flame_b200.models import layers as layers_mod
    from flame_b200.ops.varlen import VarlenMeta
    torch.manual_seed(0)
    dev = torch.device("cuda", 0)
    D, T = 256, cu[-1]
    one = getattr(layers_mod, name)(D, **kw)
    for p in one.parameters():
        torch.nn.init.normal_(p, std=0.05) if p.dim() > 1 else torch.nn.init.uniform_(p, 0.5, 1.0)
    one = one.to(dev)
    for n, p in one.named_parameters():
        if n not in ("A_log", "dt_bias", "D"):
            p.data = p.data.bfloat16()
    two = copy.deepcopy(one)
    trio = lambda m: [m.q_proj, m.k_proj, m.v_proj]  # noqa: E731
    _adjacent(trio(two))
    for m in trio(one):
        m.weight.main_grad = torch.zeros_like(m.weight, dtype=torch.float32)
    meta = VarlenMeta.from_cu_seqlens(torch.tensor(cu, dtype=torch.int32, device=dev))
    x = torch.randn(T, D, device=dev).bfloat16()
    dy = torch.randn(T, D, device=dev).bfloat16()
    res = []
    for m in (one, two):
        xi = x.clone().requires_grad_(True)
        y = m(xi, meta)
        y.backward(dy)
        res.append([y.detach(), xi.grad] + [p.weight.main_grad for p in trio(m)] +
                   [p.grad for n, p in m.named_parameters() if p.grad is not None])
    assert len(res[0]) == len(res[1])
    for a, b in zip(*res):
        a, b = a.double(), b.double()
        assert (a - b).abs().max() <= 4 * 2.0 ** -8 * a.abs().max().clamp_min(1e-6), name


@pytest.mark.gpu
@pytest.mark.parametrize("cols", [(8, 0, 8), (136, 8, 64), (72, 4, 8), (64, 0, 64), (20, 8, 8)])
@pytest.mark.parametrize("cu", [(0, 3, 70, 199), (0, 1)])
def test_pack_of_column_blocks(cols, cu):
    """Rows gathered out of a wider matrix (and gradients into one): copies, so equal bit for bit, also where the block
    does not start on 16 bytes, where the matrix' rows are not whole vectors apart, and of one row."""
    from flame_b200.ops.chunked import ChunkLayout
    from flame_b200.ops.varlen import VarlenMeta
    width, c0, n = cols
    dev = torch.device("cuda", 0)
    meta = VarlenMeta.from_cu_seqlens(torch.tensor(cu, dtype=torch.int32, device=dev))
    lay = ChunkLayout(meta)
    torch.manual_seed(0)
    base = torch.randn(cu[-1], width, device=dev).bfloat16()
    sizes = [s for s in (c0, n, width - c0 - n) if s]
    k = 1 if c0 else 0
    got = []
    for split in (lambda t: split_columns(t, sizes), lambda t: [p.contiguous() for p in t.split(sizes, 1)]):
        x = base.clone().requires_grad_(True)
        parts = split(x)
        y = lay.pack(slots.reshaped(parts[k], cu[-1], 1, n))
        w = torch.arange(y.numel(), device=dev).reshape(y.shape).remainder(7).to(y.dtype)
        (y * w).sum().backward()
        got += [(y.detach(), x.grad)]
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.gpu
@pytest.mark.parametrize("name,kw", [("DeltaNet", dict(num_heads=2)), ("GatedDeltaNet", dict(num_heads=2, head_dim=64))])
@pytest.mark.parametrize("which", ["q_conv1d", "v_conv1d"])
def test_a_convolution_without_activation_stays_without(name, kw, which):
    """Convolutions and delta rule run in one go only as SiLU convolutions.  The other side's convolutions are called as modules (a hook that
    does nothing): the same operations on packed rows, bf16 results up to a few roundings (2^-8 of the largest entry)."""
    from flame_b200.models import layers as layers_mod
    from flame_b200.ops.varlen import VarlenMeta
    torch.manual_seed(0)
    dev, D = torch.device("cuda", 0), 256
    m = getattr(layers_mod, name)(D, **kw)
    for p in m.parameters():
        torch.nn.init.normal_(p, std=0.3) if p.dim() > 1 else torch.nn.init.uniform_(p, 0.5, 1.0)
    m = m.to(dev).bfloat16()
    meta = VarlenMeta.from_cu_seqlens(torch.tensor((0, 1, 66, 131), dtype=torch.int32, device=dev))
    x, out = torch.randn(131, D, device=dev).bfloat16(), []
    getattr(m, which).activation = None
    with torch.no_grad():
        out.append(m(x, meta).double())
        handle = m.k_conv1d.register_forward_hook(lambda *a: None)
        out.append(m(x, meta).double())
        handle.remove()
        getattr(m, which).activation = "silu"
        with_silu = m(x, meta).double()
    scale = out[1].abs().max()
    assert (out[0] - out[1]).abs().max() <= 4 * 2.0 ** -8 * scale < (with_silu - out[1]).abs().max()


def test_a_longer_low_rank_gate_runs_whole():
    """GLA takes its low-rank gate projection apart only when it is the two layers that it makes itself: one with a third entry, or with one
    alone, gives what the same modules give as a module of another kind."""
    from flame_b200.models.layers import GatedLinearAttention
    from flame_b200.models.modules import Linear
    from flame_b200.ops.varlen import VarlenMeta
    torch.manual_seed(0)
    m = GatedLinearAttention(32, num_heads=2)
    for extra in (lambda s: torch.nn.Sequential(*s, torch.nn.Tanh()), lambda s: torch.nn.Sequential(Linear(32, 16))):
        m.gk_proj = extra(m.gk_proj)
        for p in m.parameters():
            torch.nn.init.normal_(p, std=0.5)

        class Whole(torch.nn.Module):
            def __init__(self, seq):
                super().__init__()
                self.seq = seq

            def forward(self, x):
                return self.seq(x)

        x, meta = torch.randn(7, 32), VarlenMeta.dense(1, 7, torch.device("cpu"))
        got = m(x, meta)
        m.gk_proj = Whole(m.gk_proj)
        torch.testing.assert_close(got, m(x, meta))
        m.gk_proj = m.gk_proj.seq


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(num_kv_heads=2), dict(num_slots=520)])
def test_gsa_activations_see_whole_rows(kw, monkeypatch):
    """Where the chunk kernels do not take GSA's projections (fewer key heads, more than 512 slots), torch's activation runs over a matrix of
    its own, not over column blocks beside the slots' gates, on which it is several times slower."""
    from flame_b200.models import layers as layers_mod
    from flame_b200.ops.varlen import VarlenMeta
    torch.manual_seed(0)
    dev = torch.device("cuda", 0)
    m = layers_mod.GatedSlotAttention(256, num_heads=4, **kw).to(dev).bfloat16()
    for p in m.parameters():
        torch.nn.init.normal_(p, std=0.05)
    _adjacent([m.q_proj, m.k_proj, m.v_proj, m.f_proj])
    seen, silu = [], torch.nn.functional.silu
    monkeypatch.setattr(torch.nn.functional, "silu", lambda t, *a: (seen.append(t.is_contiguous()), silu(t, *a))[1])
    x = torch.randn(131, 256, device=dev).bfloat16()
    m(x, VarlenMeta.from_cu_seqlens(torch.tensor((0, 1, 66, 131), dtype=torch.int32, device=dev)))
    assert seen and all(seen)


@pytest.mark.gpu
def test_gla_output_gate_is_whole_where_torch_activates_it(monkeypatch):
    """Without the fused norm, torch's activation runs over the output gate: over a matrix of its own, not a column block."""
    from flame_b200.models import layers as layers_mod
    from flame_b200.ops.varlen import VarlenMeta
    torch.manual_seed(0)
    dev = torch.device("cuda", 0)
    m = layers_mod.GatedLinearAttention(256, num_heads=2, fuse_norm=False).to(dev).bfloat16()
    for p in m.parameters():
        torch.nn.init.normal_(p, std=0.05)
    _adjacent([m.q_proj, m.k_proj, m.v_proj, m.g_proj, m.gk_proj[0]])
    seen, silu = [], torch.nn.functional.silu
    monkeypatch.setattr(torch.nn.functional, "silu", lambda t, *a: (seen.append(t.is_contiguous()), silu(t, *a))[1])
    x = torch.randn(131, 256, device=dev).bfloat16()
    m(x, VarlenMeta.from_cu_seqlens(torch.tensor((0, 1, 66, 131), dtype=torch.int32, device=dev)))
    assert seen and all(seen)


@pytest.mark.gpu
@pytest.mark.parametrize("frozen", [("A_log",), ("dt_bias",), ("A_log", "dt_bias"), ("q_proj", "k_proj", "v_proj", "a_proj", "b_proj")])
def test_frozen_parameters_of_the_delta_rule_gates_collect_nothing(frozen):
    """What is frozen keeps its gradient buffer as it is, although the kernels write the others' in place; those get what they get otherwise."""
    from flame_b200.models import layers as layers_mod
    from flame_b200.ops.varlen import VarlenMeta
    torch.manual_seed(0)
    dev, D, T = torch.device("cuda", 0), 256, 131
    m = layers_mod.GatedDeltaNet(D, num_heads=2, head_dim=64).to(dev)
    for n, p in m.named_parameters():
        torch.nn.init.normal_(p, std=0.05) if p.dim() > 1 else torch.nn.init.uniform_(p, 0.5, 1.0)
        if n not in ("A_log", "dt_bias"):
            p.data = p.data.bfloat16()
    _adjacent([m.q_proj, m.k_proj, m.v_proj, m.a_proj, m.b_proj])
    for p in m.parameters():
        p.main_grad = getattr(p, "main_grad", torch.zeros(p.shape, device=dev))
    meta = VarlenMeta.from_cu_seqlens(torch.tensor((0, 1, 66, 131), dtype=torch.int32, device=dev))
    x, dy = torch.randn(T, D, device=dev).bfloat16(), torch.randn(T, D, device=dev).bfloat16()
    res = []
    for freeze in (False, True):
        for n, p in m.named_parameters():
            p.main_grad.fill_(1.0)
            p.grad = None
            p.requires_grad_(not (freeze and n.split(".")[0] in frozen))
        m(x.clone().requires_grad_(True), meta).backward(dy)
        res.append({n: p.main_grad.clone() if p.grad is None else p.main_grad + p.grad for n, p in m.named_parameters()})
    for n, p in m.named_parameters():
        if p.requires_grad:
            assert (res[0][n] - res[1][n]).abs().max() <= 1e-5 * res[0][n].abs().max(), n
        else:
            assert (res[1][n] == 1).all() and p.grad is None, n


@pytest.mark.gpu
@pytest.mark.parametrize("name,kw,every,where", [
    ("GatedLinearAttention", dict(num_heads=2), ("q_proj", "k_proj", "v_proj", "g_proj", "gk_proj.0"), "chunked.gla_raw_gate"),
    ("GatedLinearAttention", dict(num_heads=3, use_output_gate=False), ("q_proj", "k_proj", "v_proj", "gk_proj.0"), "chunked.gla_raw_gate"),
    ("GatedSlotAttention", dict(num_heads=3, num_slots=40), ("q_proj", "k_proj", "v_proj", "f_proj"), "chunked.gsa_in_chunks"),
    ("DeltaNet", dict(num_heads=3), ("q_proj", "k_proj", "v_proj", "b_proj"), "delta_rule.conv_gated_delta_rule"),
    ("DeltaNet", dict(num_heads=3, use_gate=True, allow_neg_eigval=True), ("q_proj", "k_proj", "v_proj", "b_proj"), "delta_rule.conv_gated_delta_rule"),
    ("GatedDeltaNet", dict(num_heads=3, head_dim=64), ("q_proj", "k_proj", "v_proj", "a_proj", "b_proj"), "delta_rule.conv_gated_delta_rule"),
    ("Mamba2", dict(num_heads=8, n_groups=2), ("in_proj",), "conv.short_convs_in_chunks"),
])
@pytest.mark.parametrize("cu", [(0, 128), (0, 1, 66, 131), (0, 200, 263, 264, 300)])
def test_layer_forms_that_training_takes(name, kw, every, where, cu, monkeypatch):
    """One product for ALL projections of a layer, its gradients in one buffer, and the convolutions, gates and norms in the chunk layout, as
    the engine's flat parameters make a layer run, against each projection and convolution by itself on packed rows (weights apart, a hook
    that does nothing on the convolutions and norms): bf16 roundings of the same sums, a few steps (2^-8) of the largest entry.  And once
    more with everything saved for the backward going to the host and back: the same kernels on the same numbers (2^-8)."""
    import importlib
    from flame_b200.models import layers as layers_mod, modules
    from flame_b200.ops.varlen import VarlenMeta
    torch.manual_seed(0)
    dev, D, T = torch.device("cuda", 0), 256 if name == "Mamba2" else 384, cu[-1]
    one = getattr(layers_mod, name)(D, **kw)
    for p in one.parameters():
        torch.nn.init.normal_(p, std=0.05) if p.dim() > 1 else torch.nn.init.uniform_(p, 0.5, 1.0)
    one = one.to(dev)
    for n, p in one.named_parameters():
        if n not in ("A_log", "dt_bias", "D"):
            p.data = p.data.bfloat16()
    two = copy.deepcopy(one)
    for n, sub in one.named_modules():
        if isinstance(sub, (modules.ShortConvolution, modules.RMSNorm, modules.RMSNormGated)):
            sub.register_forward_hook(lambda *a: None)
    for m, apart in ((one, True), (two, False)):
        projections = [m.get_submodule(n) for n in every]
        _adjacent(projections)
        x = torch.randn(T, D, device=dev).bfloat16()
        if apart:  # (the same values, each at a place of its own)
            for l in projections:
                l.weight.data, l.weight.main_grad = l.weight.data.clone(), l.weight.main_grad.clone()
        assert modules.side_by_side(projections, x) == (not apart or len(every) == 1)
        for p in m.parameters():
            if not hasattr(p, "main_grad"):
                p.main_grad = torch.zeros(p.shape, device=dev)
    meta = VarlenMeta.from_cu_seqlens(torch.tensor(cu, dtype=torch.int32, device=dev))
    dy = torch.randn(T, D, device=dev).bfloat16()
    module, function = where.split(".")
    module = importlib.import_module("flame_b200.ops." + module)
    took, real = [], getattr(module, function)
    monkeypatch.setattr(module, function, lambda *a, **k: (took.append(real(*a, **k)), took[-1])[1])

    def run(m, save=None):
        for p in m.parameters():
            p.main_grad.zero_()
            p.grad = None
        xi = x.clone().requires_grad_(True)
        if save is None:
            y = m(xi, meta)
        else:
            with torch.autograd.graph.saved_tensors_hooks(*save):
                y = m(xi, meta)
        y.backward(dy)
        return [y.detach(), xi.grad] + [p.main_grad.clone() if p.grad is None else p.main_grad + p.grad for p in m.parameters()]

    want = run(one)
    fused = name.startswith("Gated") and "Delta" not in name  # (GLA and GSA have no convolution to listen to: both sides may take the form)
    assert fused or not any(t is not None for t in took)
    took.clear()
    got = run(two)
    assert took and took[0] is not None
    hooked = run(two, (lambda t: t.cpu(), lambda t: t.to(dev)))
    names = ["y", "dx"] + [n for n, _ in two.named_parameters()]
    for n, a, b, c in zip(names, got, want, hooked):
        a, b, c = a.double(), b.double(), c.double()
        assert (a - b).abs().max() <= 4 * 2.0 ** -8 * b.abs().max().clamp_min(1e-6), n
        assert (a - c).abs().max() <= 2.0 ** -8 * a.abs().max().clamp_min(1e-6), n
