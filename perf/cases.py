"""Performance cases: what a user of this framework has it compute in training.

Each case is one forward and backward pass of a layer (or a small whole model) at the widths of ``configs/*.json``, on
packed documents, through the modules a program builds from a configuration.  Parameters lie back to back in one bf16
buffer with an fp32 ``main_grad`` beside each, which is how the training engine lays out a unit, so a pass is what one
micro-batch does to that layer: clear the gradients, run forward, run backward.

``listed()`` are the cases that stand for the families and sizes in use, ``draw()`` gives further ones of the same
ranges, ``exact()`` the same numbers in 64-bit plain torch.
"""
import math
import os
import random

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMALL_MODEL = dict(num_hidden_layers=2, vocab_size=32000, max_position_embeddings=8192)


# ---------------------------------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------------------------------
def _case(name, kind, config, tokens, doc_min, doc_max, doc_seed=0, **more):
    return dict(name=name, kind=kind, config=config, tokens=tokens, doc_min=doc_min, doc_max=doc_max, doc_seed=doc_seed, **more)


def listed():
    return [
        # the smallest thing a user trains: a two-layer Transformer on a short row (smoke runs, debugging, tests)
        _case("small_model", "model", "", 1000, 64, 512, hidden=256),
        # add + norm + SwiGLU MLP of a Transformer-340M block at the flagship batch: 65,536 packed tokens
        _case("mlp_340m", "mlp", "transformer_340M", 65536, 64, 4096),
        # softmax attention of Transformer-340M (head dim 64, rotary) at the flagship batch
        _case("attention_340m", "mixer", "transformer_340M", 65536, 64, 4096),
        # sliding-window attention with head dim 128, an attention layer of Samba-1B; odd row
        _case("attention_window_1b", "mixer_attn", "samba_1B", 8191, 64, 4096),
        # stick-breaking attention on eight dense rows of 4,096, the batch that family is trained with
        _case("stickbreaking_340m", "mixer", "sba_340m", 32768, 4096, 4096),
        # language-model head with the loss: chunked GEMM + cross-entropy over a vocabulary of 32,000; odd row
        _case("head_340m", "head", "transformer_340M", 12289, 64, 4096),
        # linear-attention token mixers, one per chunk algorithm in the configurations, at batches of 16 to 64 thousand tokens
        _case("gla_340m", "mixer", "gla_340M", 65536, 64, 4096),
        _case("gsa_340m", "mixer", "gsa_340M", 32767, 64, 4096),
        _case("delta_net_340m", "mixer", "delta_net_340M", 65536, 64, 4096),
        _case("gated_deltanet_1b", "mixer", "gated_deltanet_1B", 16384, 64, 4096),
        # state-space token mixers
        _case("mamba_340m", "mixer", "mamba_340M", 32768, 64, 4096),
        _case("mamba2_340m", "mixer", "mamba2_340M", 32761, 64, 4096),
    ]


#: (kind, configuration, most tokens) of the drawn cases; a row costs less than the largest listed case
_DRAWN = [
    ("model", "", 4096), ("mlp", "transformer_340M", 65536), ("mlp", "transformer_1B", 16384),
    ("mixer", "transformer_340M", 65536), ("mixer", "transformer_1B", 16384), ("mixer", "transformer_7B", 4096),
    ("mixer_attn", "samba_1B", 16384), ("mixer", "sba_340m", 32768), ("head", "transformer_340M", 16384),
    ("mixer", "gla_340M", 65536), ("mixer", "gsa_340M", 32768), ("mixer", "gsa_1B", 8192),
    ("mixer", "delta_net_340M", 65536), ("mixer", "delta_net_1B", 16384), ("mixer", "gated_deltanet_340M", 16384),
    ("mixer", "gated_deltanet_1B", 16384), ("mixer", "mamba_340M", 32768), ("mixer", "mamba_1B", 16384),
    ("mixer", "samba_1B", 8192), ("mixer", "mamba2_340M", 32768), ("mixer", "mamba2_1B", 16384),
]


def draw(rng):
    kind, config, most = rng.choice(_DRAWN)
    lo = 500
    tokens = int(math.exp(rng.uniform(math.log(lo), math.log(most))))
    if rng.random() < 0.3:
        tokens = max(512, tokens // 64 * 64)
    doc_max = rng.choice([512, 1000, 2048, 4096, 4096])
    doc_min = rng.choice([1, 64, 256])
    if rng.random() < 0.2:
        doc_min = doc_max  # dense rows
    case = dict(kind=kind, config=config, tokens=tokens, doc_min=doc_min, doc_max=doc_max, doc_seed=rng.randrange(1 << 16))
    if kind == "model":
        case["hidden"] = rng.choice([256, 512])
    return case


def _lengths(case):
    rng = random.Random(case["doc_seed"])
    lens, left = [], case["tokens"]
    while left > 0:
        n = min(left, rng.randint(case["doc_min"], case["doc_max"]))
        lens.append(n)
        left -= n
    return lens


def _config(case):
    from flame_b200.models import ModelConfig
    if case["kind"] == "model":
        return ModelConfig("transformer", hidden_size=case["hidden"], num_heads=case["hidden"] // 64, **SMALL_MODEL)
    cfg = ModelConfig.from_pretrained(os.path.join(ROOT, "configs", case["config"] + ".json"))
    return cfg


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def _build(case, cfg, device):
    """The module a program gets from the configuration."""
    from flame_b200.models import build_model
    from flame_b200.models.modeling import Block, SambaBlock, build_mixer
    kind = case["kind"]
    with torch.device(device):
        if kind == "model":
            return build_model(cfg, device="meta", dtype=torch.bfloat16, init=False).to_empty(device=device)
        if kind == "mixer":
            return build_mixer(cfg, 0)
        if kind == "mixer_attn":
            return SambaBlock(cfg, 1).mixer
        if kind == "mlp":
            block = Block(cfg, 0)
            return torch.nn.ModuleDict({"norm": block.mlp_norm, "mlp": block.mlp})
        if kind == "head":
            from flame_b200.models.modules import Linear
            return Linear(cfg.hidden_size, cfg.vocab_size)
    raise ValueError(kind)


@torch.no_grad()
def _fill(module, cfg, gen):
    """Weights as in training: projections normal with the configuration's spread, convolutions and norms away from
    their start values, the decay parameters from the families' own initialisation."""
    from flame_b200.models import layers as L
    for name, p in module.named_parameters():
        def normal(std):
            return torch.randn(p.shape, generator=gen, device=p.device) * std
        if "conv1d.weight" in name:
            p.copy_(normal(0.4))
        elif "norm" in name and p.dim() == 1:
            p.copy_(1 + normal(0.1))
        elif name.endswith("bias") or p.dim() == 1:
            p.copy_(normal(0.1))
        else:
            p.copy_(normal(cfg.initializer_range if "embeddings" not in name else 0.5))
    cpu = torch.Generator().manual_seed(int(torch.randint(1 << 30, (1,), generator=gen, device=gen.device)))
    for m in module.modules():
        if isinstance(m, (L.GatedDeltaNet, L.Mamba2)):
            m.reset_special_parameters(cpu)
        elif isinstance(m, L.Mamba):
            m.reset_special_parameters(cfg, cpu)


def _flatten(module):
    """One bf16 buffer for all parameters and one fp32 buffer for their gradients, ``main_grad`` views attached."""
    params = list(module.named_parameters())
    sizes = [-(-p.numel() // 64) * 64 for _, p in params]
    dev = params[0][1].device
    flat = torch.zeros(sum(sizes), dtype=torch.bfloat16, device=dev)
    grad = torch.zeros(sum(sizes), dtype=torch.float32, device=dev)
    at = 0
    for (name, p), n in zip(params, sizes):
        view = flat[at:at + p.numel()].view(p.shape)
        view.copy_(p.detach())
        new = torch.nn.Parameter(view)
        new.main_grad = grad[at:at + p.numel()].view(p.shape)
        if getattr(p, "_no_weight_decay", False):
            new._no_weight_decay = True
        owner = module
        *path, leaf = name.split(".")
        for part in path:
            owner = getattr(owner, part) if not isinstance(owner, torch.nn.ModuleDict) else owner[part]
        setattr(owner, leaf, new)
        at += n
    return flat, grad


def _inputs(case, seed, device):
    cfg = _config(case)
    gen = torch.Generator(device=device).manual_seed(seed)
    module = _build(case, cfg, device)
    _fill(module, cfg, gen)
    T, D = case["tokens"], cfg.hidden_size

    def activation(scale=1.0):
        return (torch.randn(T, D, generator=gen, device=device) * scale).to(torch.bfloat16)

    s = {"cfg": cfg, "module": module, "kind": case["kind"], "lens": _lengths(case)}
    if case["kind"] == "model":
        s["ids"] = torch.randint(3, cfg.vocab_size, (1, T), generator=gen, device=device)
        return s
    s["x"] = activation()
    if case["kind"] == "mlp":
        s["residual"], s["dres"] = activation(), activation(0.5)
    if case["kind"] == "head":
        lab = torch.randint(0, cfg.vocab_size, (T,), generator=gen, device=device)
        ends = torch.tensor(s["lens"], device=device).cumsum(0) - 1
        lab[ends] = -100  # the last token of a document has no target
        s["labels"] = lab
    else:
        s["dy"] = activation(0.5)
    return s


def prepare(case, seed):
    from flame_b200.ops.varlen import VarlenMeta
    dev = torch.device("cuda")
    s = _inputs(case, seed, dev)
    s["flat"], s["grad"] = _flatten(s["module"])
    s["params"] = dict(s["module"].named_parameters())
    cu = torch.tensor([0] + list(torch.tensor(s["lens"]).cumsum(0)), dtype=torch.int32)
    s["meta"] = VarlenMeta.from_cu_seqlens(cu, case["tokens"], dev)
    for key in ("x", "residual"):
        if key in s:
            s[key].requires_grad_(True)
    return s


def run(s):
    kind, module, meta = s["kind"], s["module"], s["meta"]
    s["grad"].zero_()
    out = {}
    if kind == "model":
        res = module(input_ids=s["ids"], labels=s["ids"], meta=meta)
        res.loss.backward()
        out["loss"] = res.loss.detach()
    else:
        x = s["x"]
        x.grad = None
        if kind == "mlp":
            r = s["residual"]
            r.grad = None
            h, res = module["norm"](x, r, True)
            y = module["mlp"](h)
            torch.autograd.backward([y, res], [s["dy"], s["dres"]])
            out["y"], out["residual"], out["dresidual"] = y.detach(), res.detach(), r.grad
        elif kind == "head":
            from flame_b200.ops.cross_entropy import fused_linear_cross_entropy
            loss = fused_linear_cross_entropy(x, module.weight, s["labels"])
            loss.backward()
            out["loss"] = loss.detach()
        else:
            y = module(x, meta)
            y.backward(s["dy"])
            out["y"] = y.detach()
        out["dx"] = x.grad
    for p in s["params"].values():  # parameters without a fused accumulation, as the engine's hook treats them
        if p.grad is not None:
            p.main_grad.add_(p.grad)
            p.grad = None
    out["dw"] = {n: p.main_grad for n, p in s["params"].items()}
    return out


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def _n_params(case, cfg):
    m = _build(case, cfg, "meta")
    return sum(p.numel() for p in m.parameters()), sum(p.numel() for n, p in m.named_parameters() if p.dim() == 2 and "embeddings" not in n
                                                       and "A_log" not in n)


def work(case):
    cfg = _config(case)
    T, D, lens = case["tokens"], cfg.hidden_size, _lengths(case)
    params, dense = _n_params(case, cfg)
    flops = 6.0 * T * dense
    # x and dy in, y and dx out (bf16); weights in (bf16), their gradients out (fp32)
    nbytes = 4 * T * D * 2 + params * (2 + 4)

    def attention(heads, dim, window=0):
        pairs = 0
        for n in lens:
            w = min(window or n, n)
            pairs += w * (w + 1) // 2 + (n - w) * w
        return 3.5 * 4.0 * pairs * heads * dim  # 2 products forward, 5 backward

    mt = cfg.model_type
    if case["kind"] == "model":
        nbytes = T * 8 + params * (2 + 4)
        flops += cfg.num_hidden_layers * attention(cfg.num_heads, 64)
    elif case["kind"] == "mlp":
        nbytes += 4 * T * D * 2
    elif case["kind"] == "head":
        nbytes = 2 * T * D * 2 + T * 8 + params * (2 + 4)
    elif case["kind"] == "mixer_attn":
        flops += attention(cfg.attn["num_heads"], D // cfg.attn["num_heads"], cfg.attn["window_size"])
    elif mt in ("transformer", "sba"):
        flops += attention(cfg.num_heads, D // cfg.num_heads)
    else:
        # recurrent mixers: per token and head, state update and read forward (2 flops per product), twice that backward
        if mt == "gla":
            state, reads = int(D * cfg.expand_k) * int(D * cfg.expand_v) // cfg.num_heads, 2
        elif mt == "gsa":
            state, reads = 2 * D * cfg.num_slots, 2
        elif mt == "delta_net":
            state, reads = D * D // cfg.num_heads, 3
        elif mt == "gated_deltanet":
            state, reads = cfg.num_heads * cfg.head_dim * int(cfg.head_dim * cfg.expand_v), 3
        elif mt == "mamba2":
            state, reads = int(cfg.expand * D) * cfg.state_size, 2
        else:  # mamba, samba
            inner = cfg.intermediate_size if mt == "samba" else int(cfg.expand * D)
            state, reads = inner * cfg.state_size, 3
        flops += 3 * 2.0 * T * state * reads
    return {"bytes": float(nbytes), "flops": flops}


#: About four times the largest relative error of any output of a case against ``exact``: 0.0047 (MLP), 0.0023 (head),
#: 0.0041 to 0.0052 (attention), 0.007 to 0.02 (the other token mixers, whose gradients pass through chains of bf16
#: operands; a GLA key gradient is the 0.02, cut to 0.03), 0.0065 a layer of the model, which has two.
_REL = {"model": 0.03, "mlp": 0.02, "head": 0.01, "mixer_attn": 0.02, "transformer": 0.02, "sba": 0.02}


def tolerance(case):
    key = case["kind"] if case["kind"] in _REL else _config(case).model_type
    return {"rel": _REL.get(key, 0.03), "max": 0.5}


# ---------------------------------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------------------------------
def _positions(lens, dev):
    return torch.cat([torch.arange(n, device=dev) for n in lens])


def _linear(p, name, x):
    y = x @ p[name + ".weight"].T
    return y + p[name + ".bias"] if name + ".bias" in p else y


def _rms(x, w, eps):
    y = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _conv(p, name, x, lens, act=True):
    """Depthwise causal convolution that never looks past the start of a document."""
    w = p[name + ".weight"][:, 0]
    W = w.shape[1]
    pos = _positions(lens, x.device)
    y = p[name + ".bias"].expand_as(x) if name + ".bias" in p else torch.zeros_like(x)
    for s in range(W):
        xs = F.pad(x, (0, 0, s, 0))[:x.shape[0]]
        y = y + torch.where((pos >= s)[:, None], xs, torch.zeros_like(xs)) * w[:, W - 1 - s]
    return F.silu(y) if act else y


def _rope(x, lens, base):
    T, H, Dh = x.shape
    pos = _positions(lens, x.device).double()
    ang = pos[:, None] * base ** (-torch.arange(0, Dh, 2, device=x.device).double() / Dh)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :Dh // 2], x[..., Dh // 2:]
    return torch.cat([a * c - b * s, a * s + b * c], -1)


def _per_document(fn, tensors, lens):
    out, at = [], 0
    for n in lens:
        out.append(checkpoint(fn, *[t[at:at + n] for t in tensors], use_reentrant=False))
        at += n
    return torch.cat(out)


def _softmax_attention(q, k, v, window):
    L, H, Dh = q.shape
    rep = H // k.shape[1]
    i = torch.arange(L, device=q.device)
    hide = i[None] > i[:, None]
    if window:
        hide = hide | (i[None] <= i[:, None] - window)
    outs = []
    for h in range(H):
        s = (q[:, h] @ k[:, h // rep].T * Dh ** -0.5).masked_fill(hide, float("-inf"))
        outs.append(torch.softmax(s, -1) @ v[:, h // rep])
    return torch.stack(outs, 1)


def _stick_breaking(q, k, v):
    L, H, Dh = q.shape
    i = torch.arange(L, device=q.device)
    hide = i[None] >= i[:, None]
    outs = []
    for h in range(H):
        s = q[:, h] @ k[:, h].T * Dh ** -0.5
        stay = F.logsigmoid(-s).masked_fill(hide, 0.0)
        after = stay.flip(-1).cumsum(-1).flip(-1) - stay
        outs.append((F.logsigmoid(s).masked_fill(hide, float("-inf")) + after).exp() @ v[:, h])
    return torch.stack(outs, 1)


def _attention_layer(p, x, lens, heads, kv_heads, dim, base, window, stick=False, at=""):
    T = x.shape[0]
    q = _linear(p, at + "q_proj", x).view(T, heads, dim)
    k = _linear(p, at + "k_proj", x).view(T, kv_heads, dim)
    v = _linear(p, at + "v_proj", x).view(T, kv_heads, dim)
    if stick:
        o = _per_document(_stick_breaking, (q, k, v), lens)
    else:
        if base is not None:
            q, k = _rope(q, lens, base), _rope(k, lens, base)
        o = _per_document(lambda a, b, c: _softmax_attention(a, b, c, window), (q, k, v), lens)
    return _linear(p, at + "o_proj", o.reshape(T, heads * dim))


def _chunks(step, state, tensors, lens, chunk):
    """All documents side by side, chunk by chunk: ``state, out = step(state, *chunk of every tensor)``."""
    dev, T, n = tensors[0].device, tensors[0].shape[0], len(lens)
    Lp = -(-max(lens) // chunk) * chunk
    idx = torch.full((n, Lp), T, dtype=torch.long, device=dev)
    at = 0
    for d, length in enumerate(lens):
        idx[d, :length] = torch.arange(at, at + length, device=dev)
        at += length
    padded = [torch.cat([t, t.new_zeros(1, *t.shape[1:])])[idx] for t in tensors]
    outs = []
    for c in range(0, Lp, chunk):
        state, o = checkpoint(step, state, *[t[:, c:c + chunk] for t in padded], use_reentrant=False)
        outs.append(o)
    out = torch.cat(outs, 1).flatten(0, 1)
    where = torch.empty(T, dtype=torch.long, device=dev)
    keep = idx.flatten() < T
    where[idx.flatten()[keep]] = keep.nonzero()[:, 0]
    return out[where]


def _gla(q, k, v, g, lens, scale):
    """One decay per key channel; sixteen steps at a time, so that every exponential stays far from the range's ends."""
    def step(S, q, k, v, g):
        b = g.cumsum(1)
        last = b[:, -1:]
        A = torch.einsum("nihd,njhd->nhij", q * b.exp(), k * (-b).exp()).tril()
        o = torch.einsum("nhij,njhv->nihv", A, v) + torch.einsum("nihd,nhdv->nihv", q * b.exp(), S)
        S = S * last[:, 0].exp()[..., None] + torch.einsum("njhd,njhv->nhdv", k * (last - b).exp(), v)
        return S, o * scale
    S = torch.zeros(len(lens), q.shape[1], q.shape[2], v.shape[2], dtype=q.dtype, device=q.device)
    return _chunks(step, S, (q, k, v, g), lens, 16)


def _gla_value_decay(q, k, v, g, lens, scale):
    def step(S, q, k, v, g):
        b = g.cumsum(1)
        last = b[:, -1:]
        A = torch.einsum("nihd,njhd->nhij", q, k).tril()
        o = b.exp() * (torch.einsum("nhij,njhv->nihv", A, v * (-b).exp()) + torch.einsum("nihd,nhdv->nihv", q, S))
        S = S * last[:, 0].exp()[:, :, None] + torch.einsum("njhd,njhv->nhdv", k, v * (last - b).exp())
        return S, o * scale
    S = torch.zeros(len(lens), q.shape[1], q.shape[2], v.shape[2], dtype=q.dtype, device=q.device)
    return _chunks(step, S, (q, k, v, g), lens, 16)


def _delta(q, k, v, beta, g, lens, scale):
    def step(S, q, k, v, beta, g):
        b = g.cumsum(1).transpose(1, 2)                                     # [n, H, C]
        C = b.shape[-1]
        tri = torch.ones(C, C, dtype=torch.bool, device=b.device).tril()
        decay = (b[..., :, None] - b[..., None, :]).masked_fill(~tri, float("-inf")).exp()
        bt = beta.transpose(1, 2)[..., None]
        kk = torch.einsum("nihd,njhd->nhij", k, k) * decay
        rhs = bt * (v.transpose(1, 2) - b.exp()[..., None] * torch.einsum("nihd,nhdv->nhiv", k, S))
        eye = torch.eye(C, dtype=b.dtype, device=b.device)
        u = torch.linalg.solve_triangular(eye + bt * kk.tril(-1), rhs, upper=False, unitriangular=True)
        o = torch.einsum("nhij,nhjv->nihv", torch.einsum("nihd,njhd->nhij", q, k) * decay, u)
        o = o + torch.einsum("nihd,nhi,nhdv->nihv", q, b.exp(), S)
        last = b[..., -1:]
        S = S * last.exp()[..., None] + torch.einsum("njhd,nhj,nhjv->nhdv", k, (last - b).exp(), u)
        return S, o * scale
    S = torch.zeros(len(lens), q.shape[1], q.shape[2], v.shape[2], dtype=q.dtype, device=q.device)
    return _chunks(step, S, (q, k, v, beta, g), lens, 64)


def _selective_scan(u, delta, A, B, C, lens):
    def step(h, u, dl, B, C):
        E = (dl.cumsum(1)[..., None] * A).exp()                             # [n, c, Di, N]
        h = E * (h[:, None] + ((dl * u)[..., None] * B[:, :, None] / E).cumsum(1))
        return h[:, -1], (h * C[:, :, None]).sum(-1)
    h = torch.zeros(len(lens), *A.shape, dtype=u.dtype, device=u.device)
    return _chunks(step, h, (u, delta, B, C), lens, 8)


def _mixer(cfg, p, x, lens):
    T, D, mt = x.shape[0], cfg.hidden_size, cfg.model_type
    if mt in ("transformer", "sba"):
        kv = cfg.num_kv_heads or cfg.num_heads
        return _attention_layer(p, x, lens, cfg.num_heads, kv, D // cfg.num_heads, cfg.rope_theta, 0, mt == "sba")
    if mt == "gla":
        H = cfg.num_heads
        q, k, v = (_linear(p, n, x).view(T, H, -1) for n in ("q_proj", "k_proj", "v_proj"))
        g = F.logsigmoid(_linear(p, "gk_proj.1", _linear(p, "gk_proj.0", x))).view(T, H, -1) / cfg.gate_logit_normalizer
        o = _gla(q, k, v, g, lens, q.shape[-1] ** -0.5)
        o = _rms(o, p["g_norm_swish_gate.weight"], cfg.norm_eps) * F.silu(_linear(p, "g_proj", x)).view_as(o)
        return _linear(p, "o_proj", o.reshape(T, -1))
    if mt == "gsa":
        H = cfg.num_heads
        q, k, v = (F.silu(_linear(p, n, x)).view(T, H, -1) for n in ("q_proj", "k_proj", "v_proj"))
        f = F.logsigmoid(_linear(p, "f_proj", x)).view(T, H, -1) / cfg.gate_logit_normalizer
        s = 1 - f.exp()
        qv = torch.softmax(_gla_value_decay(q, k, s, f, lens, 1.0), -1)
        o = F.silu(_gla(qv, s, v, f, lens, 1.0).reshape(T, -1))
        return _linear(p, "o_proj", _rms(o, p.get("g_norm.weight"), cfg.norm_eps))
    if mt in ("delta_net", "gated_deltanet"):
        H = cfg.num_heads
        q, k, v = (_conv(p, n[0] + "_conv1d", _linear(p, n, x), lens).view(T, H, -1) for n in ("q_proj", "k_proj", "v_proj"))
        q, k = (t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        beta = _linear(p, "b_proj", x).sigmoid()
        if mt == "delta_net":
            g = torch.zeros_like(beta)
        else:
            g = -p["A_log"].exp() * F.softplus(_linear(p, "a_proj", x) + p["dt_bias"])
        o = _delta(q, k, v, beta, g, lens, q.shape[-1] ** -0.5)
        o = _rms(o, p["o_norm.weight"], cfg.norm_eps)
        if cfg.use_gate:
            o = o * F.silu(_linear(p, "g_proj", x)).view_as(o)
        return _linear(p, "o_proj", o.reshape(T, -1))
    if mt in ("mamba", "samba"):
        Di, N = p["A_log"].shape
        xz = _linear(p, "in_proj", x)
        h = _conv(p, "conv1d", xz[:, :Di], lens)
        ssm = _linear(p, "x_proj", h)
        R = ssm.shape[1] - 2 * N
        delta = F.softplus(_linear(p, "dt_proj", ssm[:, :R]))
        y = _selective_scan(h, delta, -p["A_log"].exp(), ssm[:, R:R + N], ssm[:, R + N:], lens) + h * p["D"]
        return _linear(p, "out_proj", y * F.silu(xz[:, Di:]))
    if mt == "mamba2":
        Di, P, G, N = int(cfg.expand * D), cfg.head_dim, cfg.n_groups, cfg.state_size
        H = Di // P
        z, xbc, dt = _linear(p, "in_proj", x).split((Di, Di + 2 * G * N, H), -1)
        xs, B, C = _conv(p, "conv1d", xbc, lens).split((Di, G * N, G * N), -1)
        dt = F.softplus(dt + p["dt_bias"])
        xs = xs.view(T, H, P)
        B, C = (t.view(T, G, N).repeat_interleave(H // G, 1) for t in (B, C))
        g = (-p["A_log"].exp() * dt)[..., None]
        y = _gla(C, B, xs * dt[..., None], g, lens, 1.0) + xs * p["D"][:, None]
        y = y.reshape(T, Di) * F.silu(z)
        return _linear(p, "out_proj", _rms(y, p["norm.weight"], cfg.norm_eps))
    raise ValueError(mt)


def _mlp(p, x, at=""):
    return _linear(p, at + "down_proj", F.silu(_linear(p, at + "gate_proj", x)) * _linear(p, at + "up_proj", x))


def _model_loss(cfg, p, ids, lens):
    ids = ids.reshape(-1)
    x = p["model.embeddings.weight"][ids]
    for i in range(cfg.num_hidden_layers):
        at = f"model.layers.{i}."
        h = _rms(x, p[at + "attn_norm.weight"], cfg.norm_eps)
        x = x + _attention_layer(p, h, lens, cfg.num_heads, cfg.num_heads, cfg.hidden_size // cfg.num_heads, cfg.rope_theta, 0, at=at + "attn.")
        x = x + _mlp(p, _rms(x, p[at + "mlp_norm.weight"], cfg.norm_eps), at + "mlp.")
    logits = _rms(x, p["model.norm.weight"], cfg.norm_eps) @ p["lm_head.weight"].T
    return F.cross_entropy(logits[:-1], ids[1:])


def exact(case, seed):
    dev = torch.device("cuda")
    s = _inputs(case, seed, dev)
    cfg, kind, lens = s["cfg"], s["kind"], s["lens"]
    p = {n: t.detach().to(torch.bfloat16).double().requires_grad_(True) for n, t in s["module"].named_parameters()}
    out = {}
    if kind == "model":
        loss = _model_loss(cfg, p, s["ids"], lens)
        loss.backward()
        out["loss"] = loss.detach()
    else:
        x = s["x"].double().requires_grad_(True)
        if kind == "mlp":
            r = s["residual"].double().requires_grad_(True)
            res = x + r
            y = _mlp(p, _rms(res, p["norm.weight"], cfg.norm_eps), "mlp.")
            torch.autograd.backward([y, res], [s["dy"].double(), s["dres"].double()])
            out["y"], out["residual"], out["dresidual"] = y.detach(), res.detach(), r.grad
        elif kind == "head":
            loss = F.cross_entropy(x @ p["weight"].T, s["labels"], ignore_index=-100)
            loss.backward()
            out["loss"] = loss.detach()
        else:
            if kind == "mixer_attn":
                a = cfg.attn
                y = _attention_layer(p, x, lens, a["num_heads"], a["num_kv_heads"], cfg.hidden_size // a["num_heads"], a["rope_theta"],
                                     a["window_size"])
            else:
                y = _mixer(cfg, p, x, lens)
            y.backward(s["dy"].double())
            out["y"] = y.detach()
        out["dx"] = x.grad
    out["dw"] = {n: t.grad if t.grad is not None else torch.zeros_like(t) for n, t in p.items()}
    return out
