"""The work this framework's speed is measured on: steps of the serving engine, driven through its public entry points
(``LmEngine.open_sequence`` / ``feed`` / ``close_sequence``) the way a server or an evaluation program drives it.

Models are the repository's own presets, cut to a few layers of their repeating pattern so that a state fits the card
several times over; widths, heads, experts and vocabulary are those of the whole model. A case is

  model    preset and number of layers, with the form of its weights (``MODELS``)
  mode     "decode": one generated token for each of ``seqs`` sequences that hold ``tokens`` tokens on average (the captured
           step the engine replays); "prompt": ``seqs`` new prompts of ``tokens`` tokens on average, read from the start
  ragged   lengths spread from about half to one and a half times the mean, else all the same

Weights are random with unit-gain projections and a damped return to the residual, as trained models have it (``DAMP``), and
query norms that make the attention concentrate on few keys. Quantised weights hold values that their format represents
exactly, so the 64-bit results need no copy of the encoders.
"""
from __future__ import annotations

import math
import zlib

import torch
import torch.nn.functional as F

from legion_b200.config import PRESETS
from legion_b200.engine.lm import EngineConfig, LmEngine
from legion_b200.loaders.tokenizer import ByteTokenizer
from legion_b200.models.decoder import Decoder
from legion_b200.models.weights import is_fp32_weight, weight_shapes

CHUNK = 8192            # prompt tokens of one step
CTX = 8192              # the server's default context size; longer cases get as much as they need

#: name -> preset, layers, form of the weights, most tokens that sequences of one decode case may hold together
MODELS = {
    "hybrid": ("qwen35-80b-a3b", 8, "nvfp4", 131072),   # 6 Gated DeltaNet + 2 gated attention layers, 512 NVFP4 experts
    "moe": ("qwen3-30b-a3b", 4, "bf16", 131072),        # attention and 128 bf16 experts
    "dense": ("dense-27b", 4, "bf16", 49152),           # attention and a wide feed-forward part
    "dense-fp8": ("dense-27b", 4, "fp8", 49152),        # the same with block-scaled e4m3 projections
    "latent": ("mla-7b", 6, "bf16", 65536),             # latent attention
}


def listed():
    def case(name, model, mode, seqs, tokens, ragged=False):
        return dict(name=name, model=model, mode=mode, seqs=seqs, tokens=tokens, ragged=ragged)
    return [
        # one person chats with the flagship: every token waits for one chain of small launches
        case("chat-1", "hybrid", "decode", 1, 1000),
        # a small team on it, and a busy server with chats of all ages
        case("chat-16", "hybrid", "decode", 16, 1024),
        case("chat-64", "hybrid", "decode", 64, 1500, True),
        # a short question arrives: time to first token
        case("turn-217", "hybrid", "prompt", 1, 217),
        # a whole report or source tree is read before the first answer
        case("document-32k", "hybrid", "prompt", 1, 32768),
        # assistants with long histories on a bf16 mixture of experts
        case("history-8k", "moe", "decode", 16, 8192),
        # a batch of questions of mixed lengths admitted in one step
        case("batch-9", "moe", "prompt", 9, 611, True),
        # a dense model: users in the middle of their chats, and one long prompt
        case("dense-21", "dense", "decode", 21, 2048, True),
        case("dense-8k", "dense", "prompt", 1, 8192),
        # the same model from an FP8 checkpoint, few users
        case("fp8-7", "dense-fp8", "decode", 7, 3001, True),
        # latent attention: users with middling histories, and a prompt that no tile divides
        case("latent-16", "latent", "decode", 16, 4096),
        case("latent-6k", "latent", "prompt", 1, 6001),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    model = rng.choice(["hybrid", "hybrid", "hybrid", "moe", "moe", "dense", "dense-fp8", "latent", "latent"])
    if rng.random() < 0.5:
        seqs = _log(rng, 1, 64)
        tokens = _log(rng, 64, min(8192, MODELS[model][3] // (2 * seqs)))
        return dict(model=model, mode="decode", seqs=seqs, tokens=tokens, ragged=rng.random() < 0.7)
    if rng.random() < 0.5:
        return dict(model=model, mode="prompt", seqs=1, tokens=_log(rng, 33, 24576 if model == "hybrid" else 12288), ragged=False)
    seqs = _log(rng, 2, 12)
    return dict(model=model, mode="prompt", seqs=seqs, tokens=_log(rng, 24, 5400 // seqs), ragged=True)


def _lengths(case):
    n, mean = case["seqs"], case["tokens"]
    if not case["ragged"]:
        return [mean] * n
    golden = (math.sqrt(5.0) - 1) / 2          # evenly spread, in no order
    return [max(1, int(mean * (0.5 + (i + 1) * golden % 1.0))) for i in range(n)]


def _config(case):
    preset, layers, form, _ = MODELS[case["model"]]
    cfg = PRESETS[preset]()
    cfg.n_layer, cfg.layer_kinds = layers, cfg.layer_kinds[:layers]
    return cfg, form


# ---------------------------------------------------------------------------------------------------------- inputs
def _gen(name, seed):
    return torch.Generator(device="cuda").manual_seed((zlib.crc32(name.encode()) << 20) + seed % (1 << 20))


#: gain of the projections back to the residual: 4-bit activations put an error of a tenth on an expert's result, and models
#: that are served that way bear it because a sublayer moves the residual by little
DAMP = {"bf16": 0.5, "fp8": 0.5, "nvfp4": 0.125}
RETURNS = ("attn.o", "gdn.out", "mla.o", "mlp.down", "moe.down", "moe.sh_down")
EXPERTS = ("moe.gate_up", "moe.down", "moe.sh_gate_up", "moe.sh_down")
FP8 = Decoder.FP8_LEAVES


def _nvfp4_values(t, std):
    """Rounds N(0, 1) values to a sign, {0, .5, 1, 1.5, 2, 3, 4, 6}, a scale per 16 columns and a power of two; every block's
    largest value is 6 and every row holds the largest scale, so that encoding it finds these very scales again."""
    t.mul_(2.2)
    a = t.abs().clamp_(max=6.0)
    q = torch.where(a < 2, (a * 2).round_().div_(2), torch.where(a < 4, a.round(), (a / 2).round_().mul_(2)))
    q.copysign_(t)
    b = q.view(*q.shape[:-1], -1, 16)
    b[..., 3] = torch.copysign(torch.full_like(b[..., 3], 6.0), b[..., 3])
    scale = 8 + torch.randint(0, 7, b.shape[:-1], device=t.device, generator=_gen("scale", t.shape[-1]), dtype=torch.int32)
    scale[..., 0] = 14
    b.mul_(scale.unsqueeze(-1).to(t.dtype))
    return q.mul_(2.0 ** round(math.log2(std / (2.4 * 11))))


def _fp8_values(t, std):
    """Rounds N(0, 1) values to e4m3 times a power of two; every 128 x 128 block holds the format's largest value."""
    q = (t * 100).clamp_(-448, 448).to(torch.float8_e4m3fn).to(t.dtype)
    q[..., ::128, ::128] = 448
    return q.mul_(2.0 ** round(math.log2(std / 100)))


def _weight(name, shape, form, seed):
    leaf = name.split(".", 1)[1] if "." in name else name
    g, last = _gen(name, seed), name.rsplit(".", 1)[-1]
    if last.endswith("norm"):
        t = 1 + 0.1 * torch.randn(shape, device="cuda", generator=g)
        t = t * 1.6 if last in ("q_norm", "k_norm") else t
    elif last == "A":
        t = -torch.exp(math.log(0.01) + math.log(100.0) * torch.rand(shape, device="cuda", generator=g))
    elif last in ("dt_bias", "conv_w"):
        t = torch.randn(shape, device="cuda", generator=g) * (0.1 if last == "dt_bias" else 0.4)
    else:
        t = torch.randn(shape, device="cuda", generator=g, dtype=torch.bfloat16)
        std = (DAMP[form] if leaf in RETURNS else 2.0 if last == "router" else 1.0) / math.sqrt(shape[-1])
        if form == "nvfp4" and leaf in EXPERTS:
            t = _nvfp4_values(t, std)
        elif form == "fp8" and leaf in FP8:
            t = _fp8_values(t, std)
        elif name != "tok_embd":
            t.mul_(std)
    return t if is_fp32_weight(name) else t.to(torch.bfloat16)


def _tokens(case, cfg, seed):
    g = torch.Generator().manual_seed(seed)
    n = sum(_lengths(case)) + case["seqs"]
    ids = torch.randint(0, cfg.vocab, (n,), generator=g).tolist()
    out = []
    for length in _lengths(case):
        out.append(ids[:length + (case["mode"] == "decode")])       # a decode step's token comes last
        ids = ids[length + 1:]
    return out


def _steps(case):
    """Tokens of each step that reads the prompts: one step for several, even chunks for a long one."""
    lengths = _lengths(case)
    if len(lengths) == 1:
        n = -(-lengths[0] // CHUNK)
        return -(-lengths[0] // n)
    return max(lengths)


def prepare(case, seed):
    torch.cuda.set_device(0)
    cfg, form = _config(case)
    w = {k: _weight(k, s, form, seed) for k, s in weight_shapes(cfg).items()}
    lengths = _lengths(case)
    ctx = max(CTX, -(-(max(lengths) + 256) // 1024) * 1024)
    model = Decoder(cfg, w, max_position=ctx + 8)
    model.fuse_gdn_in_proj()
    model.fuse_mla_in_proj()
    model.absorb_mla_q()
    if form == "nvfp4":
        model.fold_shared_experts()
        model.quantize_experts_nvfp4()
    elif form == "fp8":
        model.quantize_weights_fp8()
    eng = LmEngine(model, ByteTokenizer(cfg.vocab), EngineConfig(
        ctx_size=ctx, max_seqs=len(lengths), max_batch_tokens=CHUNK, prefill_chunk=CHUNK, block_size=64, prefix_cache=False,
        kv_cache_tokens=sum(-(-(n + 1) // 64) * 64 for n in lengths) + 64, device="cuda:0", model_name=MODELS[case["model"]][0]),
        start=False)
    state = dict(mode=case["mode"], eng=eng, tokens=_tokens(case, cfg, seed), step=_steps(case))
    if case["mode"] == "decode":
        # as a server warms up: one short exchange captures the step, then the chats so far are read
        warm = [eng.open_sequence("warm") for _ in lengths]
        for n in (2, 1):
            eng.feed([(s, [0] * n, []) for s in warm])
        for s in reversed(warm):
            eng.close_sequence(s)
        state["seqs"] = []
        for i, t in enumerate(state["tokens"]):
            s = eng.open_sequence(str(i))
            for at in range(0, len(t) - 1, CHUNK):
                eng.feed([(s, t[at:min(at + CHUNK, len(t) - 1)], [])])
            state["seqs"].append(s)
    return state


# ------------------------------------------------------------------------------------------------------------ a pass
def run(state):
    eng, tokens = state["eng"], state["tokens"]
    if state["mode"] == "decode":
        logits = eng.feed([(s, t[-1:], [0]) for s, t in zip(state["seqs"], tokens)])
        for s in state["seqs"]:         # the next pass generates the same token again
            s.tokens.pop()
            s.n_computed -= 1
    else:
        seqs = [eng.open_sequence(str(i)) for i in range(len(tokens))]
        longest = max(map(len, tokens))
        for at in range(0, longest, state["step"]):
            end = min(at + state["step"], longest)
            logits = eng.feed([(s, t[at:end], [len(t) - at - 1] if end >= len(t) else []) for s, t in zip(seqs, tokens)])
        for s in reversed(seqs):
            eng.close_sequence(s)
    out = {"logits": logits}
    for il, k in eng.kv.k.items():
        out[f"k{il}"] = k
        if eng.kv.v[il] is not k:
            out[f"v{il}"] = eng.kv.v[il]
    if eng.states is not None:
        for il in eng.states.ssm:
            out[f"ssm{il}"] = eng.states.ssm[il][:len(tokens)]
            out[f"conv{il}"] = eng.states.conv[il][:len(tokens)]
    return out


# -------------------------------------------------------------------------------------------------- what it cannot do without
def work(case):
    cfg, form = _config(case)
    lengths = _lengths(case)
    decode = case["mode"] == "decode"
    rows = len(lengths) if decode else sum(lengths)
    per = {"nvfp4": 0.5625, "fp8": 1.0, "bf16": 2.0}
    flops = 2.0 * len(lengths) * cfg.vocab * cfg.hidden
    nbytes = 2.0 * cfg.vocab * cfg.hidden + 4.0 * len(lengths) * cfg.vocab + 2.0 * rows * cfg.hidden
    pairs = sum(n + 1 for n in lengths) if decode else sum(n * (n + 1) / 2 for n in lengths)    # (query, key) pairs
    for name, shape in weight_shapes(cfg).items():
        if not name.startswith("l"):
            continue
        leaf, n = name.split(".", 1)[1], math.prod(shape)
        size = per[form] if (form == "nvfp4" and leaf in EXPERTS) or (form == "fp8" and leaf in FP8) else 2.0
        if leaf in ("moe.gate_up", "moe.down"):
            share = cfg.top_k / cfg.n_expert
            nbytes += size * n * (1 - (1 - share) ** rows)
            flops += 2.0 * rows * n * share
        elif len(shape) == 2 and leaf != "gdn.conv_w":
            nbytes += size * n
            flops += 2.0 * rows * n
    for kind in cfg.layer_kinds:
        if kind == "attn":
            cell = 4.0 * cfg.n_kv_head * cfg.head_dim
            flops += 4.0 * pairs * cfg.n_head * cfg.head_dim
        elif kind == "mla":
            cell = 2.0 * (cfg.kv_lora + cfg.qk_rope_dim)
            flops += 2.0 * pairs * cfg.n_head * (cfg.qk_nope_dim + cfg.qk_rope_dim + cfg.v_head_dim)
        else:
            state = cfg.gdn_v_heads * cfg.gdn_k_dim * cfg.gdn_v_dim
            nbytes += 8.0 * len(lengths) * (state + cfg.gdn_conv_channels() * (cfg.gdn_conv - 1))
            flops += 6.0 * rows * state
            continue
        nbytes += cell * (sum(lengths) + rows if decode else rows)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # bf16 activations between layers: 0.006 to 0.011 off the 64-bit results in the logits. 4- and 8-bit activations and the
    # choice of experts also turn a last bit into a whole step of theirs, for a few values
    return {"rel": 0.03}


# ------------------------------------------------------------------------------------------------------ in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.double()


def _rope(x, rot, theta):
    """x [n, heads, d]: columns (i, i + rot / 2) turn by position * theta^(-2 i / rot)."""
    half = rot // 2
    freq = theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    a = torch.arange(x.shape[0], device=x.device, dtype=torch.float64)[:, None, None] * freq
    c, s, p, q = a.cos(), a.sin(), x[..., :half], x[..., half:rot]
    return torch.cat([p * c - q * s, q * c + p * s, x[..., rot:]], -1)


def _softmax_rows(q, k, v, scale):
    """Causal attention of one sequence: q [n, H, d], k [n, G, d], v [n, G, e]."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(n, H, v.shape[2], device=q.device, dtype=torch.float64)
    step = max(16, (1 << 27) // (n * H))
    for a in range(0, n, step):
        b = min(n, a + step)
        s = torch.einsum("qgrd,kgd->grqk", q[a:b].view(b - a, G, H // G, -1), k[:b]) * scale
        s.masked_fill_(torch.arange(b, device=q.device)[None] > torch.arange(a, b, device=q.device)[:, None], -math.inf)
        out[a:b] = torch.einsum("grqk,kge->qgre", s.softmax(-1), v[:b]).reshape(b - a, H, -1)
    return out


def _attention(cfg, w, x):
    n, D, H, G = x.shape[0], cfg.head_dim, cfg.n_head, cfg.n_kv_head
    qkv = x @ w("attn.qkv").t()
    wide = H * D * (2 if cfg.gated_attn else 1)
    q = qkv[:, :wide].view(n, H, -1)
    k, v = qkv[:, wide:wide + G * D].view(n, G, D), qkv[:, wide + G * D:].view(n, G, D)
    gate, q = q[..., D:], q[..., :D]
    q = _rope(_rms(q, w("attn.q_norm"), cfg.rms_eps), cfg.rope_dim, cfg.rope_theta)
    k = _rope(_rms(k, w("attn.k_norm"), cfg.rms_eps), cfg.rope_dim, cfg.rope_theta)
    o = _softmax_rows(q, k, v, D ** -0.5)
    return (o * gate.sigmoid() if cfg.gated_attn else o).reshape(n, -1) @ w("attn.o").t()


def _latent(cfg, w, x):
    n, H, L = x.shape[0], cfg.n_head, cfg.kv_lora
    dn, dr, dv = cfg.qk_nope_dim, cfg.qk_rope_dim, cfg.v_head_dim
    q = (x @ w("mla.q").t()).view(n, H, dn + dr)
    kva = x @ w("mla.kv_a").t()
    kv = (_rms(kva[:, :L], w("mla.kv_a_norm"), cfg.rms_eps) @ w("mla.kv_b").t()).view(n, H, dn + dv)
    pe = _rope(kva[:, None, L:], dr, cfg.rope_theta).expand(n, H, dr)
    q = torch.cat([q[..., :dn], _rope(q[..., dn:], dr, cfg.rope_theta)], -1)
    o = _softmax_rows(q, torch.cat([kv[..., :dn], pe], -1), kv[..., dn:], (dn + dr) ** -0.5)
    return o.reshape(n, -1) @ w("mla.o").t()


def _delta(cfg, w, x):
    """Gated DeltaNet of one sequence from a cleared state, 64 tokens at a time: inside a block the corrections solve a
    unit lower-triangular system. Also returns the state [heads, k, v] and the last inputs of the convolution."""
    n, nk, nv, dk, dv = x.shape[0], cfg.gdn_k_heads, cfg.gdn_v_heads, cfg.gdn_k_dim, cfg.gdn_v_dim
    mixed, taps = x @ w("gdn.in_qkv").t(), cfg.gdn_conv
    z, ba = (x @ w("gdn.in_z").t()).view(n, nv, dv), x @ w("gdn.in_ba").t()
    padded = F.pad(mixed, (0, 0, taps - 1, 0))
    cw = w("gdn.conv_w")
    y = F.silu(sum(padded[i:i + n] * cw[:, i] for i in range(taps)))
    beta, g = ba[:, :nv].sigmoid(), w("gdn.A") * F.softplus(ba[:, nv:] + w("gdn.dt_bias"))
    q, k, v = y[:, :nk * dk].view(n, nk, dk), y[:, nk * dk:2 * nk * dk].view(n, nk, dk), y[:, 2 * nk * dk:].view(n, nv, dv)
    unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)      # noqa: E731
    heads = lambda t: t.repeat_interleave(nv // nk, 1)                             # noqa: E731
    m = -(-n // 64)

    def blocks(t):      # [n, heads, ...] -> [blocks, heads, 64, ...]; rows behind the end change nothing
        t = F.pad(t, (0, 0, 0, 0, 0, 64 * m - n) if t.dim() == 3 else (0, 0, 0, 64 * m - n))
        return t.view(m, 64, *t.shape[1:]).transpose(1, 2)
    q, k, v, beta, g = (blocks(t) for t in (heads(unit(q)) * dk ** -0.5, heads(unit(k)), v, beta, g))
    cum = g.cumsum(-1)                                                  # [blocks, heads, 64]
    low = torch.ones(64, 64, device=x.device, dtype=torch.bool).tril()
    ratio = (cum[..., :, None] - cum[..., None, :]).masked_fill(~low, -math.inf).exp()
    A = ((k @ k.mT) * ratio * beta[..., None]).tril(-1) + torch.eye(64, device=x.device, dtype=torch.float64)
    u = torch.linalg.solve_triangular(A, v * beta[..., None], upper=False, unitriangular=True)
    wk = torch.linalg.solve_triangular(A, k * (beta * cum.exp())[..., None], upper=False, unitriangular=True)
    inner, qd = (q @ k.mT) * ratio, q * cum.exp()[..., None]
    kd = k * (cum[..., -1:] - cum).exp()[..., None]
    S = torch.zeros(nv, dk, dv, device=x.device, dtype=torch.float64)
    o = torch.empty(m, nv, 64, dv, device=x.device, dtype=torch.float64)
    for i in range(m):
        d = u[i] - wk[i] @ S
        o[i] = qd[i] @ S + inner[i] @ d
        S = S * cum[i, :, -1, None, None].exp() + kd[i].mT @ d
    o = o.transpose(1, 2).reshape(64 * m, nv, dv)[:n]
    o = _rms(o, w("gdn.norm"), cfg.rms_eps) * F.silu(z)
    return o.reshape(n, -1) @ w("gdn.out").t(), S, padded[n:].t()


def _gated(x, gate_up, down):
    g, u = (x @ gate_up.double().t()).chunk(2, -1)
    return (F.silu(g) * u) @ down.double().t()


def _feed_forward(cfg, w, x, moe):
    if not moe:
        return torch.cat([_gated(c, w("mlp.gate_up"), w("mlp.down")) for c in x.split(CHUNK)])
    top, ids = (x @ w("moe.router").t()).softmax(-1).topk(cfg.top_k)
    top = top / top.sum(-1, keepdim=True)
    gate_up, down, y = w("moe.gate_up", False), w("moe.down", False), torch.zeros_like(x)
    order = ids.reshape(-1).argsort()
    ends = torch.bincount(ids.reshape(-1), minlength=cfg.n_expert).cumsum(0).tolist()
    for e, (a, b) in enumerate(zip([0] + ends, ends)):
        if a < b:
            at = order[a:b] // cfg.top_k
            y.index_add_(0, at, _gated(x[at], gate_up[e], down[e]) * top.reshape(-1)[order[a:b], None])
    if cfg.shared_ff:
        y += _gated(x, w("moe.sh_gate_up"), w("moe.sh_down")) * (x @ w("moe.sh_gate").t()).sigmoid()
    return y


@torch.no_grad()
def exact(case, seed):
    cfg, form = _config(case)
    tokens = _tokens(case, cfg, seed)
    shapes = weight_shapes(cfg)
    rows = sum(map(len, tokens))
    active = sum(math.prod(s) * (cfg.top_k / cfg.n_expert if k.split(".")[-1] in ("gate_up", "down") and ".moe." in k else 1)
                 for k, s in shapes.items() if k.startswith("l"))
    if 2.0 * rows * active > 2.5e14:
        return None                 # about ten seconds of double-precision products
    every = lambda name: _weight(name, shapes[name], form, seed)       # noqa: E731
    embed = every("tok_embd")
    x = embed[torch.tensor([t for s in tokens for t in s], device="cuda")].double()
    del embed
    cut = [len(t) for t in tokens]
    out = {}
    for il, kind in enumerate(cfg.layer_kinds):
        kept = {}

        def w(leaf, double=True):
            if leaf not in kept:
                kept[leaf] = every(f"l{il}.{leaf}")
                kept[leaf] = kept[leaf].double() if double else kept[leaf]
            return kept[leaf]
        h = _rms(x, w("attn_norm"), cfg.rms_eps).split(cut)
        if kind == "gdn":
            parts = [_delta(cfg, w, t) for t in h]
            out[f"ssm{il}"], out[f"conv{il}"] = (torch.stack([p[j] for p in parts]) for j in (1, 2))
            x = x + torch.cat([p[0] for p in parts])
            del parts
        else:
            x = x + torch.cat([(_latent if kind == "mla" else _attention)(cfg, w, t) for t in h])
            out[f"k{il}"] = None
            if kind != "mla":
                out[f"v{il}"] = None
        x = x + _feed_forward(cfg, w, _rms(x, w("ffn_norm"), cfg.rms_eps), cfg.is_moe_layer(il))
    last = torch.tensor(cut, device="cuda").cumsum(0) - 1
    out["logits"] = _rms(x[last], every("output_norm"), cfg.rms_eps) @ every("output").double().t()
    return out
