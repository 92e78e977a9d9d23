"""Prompt-sized steps: the de-quantising expert GEMM and latent attention in its per-head form, against plain operations."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def sm():
    from legion_b200.ops import sm100
    return sm100


def _rnd(*shape, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).to(DEV, torch.bfloat16)


# token tiles of 32 / 64 / 128, one and several raw stages of K, experts without a token, a last tile of one token
@pytest.mark.parametrize("T,E,k,H,F", [(33, 16, 2, 256, 256), (70, 32, 1, 512, 256), (321, 8, 1, 768, 512), (513, 4, 1, 256, 256),
                                        (130, 64, 3, 1024, 512)])
def test_moe_dequantised_prompt(T, E, k, H, F):
    from legion_b200.ops.sm100 import QWeight, Workspace
    qgu = QWeight.quantize(_rnd(E, 2 * F, H, scale=H ** -0.5), dual_rows=F)
    qd = QWeight.quantize(_rnd(E, H, F, scale=F ** -0.5, seed=1))
    x = _rnd(T, H, seed=2)
    g = torch.Generator().manual_seed(T)
    ids = torch.stack([torch.randperm(E - 1, generator=g)[:k] for _ in range(T)]).int().to(DEV)      # the last expert: none
    wts = torch.rand(T, k, generator=g).to(DEV)
    out = sm().moe_experts(x, ids, wts, qgu, qd, F).double()
    assert Workspace.get(DEV).check() == 0
    gu, dn = qgu.dequantize(torch.float32).double(), qd.dequantize(torch.float32).double()
    want = torch.zeros(T, H, dtype=torch.float64, device=DEV)
    for e in range(E):
        t, j = (ids == e).nonzero(as_tuple=True)
        a, b = (x[t].double() @ gu[e].t()).chunk(2, -1)
        h = (torch.nn.functional.silu(a) * b).to(torch.bfloat16).double()          # handed on in bf16
        want.index_add_(0, t, (h @ dn[e].t()).to(torch.bfloat16).double() * wts[t, j, None].double())
    # one bf16 rounding of the output, of the pair rows and (of a value near a tie) of the activations: 3 * 2^-9
    err = (out - want).norm() / want.norm()
    assert err < 3 * 2.0 ** -9, err


# a long portion alone, behind cached tokens, beside short portions and a decode row; sizes around the pages of 64
@pytest.mark.parametrize("lens,cached", [([192], 0), ([257, 3], 64), ([200, 1, 320], 37)])
def test_latent_prompt_per_head_form(lens, cached, monkeypatch):
    from legion_b200.config import ModelConfig
    from legion_b200.engine.lm import EngineConfig, build_engine
    from legion_b200.models.weights import random_weights
    cfg = ModelConfig(arch="deepseek_v3", n_layer=2, hidden=256, vocab=512, n_head=4, n_kv_head=4, head_dim=192, kv_lora=512,
                      qk_nope_dim=128, qk_rope_dim=64, v_head_dim=128, qk_norm=False, dense_ff=512)
    w = random_weights(cfg, DEV, torch.bfloat16, seed=0, std=0.05)
    out = []
    for least in (192, 1 << 30):                    # the per-head form, then everything in the latent space
        monkeypatch.setattr(sm(), "LATENT_EXPAND_MIN", least)
        eng = build_engine(cfg, weights=dict(w), device=DEV, engine_cfg=EngineConfig(
            ctx_size=1024, max_seqs=4, block_size=64, prefill_chunk=1024, max_batch_tokens=1024, prefix_cache=False), start=False)
        toks = [torch.randint(0, 512, (n + cached,), generator=torch.Generator().manual_seed(n)).tolist() for n in lens]
        seqs = [eng.open_sequence(str(i)) for i in range(len(lens))]
        if cached:
            eng.feed([(s, t[:cached], []) for s, t in zip(seqs, toks)])
        logits = eng.feed([(s, t[cached:], [n - 1]) for s, t, n in zip(seqs, toks, lens)])
        out.append((logits.double().cpu(), [k.double().cpu() for k in eng.kv.k.values()]))
        eng.shutdown()
    (a, ka), (b, kb) = out
    # two orders of bf16 roundings (keys and values against queries and attended latents), two layers
    assert (a - b).norm() < 0.01 * b.norm(), (a - b).norm() / b.norm()
    assert torch.equal(ka[0], kb[0]) and (ka[1] - kb[1]).norm() < 0.01 * kb[1].norm()


# tiles of 256 tokens with a remainder, features that end inside a pair of SMs (of one weight, and of gate and up: 2056), a last K
# block that is not whole
@pytest.mark.parametrize("T,N,K", [(1300, 4104, 584), (2304, 2560, 512), (1281, 4352, 1024), (1300, 4112, 584)])
def test_prompt_gemm_on_pairs(T, N, K):
    x, w, res = _rnd(T, K), _rnd(N, K, scale=K ** -0.5, seed=1), _rnd(T, N, seed=2)
    scale = torch.rand(T, generator=torch.Generator().manual_seed(3)).to(DEV)
    want = x.double() @ w.double().t()
    gate, up = want[:, :N // 2], want[:, N // 2:]
    for out, exact in ((sm().linear(x, w), want), (sm().linear(x, w, residual=res), want + res.double()),
                       (sm().linear(x, w, tok_scale=scale), want * scale.double()[:, None]),
                       (sm().gate_up_act(x, w, N // 2), torch.nn.functional.silu(gate) * up)):
        # fp32 sums of exact products of N(0, 1) values (about K^0.5 * 2^-24), fast exponential, one bf16 rounding
        assert (out.double() - exact).abs().max() < 2.0 ** -8 * exact.abs().max()
        assert (out.double() - exact).norm() < 2.0 ** -8 * exact.norm()
    assert sm().Workspace.get(DEV).check() == 0


# groups of 0, 1, 127, 128, 129 tokens and more over token tiles of 128, both expert products
def test_grouped_gemm_on_pairs():
    E, H, F = 48, 512, 640
    counts = [0, 1, 127, 128, 129, 300] * 8
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])
    ids = ids[torch.randperm(len(ids), generator=torch.Generator().manual_seed(0))].to(DEV)[:, None]
    T = len(ids)
    assert 64 * E < T <= 128 * E
    x, gu, dn = _rnd(T, H), _rnd(E, 2 * F, H, scale=H ** -0.5, seed=1), _rnd(E, H, F, scale=F ** -0.5, seed=2)
    wts = torch.rand(T, 1, generator=torch.Generator().manual_seed(4)).to(DEV)
    out = sm().moe_experts(x, ids, wts, gu, dn, F).double()
    assert sm().Workspace.get(DEV).check() == 0
    # the down projection runs on pairs from 64 tiles of 128 tokens on
    assert sm().Workspace.get(DEV)._cache["moe_plan", T, 1, E, 128, H, F].max_tiles >= 64
    want = torch.empty(T, H, dtype=torch.float64, device=DEV)
    for e in range(E):
        t = (ids[:, 0] == e).nonzero()[:, 0]
        a, b = (x[t].double() @ gu[e].double().t()).chunk(2, -1)
        h = (torch.nn.functional.silu(a) * b).to(torch.bfloat16).double()
        want[t] = (h @ dn[e].double().t()) * wts[t].double()
    # three bf16 roundings: the activations (of values near a tie), the pair rows, the output
    assert (out - want).norm() < 3 * 2.0 ** -9 * want.norm()


# token counts between decode steps and full tiles: every tile and split the dispatch takes
@pytest.mark.parametrize("T", [33, 65, 217, 600])
@pytest.mark.parametrize("N,K", [(1, 2048), (512, 2048), (2048, 4096), (12352, 2048), (576, 72)])
def test_short_prompt_gemm(T, N, K):
    x, w = _rnd(T, K), _rnd(N, K, scale=K ** -0.5, seed=1)
    want = x.double() @ w.double().t()
    for dt, eps in ((torch.bfloat16, 2.0 ** -8), (torch.float32, 2.0 ** -18)):
        assert (sm().linear(x, w, out_dtype=dt).double() - want).norm() < eps * want.norm()
    assert sm().Workspace.get(DEV).check() == 0


# pairs of 256 query rows: one row more than a tile, an empty second tile, full pairs, short sequences beside long ones, cached
# tokens in front; blocks of 128 keys with a remainder; head sizes between and at the kernel's, pages of a part of its tiles
@pytest.mark.parametrize("q_lens,cached,page", [([129], 0, 64), ([256, 1, 130], 70, 16), ([257, 511], 128, 32), ([1100, 128], 333, 64),
                                                ([1024], 0, 16), ([1300, 5], 61, 32)])
@pytest.mark.parametrize("Hq,Hkv,dk,dv", [(4, 2, 128, 128), (2, 2, 192, 128), (8, 1, 160, 96), (2, 1, 136, 72), (2, 1, 72, 72)])
def test_prefill_attention_on_pairs(q_lens, cached, page, Hq, Hkv, dk, dv):
    n, T = len(q_lens), sum(q_lens)
    ctx = [q + cached for q in q_lens]
    width = -(-max(ctx) // page)
    k, v = _rnd(n * width, page, Hkv, dk, seed=1), _rnd(n * width, page, Hkv, dv, seed=2)
    q = _rnd(T, Hq, dk, scale=2.0, seed=3)
    bt = torch.randperm(n * width, generator=torch.Generator().manual_seed(0)).int().view(n, width).to(DEV)
    cu = torch.tensor([sum(q_lens[:i]) for i in range(n + 1)], dtype=torch.int32, device=DEV)
    out = sm().prefill_attn(q, k, v, cu, torch.tensor(ctx, dtype=torch.int32, device=DEV), bt, max(q_lens), dk ** -0.5, pairs=True)
    assert sm().Workspace.get(DEV).check() == 0
    for i in range(n):
        kk = k[bt[i].long()].reshape(-1, Hkv, dk)[:ctx[i]].double().repeat_interleave(Hq // Hkv, 1)
        vv = v[bt[i].long()].reshape(-1, Hkv, dv)[:ctx[i]].double().repeat_interleave(Hq // Hkv, 1)
        a, b = sum(q_lens[:i]), sum(q_lens[:i + 1])
        s = torch.einsum("qhd,khd->hqk", q[a:b].double(), kk) * dk ** -0.5
        later = torch.arange(ctx[i], device=DEV)[None] > torch.arange(cached, ctx[i], device=DEV)[:, None]
        want = torch.einsum("hqk,khd->qhd", s.masked_fill(later, float("-inf")).softmax(-1), vv)
        # bf16 probabilities and output, 2^-9 each; single rows up to 2^-6 of the largest value
        assert (out[a:b].double() - want).norm() < 2.0 ** -8 * want.norm()
        assert (out[a:b].double() - want).abs().max() < 2.0 ** -6 * want.abs().max()


# tiles of 32, 64, 128 and 256 tokens with a remainder, several per head; rows of an odd width leave one by one
@pytest.mark.parametrize("T", [1, 33, 100, 257, 1000])
@pytest.mark.parametrize("nh,nf,rows", [(3, 128, 192), (5, 72, 72), (2, 130, 256)])
@pytest.mark.parametrize("own", [False, True])
def test_per_head_products_keep_nothing_for_a_token_count(T, nh, nf, rows, own):
    K = 64
    x, w = _rnd(T, nh * K if own else K), _rnd(nh * rows, K, scale=K ** -0.5, seed=1)
    cache = sm().Workspace.get(DEV)._cache
    before = set(cache)
    out = torch.full((T * nh + 4, nf), 3.0, dtype=torch.bfloat16, device=DEV)
    sm().head_linear(x, w, nh, rows, nf, K, K if own else 0, out[:T * nh])
    assert set(cache) == before and sm().Workspace.get(DEV).check() == 0
    wh = w.view(nh, rows, K)[:, :nf].double()
    want = torch.einsum("thk,hnk->thn" if own else "tk,hnk->thn", x.double().view(T, nh, K) if own else x.double(), wh)
    assert (out[:T * nh].view(T, nh, nf).double() - want).abs().max() < 2.0 ** -8 * want.abs().max()      # one bf16 rounding
    assert (out[T * nh:] == 3).all()


# contexts shorter than their portions (and none at all): rows in front of the first token see nothing and give zeros
@pytest.mark.parametrize("dk,dv,q_lens", [(192, 128, (700, 300, 400)), (128, 128, (2048, 300, 1100))])
@pytest.mark.parametrize("pairs", [False, True])
def test_prefill_attention_rows_without_a_key(dk, dv, q_lens, pairs):
    Hq, Hkv, page, ctx = 4, 2, 64, (q_lens[0], 0, 150)
    width, T = -(-q_lens[0] // page), sum(q_lens)
    k, v = _rnd(3 * width, page, Hkv, dk, seed=1), _rnd(3 * width, page, Hkv, dv, seed=2)
    q = _rnd(T, Hq, dk, seed=3)
    bt = torch.arange(3 * width, dtype=torch.int32, device=DEV).view(3, width)
    cu = torch.tensor([sum(q_lens[:i]) for i in range(4)], dtype=torch.int32, device=DEV)
    out = torch.full((T, Hq, dv), 7.0, dtype=torch.bfloat16, device=DEV)
    sm().prefill_attn(q, k, v, cu, torch.tensor(ctx, dtype=torch.int32, device=DEV), bt, max(q_lens), dk ** -0.5, out=out, pairs=pairs)
    assert sm().Workspace.get(DEV).check() == 0
    parts = out.double().split(q_lens)
    assert not parts[1].any() and not parts[2][:q_lens[2] - 150].any()
    for i, n in ((0, q_lens[0]), (2, 150)):
        kk = k[bt[i].long()].reshape(-1, Hkv, dk)[:n].double().repeat_interleave(Hq // Hkv, 1)
        vv = v[bt[i].long()].reshape(-1, Hkv, dv)[:n].double().repeat_interleave(Hq // Hkv, 1)
        s = torch.einsum("qhd,khd->hqk", q.split(q_lens)[i][-n:].double(), kk) * dk ** -0.5
        s.masked_fill_(torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1), float("-inf"))
        want = torch.einsum("hqk,khd->qhd", s.softmax(-1), vv)
        # bf16 probabilities and output, 2^-9 each
        assert (parts[i][-n:] - want).norm() < 2.0 ** -8 * want.norm()


# query and key preparation and the gate (eight columns per thread, one where rows do not lie on 16 bytes): partial and whole rotation,
# a token without a cell, a last warp that is not full
@pytest.mark.parametrize("T,Hq,Hkv,D,rot,gated,shift", [(5, 3, 1, 64, 64, False, 0), (130, 4, 2, 128, 128, False, 0), (33, 2, 1, 256, 64, True, 0),
                                                        (7, 5, 3, 128, 0, False, 0), (9, 3, 1, 128, 64, True, 1)])
def test_qk_prep_and_gate(T, Hq, Hkv, D, rot, gated, shift):
    from legion_b200.ops import reference as ref
    S = D * (2 if gated else 1)
    wide = Hq * S + 2 * Hkv * D
    qkv = _rnd(T, wide + shift)[:, shift:]
    qw, kw = (1 + 0.1 * torch.randn(D, generator=torch.Generator().manual_seed(i)).to(DEV) for i in (1, 2))
    cs = ref.rope_cos_sin(512, max(rot, 64), 1e4, None, device=DEV)
    pos = torch.randint(0, 512, (T,), generator=torch.Generator().manual_seed(3)).int().to(DEV)
    slots = torch.randperm(4 * 64, generator=torch.Generator().manual_seed(4))[:T].to(DEV)
    slots[T // 2] = -1
    kc, vc = torch.zeros(4, 64, Hkv, D, dtype=torch.bfloat16, device=DEV), torch.zeros(4, 64, Hkv, D, dtype=torch.bfloat16, device=DEV)
    out = sm().qk_norm_rope_append(qkv, Hq, Hkv, D, qw, kw, 1e-6, 0.0, cs, rot, pos, slots, kc, vc, gated)
    x = qkv.double()
    heads = x[:, :Hq * S].view(T, Hq, S)

    def prep(v, w):
        v = v * torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-6) * w.double()
        if rot:
            c, s = cs[pos.long()].double()[:, None, :rot].chunk(2, -1)
            a, b = v[..., :rot // 2].clone(), v[..., rot // 2:rot].clone()
            v = torch.cat([a * c - b * s, b * c + a * s, v[..., rot:]], -1)
        return v
    # one bf16 rounding of fp32 values
    close = lambda a, b: ((a.double() - b).abs() <= 2.0 ** -8 * b.abs() + 1e-5).all()       # noqa: E731
    assert close(out, prep(heads[..., :D], qw))
    live = slots >= 0
    k = prep(x[:, Hq * S:Hq * S + Hkv * D].view(T, Hkv, D), kw)
    assert close(kc.view(-1, Hkv, D)[slots[live]], k[live])
    assert torch.equal(vc.view(-1, Hkv, D)[slots[live]].double(), x[:, Hq * S + Hkv * D:].view(T, Hkv, D)[live])
    assert int((kc.view(-1, Hkv * D).abs().sum(-1) > 0).sum()) == T - 1
    if gated:
        o = sm().sigmoid_gate(out, qkv, Hq, D)
        assert close(o.view(T, Hq, D), out.double() * torch.sigmoid(heads[..., D:]))
