"""Rules that choose between kernels, at sizes where both sides were measured."""
from types import SimpleNamespace

import pytest
import torch

from legion_b200.engine.cuda_graphs import DecodeGraphs
from legion_b200.ops import sm100


# longest portion, others, their length, keys in front of the longest, heads, head size -> on pairs of SMs
@pytest.mark.parametrize("longest,others,rows,cached,heads,dk,pairs", [
    (1023, 0, 0, 0, 32, 128, False), (1100, 15, 80, 0, 32, 128, False), (1100, 8, 300, 0, 32, 128, False),
    (2048, 15, 128, 0, 32, 128, False), (1100, 15, 80, 0, 40, 128, False), (4096, 0, 0, 0, 32, 128, True),
    (2048, 0, 0, 0, 40, 128, True), (2048, 0, 0, 2048, 32, 128, True), (1600, 0, 0, 0, 8, 128, True),
    (130, 0, 0, 0, 32, 192, False), (256, 0, 0, 0, 32, 192, False), (1100, 15, 80, 0, 32, 192, False),
    (300, 7, 300, 0, 128, 192, False), (128, 0, 0, 4096, 32, 192, False), (130, 0, 0, 2048, 32, 192, True),
    (512, 0, 0, 0, 32, 192, True), (2048, 15, 128, 0, 32, 192, True), (6001, 0, 0, 0, 32, 192, True), (600, 7, 600, 0, 32, 192, True),
])
def test_prompt_attention_takes_the_faster_kernel(longest, others, rows, cached, heads, dk, pairs):
    ctx = -(-(longest + cached) // 64) * 64
    assert sm100.attn_on_pairs(longest + others * rows, 1 + others, longest, ctx, heads, dk) is pairs


# tokens, features, K, gate and up, float32 -> token tile, where both sides were measured
@pytest.mark.parametrize("T,n,K,dual,f32,bn", [
    (128, 512, 2048, False, False, 32), (64, 1024, 2048, True, False, 32), (256, 768, 768, False, False, 32),
    (300, 5120, 5120, False, False, 128), (130, 6176, 2048, True, False, 64),
    (64, 2048, 2048, False, False, 64), (256, 2048, 2048, False, False, 256), (512, 2048, 2048, False, True, 256),
    (512, 3072, 1024, False, True, 256), (64, 768, 768, False, True, 64), (96, 12352, 2048, False, False, 128),
    (256, 576, 4096, False, False, 32), (384, 576, 4096, False, False, 256), (96, 576, 4096, False, False, 32), (48, 576, 4096, False, False, 64),
    (130, 3072, 1024, False, False, 256), (217, 1024, 2048, True, False, 128), (1024, 3072, 1024, False, False, 256), (4096, 5120, 5120, False, False, 256)])
def test_short_prompt_products_take_the_faster_tile(T, n, K, dual, f32, bn):
    got, sk = sm100._pick_tile(T, n, K, dual, f32)
    wide = sm100.pick_bn(T, dual)
    assert got == bn and sk == sm100._pick_split_k(-(-T // wide), -(-n // 128), K)


# a batch without rows, rows that are fewer than the longest portion said to be there, one sequence of no rows beside a long one
@pytest.mark.parametrize("T,n,longest,ctx", [(0, 1, 0, 0), (10, 1, 4096, 64), (4096, 2, 4096, 4096)])
def test_prompt_attention_rule_takes_any_sizes(T, n, longest, ctx):
    for dk in (64, 128, 192, 256):
        assert isinstance(sm100.attn_on_pairs(T, n, longest, ctx, 32, dk), bool)


# weights of the experts -> rows of a decode step that run as two halves
@pytest.mark.parametrize("kind,two", [(None, ()), ("QWeight", ()), ("Nv4Weight", (96, 128)), ("Fp8Weight", (64,))])
def test_decode_steps_that_run_as_two_halves(kind, two, monkeypatch):
    monkeypatch.setitem(sm100.TUNE, "decode_lanes", 1)
    w = {"l0.attn.o": object.__new__(sm100.Nv4Weight), "l0.mlp.down": object.__new__(sm100.Fp8Weight),
         "l1.moe.down": object.__new__(getattr(sm100, kind)) if kind else None}
    eng = SimpleNamespace(mcfg=SimpleNamespace(parallel_sublayers=False), dp_world=1,
                          model=SimpleNamespace(w=w, pctx=SimpleNamespace(world=1), expert_cache=None))
    g = SimpleNamespace(eng=eng)
    g._halves = lambda B: DecodeGraphs._halves(g, B)
    rows = (1, 48, 64, 96, 128, 192, 256)
    assert tuple(B for B in rows if DecodeGraphs._lanes(g, B) == 2) == two
    monkeypatch.setitem(sm100.TUNE, "decode_lanes", 2)
    assert tuple(B for B in rows if DecodeGraphs._lanes(g, B) == 2) == (64, 96, 128, 192, 256)
    eng.model.pctx.world = 2
    assert all(DecodeGraphs._lanes(g, B) == 1 for B in rows)


def test_nvfp4_experts_refuse_always_chosen_experts_in_the_tables():
    """Their tile bound and their combine know the pairs and one shared slot."""
    E, k, T = 8, 2, 3
    w = sm100.Nv4Weight(torch.zeros(E + 2, 512, 128, dtype=torch.uint8), None, torch.ones(E + 2))
    ids = torch.zeros(T, k, dtype=torch.int32)
    r = sm100.Routing(ids, torch.ones(T, k), SimpleNamespace(n_slots=E + 2, bn=32, stride=32, hq=None, y_pairs=None), None, 0, E)
    r.shared_rows = 2
    with pytest.raises(NotImplementedError):
        sm100._moe_experts_nv4(torch.zeros(T, 256, dtype=torch.bfloat16), ids, r.wts, w, w, 256, 0, None, None, None, None, None, r)


# tokens of a step and context: the smallest long portion behind a long history, one at the limit, a whole prompt
@pytest.mark.parametrize("tokens,ctx", [(192, 4096), (192, 65536), (2048, 16384), (4096, 4096), (300, 512)])
def test_memory_plan_counts_the_expanded_keys_of_latent_prompts(tokens, ctx, monkeypatch):
    from legion_b200.config import ModelConfig
    from legion_b200.engine import memory_plan
    from legion_b200.engine.lm import EngineConfig, LmEngine
    heads, dim, rot, vdim, rank, seqs = 8, 128, 64, 128, 512, 3
    kv_b, cache = torch.empty(heads * (dim + vdim), rank, dtype=torch.bfloat16), torch.empty(1, 64, 1, rank + rot, dtype=torch.bfloat16)
    q = torch.empty(tokens, heads, dim + rot, dtype=torch.bfloat16)
    most = 0
    for portions in range(1, seqs + 1):
        if tokens // portions < sm100.LATENT_EXPAND_MIN:
            continue
        for pages in (1, ctx // 128 * portions, -(-ctx // 64) * portions):
            p = sm100.LatentPart()
            p.expand, p.pages = True, torch.empty(2, max(1, pages), dtype=torch.int32)
            if sm100.mla_expand_ok(q, kv_b, cache, p, heads, dim, rot, vdim, rank):
                most = max(most, max(1, pages) * 64 * (heads * (dim + rot + vdim) + rank) * 2)
    granted = sm100.mla_expand_bytes(tokens, seqs, ctx, heads, dim, rot, vdim, rank)
    assert 0 < most <= granted
    cfg = ModelConfig(arch="deepseek_v3", n_layer=1, hidden=1024, vocab=512, n_head=heads, n_kv_head=heads, head_dim=dim + rot, kv_lora=rank,
                      qk_nope_dim=dim, qk_rope_dim=rot, v_head_dim=vdim, qk_norm=False, dense_ff=512)
    eng = SimpleNamespace(mcfg=cfg, ring_len=0, hybrid=False, cfg=EngineConfig(ctx_size=ctx, max_seqs=seqs, max_batch_tokens=tokens,
                                                                              block_size=64, kv_cache_tokens=-1))
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda dev: (100 << 30, 180 << 30))
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda dev: 0)
    LmEngine._plan_memory(eng, SimpleNamespace(dtype=torch.bfloat16, n_kv_l=heads, n_head_l=heads, pctx=SimpleNamespace(tp=1)),
                          torch.device("cpu"), 0, None, 64)
    assert eng.memory_plan.workspace_bytes == memory_plan.workspace_reserve(1024, 512, tokens, seqs, 0, 0, 0) + granted
