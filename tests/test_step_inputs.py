"""The input record of a step: native packer and Python form give the same tensors."""
from types import SimpleNamespace

import pytest
import torch

from legion_b200.engine.lm import LmEngine
from legion_b200.kv import blocks as kv_blocks


def _seq(blocks, slot, media=None):
    table = kv_blocks.BlockTable()
    table.blocks = blocks
    return SimpleNamespace(table=table, slot=slot, media=media, rope_pos=lambda p: p + 1000)


# one token, a block's end, several blocks with positions from the middle, no wanted rows, rotary positions of their own
@pytest.mark.parametrize("items,rows", [
    ([(_seq([5], 3), 0, [7])], [0]),
    ([(_seq([2, 9, 4], 0), 0, list(range(48)))], []),
    ([(_seq([1, 8, 6], 2), 20, list(range(100, 121))), (_seq([3], 1), 15, [11]), (_seq([0, 7], 4, media=1), 9, [1, 2, 3, 4, 5, 6, 7, 8])],
     [20, 21, 29]),
])
def test_native_and_python_step_inputs_agree(items, rows, monkeypatch):
    if kv_blocks.NATIVE is None:
        pytest.skip("native host runtime not built")
    eng = SimpleNamespace(pool=kv_blocks.BlockPool(16, 16), device=torch.device("cpu"))
    a = LmEngine._step_inputs(eng, items, rows)
    monkeypatch.setattr(kv_blocks, "NATIVE", None)
    b = LmEngine._step_inputs(eng, items, rows)
    for name in ("token_ids", "positions", "cu_q", "ctx_lens", "block_table", "slots", "state_slots", "logit_rows"):
        x, y = getattr(a, name), getattr(b, name)
        assert x.dtype == y.dtype and torch.equal(x, y), name
    assert a.token_ids.tolist() == [t for _, _, toks in items for t in toks] and a.logit_rows.tolist() == rows
    assert a.slots.tolist() == [s.table.blocks[p // 16] * 16 + p % 16 for s, p0, t in items for p in range(p0, p0 + len(t))]
    assert a.positions.tolist() == [p + (1000 if s.media else 0) for s, p0, t in items for p in range(p0, p0 + len(t))]


def test_native_step_inputs_refuse_positions_beyond_the_table():
    if kv_blocks.NATIVE is None:
        pytest.skip("native host runtime not built")
    eng = SimpleNamespace(pool=kv_blocks.BlockPool(16, 16), device=torch.device("cpu"))
    with pytest.raises(IndexError):
        LmEngine._step_inputs(eng, [(_seq([5], 3), 10, list(range(8)))], [0])


# a token id, a rotary position: refused by both forms
@pytest.mark.parametrize("tokens,media", [([7, 2 ** 31], None), ([-2 ** 31 - 1], None), ([7], 1)])
def test_step_inputs_refuse_values_beyond_32_bits(tokens, media, monkeypatch):
    eng = SimpleNamespace(pool=kv_blocks.BlockPool(16, 16), device=torch.device("cpu"))
    seq = _seq([5], 3, media)
    seq.rope_pos = lambda p: p + 2 ** 31
    with pytest.raises(RuntimeError):
        LmEngine._step_inputs(eng, [(seq, 0, tokens)], [0])
    monkeypatch.setattr(kv_blocks, "NATIVE", None)
    with pytest.raises(RuntimeError):
        LmEngine._step_inputs(eng, [(seq, 0, tokens)], [0])
