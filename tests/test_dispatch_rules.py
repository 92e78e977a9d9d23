"""Rules that choose between kernels, at sizes where both sides were measured."""
import pytest

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


# a batch without rows, rows that are fewer than the longest portion said to be there, one sequence of no rows beside a long one
@pytest.mark.parametrize("T,n,longest,ctx", [(0, 1, 0, 0), (10, 1, 4096, 64), (4096, 2, 4096, 4096)])
def test_prompt_attention_rule_takes_any_sizes(T, n, longest, ctx):
    for dk in (64, 128, 192, 256):
        assert isinstance(sm100.attn_on_pairs(T, n, longest, ctx, 32, dk), bool)
