"""Decode-sized steps: attention under more splits than a sequence has tiles, expert products with sparse token columns."""
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


# tiles of 128 keys: none left for most splits, one key in the last, exactly full, more tiles than splits
@pytest.mark.parametrize("splits", [1, 5, 64])
@pytest.mark.parametrize("ctx,heads,D", [((1, 127, 128, 129), (8, 2), 128), ((1000,), (16, 2), 256), ((8192, 3), (4, 4), 72)])
def test_decode_attention_live_splits(ctx, heads, D, splits):
    B, (Hq, Hkv) = len(ctx), heads
    width = -(-max(ctx) // 64)
    k, v = _rnd(B * width, 64, Hkv, D, seed=1), _rnd(B * width, 64, Hkv, D, seed=2)
    bt = torch.randperm(B * width, generator=torch.Generator().manual_seed(0)).int().view(B, width).to(DEV)
    q, scale = _rnd(B, Hq, D, seed=3), D ** -0.5
    cl = torch.tensor(ctx, dtype=torch.int32, device=DEV)
    raw = torch.empty(B * Hq * D + 1, dtype=torch.bfloat16, device=DEV)
    for out in (raw[:-1].view(B, Hq, D), raw[1:].view(B, Hq, D)):          # 16-byte aligned rows, and rows that are not
        for _ in range(2):                                              # the arrival counters are left at zero
            sm().paged_decode(q, k, v, bt, cl, scale, n_splits=splits, out=out)
        for b, n in enumerate(ctx):
            kk = k[bt[b].long()].reshape(-1, Hkv, D)[:n].double().repeat_interleave(Hq // Hkv, 1)
            vv = v[bt[b].long()].reshape(-1, Hkv, D)[:n].double().repeat_interleave(Hq // Hkv, 1)
            p = (torch.einsum("hd,khd->hk", q[b].double(), kk) * scale).softmax(-1)
            want = torch.einsum("hk,khd->hd", p, vv)
            # bf16 probabilities (2^-9 each) and output (2^-9)
            assert (out[b].double() - want).norm() < 2.0 ** -8 * want.norm()
    assert sm().Workspace.get(DEV).check() == 0
