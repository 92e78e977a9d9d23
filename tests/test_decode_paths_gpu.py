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


# token tiles of 64: an expert with a single token, with eight, nine and all of them, tokens in one half and in both; the last sizes
# have tiles for two CTAs per SM (2 x 148 of gate and up) and eight feature tiles of the down projection
@pytest.mark.parametrize("T", [33, 40, 64])
@pytest.mark.parametrize("E,k,H,F", [(96, 2, 256, 256), (64, 4, 512, 512), (96, 4, 1024, 512)])
def test_nvfp4_experts_sparse_columns(T, E, k, H, F):
    S = sm()
    gu, dn = _rnd(E, 2 * F, H, scale=H ** -0.5), _rnd(E, H, F, scale=F ** -0.5, seed=1)
    x = _rnd(T, H, seed=2)
    # router weights that send every token to expert 0, nine of them to expert 1, eight to expert 2
    w_r = _rnd(E, H, scale=H ** -0.5, seed=3).float()
    inv = torch.linalg.pinv(x.double().cpu()).to(DEV)
    hit = torch.zeros(T, 3, device=DEV, dtype=torch.float64)
    hit[:, 0] = 9.0
    hit[:, 1:] = -4.0
    hit[:9, 1], hit[T - 8:, 2] = 6.0, 6.0
    w_r[:3] = (inv @ hit).t().float()
    w_r = w_r.to(torch.bfloat16)
    qgu, qdn = S.Nv4Weight.quantize_cuda(gu, dual_rows=F), S.Nv4Weight.quantize_cuda(dn)
    r = S.router(x, w_r, k, slot_stride=128)
    counts = torch.bincount(r.ids.flatten().long(), minlength=3)
    assert counts[0] == T and counts[1] >= 9 and counts[2] >= 8
    out = S.moe_experts(x, r.ids, r.wts, qgu, qdn, F, routing=r).double()
    assert S.Workspace.get(DEV).check() == 0
    dgu, ddn = qgu.dequantize(torch.float32).double(), qdn.dequantize(torch.float32).double()
    xq = S.nv4_quant_act(x).dequantize()[:T].double()
    want = torch.zeros(T, H, dtype=torch.float64, device=DEV)
    for e in r.ids.unique().tolist():
        t, j = (r.ids == e).nonzero(as_tuple=True)
        a, b = (xq[t] @ dgu[e].t()).chunk(2, -1)
        want.index_add_(0, t, (torch.nn.functional.silu(a) * b) @ ddn[e].t() * r.wts[t, j, None].double())
    # activations in 4 bits with a scale per 16: a tenth of their size, summed over F of them and the experts of a token
    assert (out - want).norm() < 0.12 * want.norm()
    # the same sums as in token tiles of 32
    for part in (slice(0, 32), slice(32, T)):
        h = S.router(x[part].contiguous(), w_r, k, slot_stride=128)
        assert torch.equal(h.ids, r.ids[part]) and torch.equal(h.wts, r.wts[part])
        assert torch.equal(S.moe_experts(x[part].contiguous(), h.ids, h.wts, qgu, qdn, F, routing=h).double(), out[part])
