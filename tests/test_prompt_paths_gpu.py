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
