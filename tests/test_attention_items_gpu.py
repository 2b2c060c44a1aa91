"""Attention forward over many work items a thread block: the products of one item follow those of the one before, and its
output is read while they do."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,L,Hq,Hkv,D", [
    (80, 1, 8, 4, 128),        # items of one tile, two to three a block
    (80, 128, 8, 4, 128),
    (60, 129, 8, 4, 128),      # items of one and of two tiles in turn
    (70, 100, 8, 4, 64),
    (50, 300, 3, 1, 128),      # one query head an item
    (1, 257, 2, 1, 128),       # fewer items than blocks
])
@pytest.mark.parametrize("grow", [0.0, 8.0])     # scores that grow along the keys: the running maximum is exceeded in most tiles
def test_items_in_one_sequence(B, L, Hq, Hkv, D, grow):
    torch.manual_seed(L + Hq)
    q, k, v = [torch.randn(B, L, H, D, device="cuda") for H in (Hq, Hkv, Hkv)]
    k = k * (1.0 + grow * torch.arange(L, device="cuda").view(1, L, 1, 1) / L)
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    with torch.no_grad():
        got = ops.causal_attention(q, k, v)
        again = ops.causal_attention(q, k, v)
    want = ref.causal_attention(q.float(), k.float(), v.float(), D ** -0.5)
    assert torch.equal(got, again)
    # probabilities and results in bf16: 2^-9 each
    assert torch.isfinite(got).all() and ((got.float() - want).norm() / want.norm()).item() < 1e-2
    assert (got.float() - want).abs().max().item() < 0.05 * want.abs().max().item()


@pytest.mark.parametrize("B,L,C,S,W", [(12, 700, 64, 2, 2), (3, 1500, 128, 1, 3)])
def test_items_with_summaries(B, L, C, S, W):
    torch.manual_seed(L)
    Hq, Hkv, D, Ns = 8, 4, 128, (L + C - 1) // C * S
    t = [torch.randn(B, T, H, D, device="cuda").bfloat16()
         for T, H in ((L, Hq), (L, Hkv), (L, Hkv), (Ns, Hq), (Ns, Hkv), (Ns, Hkv))]
    with torch.no_grad():
        got = ops.ksa_attention(*t, C, S, W)
        want = ref.ksa_attention(*[x.float() for x in t], C, S, W)
    for a, b in zip(got, want):
        assert torch.isfinite(a).all() and ((a.float() - b).norm() / b.norm()).item() < 1e-2
