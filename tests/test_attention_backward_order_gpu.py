"""Attention backward in both orders of its grid (all heads of a key tile first, or all key tiles of a head), with several batches and
ragged last tiles, and with one and several steps a block."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _close(got, want):
    # probabilities and their gradients are rounded to bf16 before each product, results to bf16
    assert torch.isfinite(got).all() and ((got.float() - want).norm() / want.norm()).item() < 2e-2


@pytest.mark.parametrize("B,L,Hq,Hkv,C,S,W", [
    (2, 1500, 4, 2, 64, 1, 1),      # a window of two chunks: head by head
    (3, 1029, 6, 2, 128, 2, 1),
    (2, 513, 4, 2, 128, 1, 3),      # a window over the whole sequence: tile by tile
    (3, 129, 2, 2, 64, 1, 1),       # one head a group: blocks of one and of two steps
    (1, 100, 1, 1, 128, 1, 8),
])
def test_summary_attention_gradients(B, L, Hq, Hkv, C, S, W):
    torch.manual_seed(L)
    Ns = (L + C - 1) // C * S
    t = [torch.randn(B, T, H, 128, device="cuda").bfloat16()
         for T, H in ((L, Hq), (L, Hkv), (L, Hkv), (Ns, Hq), (Ns, Hkv), (Ns, Hkv))]
    xs, fs = [x.clone().requires_grad_() for x in t], [x.float().requires_grad_() for x in t]
    got, want = ops.ksa_attention(*xs, C, S, W), ref.ksa_attention(*fs, C, S, W)
    g = [torch.randn(o.shape, device="cuda").bfloat16() for o in got]
    torch.autograd.backward(list(got), g)
    torch.autograd.backward(list(want), [x.float() for x in g])
    for x, f in zip(xs, fs):
        _close(x.grad, f.grad)


@pytest.mark.parametrize("B,L,window", [(3, 300, -1), (1, 1, -1), (2, 128, -1), (2, 1100, 100), (2, 600, 500)])
def test_causal_gradients(B, L, window):
    torch.manual_seed(L)
    t = [torch.randn(B, L, H, 128, device="cuda").bfloat16() for H in (4, 2, 2)]
    xs, fs = [x.clone().requires_grad_() for x in t], [x.float().requires_grad_() for x in t]
    got, want = ops.causal_attention(*xs, window=window), ref.causal_attention(*fs, 128 ** -0.5, window)
    g = torch.randn(B, L, 4, 128, device="cuda").bfloat16()
    got.backward(g)
    want.backward(g.float())
    if L == 1:                       # one key: its probability is one, so the scores' gradients are rounding alone
        _close(xs[2].grad, fs[2].grad)
        return
    for x, f in zip(xs, fs):
        _close(x.grad, f.grad)
