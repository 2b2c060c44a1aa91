"""Attention backward with the saved output at an address of its own, as a saved-tensor hook may hand it back."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 4, 5])                 # bf16 elements: 16-, 8- and 2-byte alignment
@pytest.mark.parametrize("B,L,summary", [(1, 128, False), (2, 300, True)])
def test_output_at_any_address(offset, B, L, summary):
    torch.manual_seed(L)
    Hq, Hkv, D, C, S, W = 4, 2, 128, 128, 1, 1
    Ns = L // C if summary else 0
    rows = B * (L + Ns)
    qkv = torch.randn(rows, (Hq + 2 * Hkv) * D, device="cuda").bfloat16()
    g = torch.randn(rows, Hq * D, device="cuda").bfloat16()

    def grad(unpack):
        x = qkv.clone().requires_grad_()
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            ops.attention_packed(x, B, L, Ns, Hq, Hkv, D, C, S, W if summary else ops.UNBOUNDED_WINDOW).backward(g)
        _lib.check_status()
        return x.grad.float()

    def moved(t):
        if t.shape != g.shape:
            return t
        buf = torch.full((t.numel() + 8,), float("nan"), device="cuda", dtype=t.dtype)
        out = buf[offset:offset + t.numel()].view(t.shape)
        out.copy_(t)
        assert out.data_ptr() % 16 == offset * 2 % 16
        return out

    want, got = grad(lambda t: t), grad(moved)
    # the sums of dQ come in another order each time: one rounding to bf16 may go the other way
    assert (got - want).norm() <= 2.0 ** -8 * want.norm()
