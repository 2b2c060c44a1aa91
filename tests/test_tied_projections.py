"""Text rows and summary rows that share one weight, or whose weights' gradients share memory: the summary rows' gradient adds to what the
text rows' has written, so it may not run beside it."""
import types

import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

D, N = 64, 96


def _weights(kind, device):
    """(w_a, w_b, their gradient buffers) with one weight, two of one buffer, two of buffers that overlap, and two apart."""
    def weight():
        return (torch.randn(N, D, device=device) * 0.05).bfloat16().requires_grad_()
    wa = weight()
    wb = wa if kind == "tied" else weight()
    pool = torch.zeros(3 * N, D, device=device)
    at = {"tied": 0, "one buffer": 0, "overlapping": N - 1, "neighbours": N, "apart": 2 * N}[kind]
    wa.main_grad = pool[:N]
    wb.main_grad = pool[at:at + N]
    return wa, wb, pool


KINDS = ["tied", "one buffer", "overlapping", "neighbours", "apart"]


@pytest.mark.parametrize("n_a", [16, 17, 40])
@pytest.mark.parametrize("kind", KINDS)
def test_who_runs_beside(kind, n_a, monkeypatch):
    torch.manual_seed(0)
    wa, wb, _ = _weights(kind, "cpu")
    asked = []

    class Calls:
        @staticmethod
        def dual_linear(x, w_a, w_b, n, *_):
            return torch.empty(x.shape[0], D)

        @staticmethod
        def linear_dw(dy, x, lo, hi, out, acc, pair_min, beside):
            asked.append((lo, beside))
            return out
    monkeypatch.setattr(ops, "_native", Calls)
    R = n_a + 5
    ctx = types.SimpleNamespace(saved_tensors=(torch.randn(R, D), wa, wb), n_a=n_a, needs_input_grad=(True, True, True, False))
    ops._DualLinearFn.backward(ctx, torch.randn(R, N))
    assert asked == [(0, 0), (n_a, int(n_a > 16 and kind in ("neighbours", "apart")))]


def test_shared_memory():
    t = torch.zeros(8, 8)
    assert ops._share_memory(t, t) and ops._share_memory(t[:4], t[3:]) and not ops._share_memory(t[:4], t[4:])
    assert ops._share_memory(t[:, :4], t[:, 4:])              # rows that interleave
    assert not ops._share_memory(t, None) and not ops._share_memory(t[:0], t) and not ops._share_memory(t, torch.zeros(8, 8))


@pytest.mark.gpu
@pytest.mark.parametrize("n_a,n_b", [(17, 3), (333, 2), (2100, 300)])
@pytest.mark.parametrize("kind", ["tied", "one buffer", "apart"])
def test_gradients(kind, n_a, n_b):
    """Several calls that accumulate, bit for bit what ordinary launches give."""
    def run():
        torch.manual_seed(n_a)
        wa, wb, pool = _weights(kind, "cuda")
        for _ in range(4):
            x = torch.randn(n_a + n_b, D, device="cuda").bfloat16().requires_grad_()
            ops.dual_linear(x, wa, wb, n_a).backward(torch.randn(n_a + n_b, N, device="cuda").bfloat16())
            if kind == "one buffer":
                wa._grad_written = wb._grad_written = True
        return pool
    before = _lib.set_dependent_launch(_lib.ORDINARY)
    try:
        want = run()
    finally:
        _lib.set_dependent_launch(before)
        torch.cuda.synchronize()
    assert float(want.abs().sum()) > 0
    for _ in range(3):
        assert torch.equal(run(), want)
