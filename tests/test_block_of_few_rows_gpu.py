"""The second product of a feed-forward block reads its weights while the first is at work: weights that a kernel writes just before the block."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.models.qwen3_ksa import SwiGluMlp
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 4, 5, 8, 9, 16, 17])
def test_weights_written_just_before(rows):
    torch.manual_seed(rows)
    D, F = 512, 2048
    mlp = SwiGluMlp(D, F).cuda().bfloat16()
    norm = torch.ones(D, device="cuda").bfloat16()
    x, delta = [torch.randn(rows, D, device="cuda").bfloat16() for _ in range(2)]
    a = [(torch.randn(D, 1024, device="cuda") * 0.03).bfloat16() for _ in range(4)]
    b = [(torch.randn(F, 1024, device="cuda") * 0.03).bfloat16() for _ in range(4)]
    g = [(torch.randn(2 * F, D, device="cuda") * 0.03).bfloat16() for _ in range(4)]

    def chain():
        got = []
        with torch.no_grad():
            for p, q, w in zip(a, b, g):
                mlp.w13.weight.copy_(w)
                ops.gemm(p, q, out=mlp.w2.weight.data)        # a product that lets its successors start early
                res, y = mlp.forward_after_norm(x, delta, norm, 1e-6)
                got += [res, y, ops.linear(y, mlp.w2.weight.t().contiguous())]
        return got
    got = [chain() for _ in range(3)]
    before = _lib.set_dependent_launch(_lib.ORDINARY)
    try:
        want = chain()
    finally:
        _lib.set_dependent_launch(before)
    for c in got:
        for u, v in zip(c, want):       # one or two rows take the ring here and a warp per weight row in ordinary launches: the order of fp32 sums
            assert ((u.float() - v.float()).norm() / v.float().norm()).item() < (4e-3 if rows <= 2 else 1e-9)
    _lib.check_status()
