"""Summary-query attention with every number of queries per group that has a kernel of its own, against the fp32 formulas."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,S", [(2, 2, 1), (4, 2, 1), (6, 2, 1), (8, 2, 1), (8, 2, 2)])
@pytest.mark.parametrize("L", [256, 300])
def test_queries_per_group(Hq, Hkv, S, L):
    torch.manual_seed(Hq * S)
    C, W, D = 128, 2, 128
    Ns = (L + C - 1) // C * S
    t = [torch.randn(1, T, H, D, device="cuda").bfloat16()
         for T, H in ((L, Hq), (L, Hkv), (L, Hkv), (Ns, Hq), (Ns, Hkv), (Ns, Hkv))]
    xs, fs = [x.clone().requires_grad_() for x in t], [x.float().requires_grad_() for x in t]
    got, want = ops.ksa_attention(*xs, C, S, W), ref.ksa_attention(*fs, C, S, W)
    g = [torch.randn(o.shape, device="cuda").bfloat16() for o in got]
    torch.autograd.backward(list(got), g)
    torch.autograd.backward(list(want), [x.float() for x in g])
    # bf16 results (2^-9), and in the backward pass probabilities and their gradients rounded to bf16 before each product
    for a, b, tol in [*zip(got, want, (1e-2, 1e-2)), *[(x.grad, f.grad, 2e-2) for x, f in zip(xs, fs)]]:
        assert torch.isfinite(a).all() and ((a.float() - b).norm() / b.norm()).item() < tol
