"""The TMA-store epilogue of the CTA-pair GEMM at the edges of its boxes, against fp32 matrix products."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"
# the one rounding to bf16 is at most 2^-8 of every element; sums are fp32
TOL = 4e-3


def bf(*shape, scale=1.0):
    return (torch.randn(*shape, device=DEV) * scale).bfloat16()


def rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm()).item()


@pytest.mark.parametrize("M,N,K", [(1000, 264, 72), (8256, 72, 200), (300, 4104, 64), (257, 520, 320)])
@pytest.mark.parametrize("fp32", [False, True])
def test_pair_gemm_stores_ragged_tiles(M, N, K, fp32):
    """Rows and columns that do not fill the 32-row, 128-byte boxes of the stores; a row pitch wider than the row."""
    a, b = bf(M, K), bf(N, K, scale=0.1)
    want = a.float() @ b.float().t()
    big = torch.full((M, N + 8), float("nan"), device=DEV, dtype=torch.float32 if fp32 else torch.bfloat16)
    out = big[:, :N]
    ops.gemm(a, b, out=out, pair=True)
    _lib.check_status()
    assert rel(out, want) < (1e-5 if fp32 else TOL) and bool(big[:, N:].isnan().all())
    if fp32:
        ops.gemm(a, b, out=out, accumulate=True, alpha=-0.5, pair=True)
        _lib.check_status()
        assert rel(out, 0.5 * want) < 1e-5 and bool(big[:, N:].isnan().all())
