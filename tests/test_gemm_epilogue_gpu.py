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


# rows x columns with several tiles for every CTA pair and a last column tile that ends after 1, 2, 3, 7 pieces of 32 fp32 columns
# or 1, 3, 4 pieces of 64 bf16 columns: the next tile's stores follow on either staging buffer
@pytest.mark.parametrize("M,N", [(38400, 264), (8256, 2112), (16640, 2144), (8256, 2240), (8256, 2272), (9000, 2880),
                                 (8256, 4104)])
@pytest.mark.parametrize("K", [64, 128])
def test_pair_gemm_staging_across_tiles(M, N, K):
    """Short reductions, so that nothing but the staging buffers orders the stores of consecutive tiles."""
    torch.manual_seed(N)
    a, b = bf(M, K), bf(N, K, scale=0.1)
    want = (a.double() @ b.double().t()).float()
    # fp32 sums of K products of bf16 values in any order
    bound = (K * 2.0 ** -23) * (a.float().abs() @ b.float().abs().t())
    init = torch.randn(M, N, device=DEV)
    for _ in range(3):
        c = torch.full((M, N), float("nan"), device=DEV, dtype=torch.bfloat16)
        ops.gemm(a, b, out=c, pair=True)
        assert bool(((c.float() - want).abs() <= 2.0 ** -8 * want.abs() + bound).all())
        c = torch.full((M, N), float("nan"), device=DEV)
        ops.gemm(a, b, out=c, pair=True)
        assert bool(((c - want).abs() <= bound).all())
        c = init.clone()
        ops.gemm(a, b, out=c, accumulate=True, pair=True)
        assert bool(((c - (init + want)).abs() <= bound + 2.0 ** -22 * (init.abs() + want.abs())).all())
    _lib.check_status()
