"""GEMM on CTA pairs: a last wave of few tiles is worked on as halves of 128 columns."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles_m,tiles_n,M,N,K", [
    (1, 1, 256, 256, 64), (1, 1, 40, 136, 200), (1, 1, 256, 120, 72), (37, 1, 37 * 256 - 9, 248, 136), (38, 1, 38 * 256, 256, 128),
    (25, 3, 25 * 256 - 130, 520, 136), (25, 3, 6400, 768, 1024), (37, 3, 37 * 256, 768, 72), (16, 7, 4096, 1664, 264), (19, 4, 4864, 1024, 64)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_last_wave(tiles_m, tiles_n, M, N, K, a_mn, b_mn):
    torch.manual_seed(M + N)
    assert -(-M // 256) == tiles_m and -(-N // 256) == tiles_n
    M = (M + 7) // 8 * 8
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = (torch.randn(N, K, device="cuda") * 0.1).bfloat16()
    ref, mags = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    x, w = a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b
    c = ops.gemm(x, w, a_mn_major=a_mn, b_mn_major=b_mn, pair=True)
    base = torch.randn(M, N, device="cuda")
    f = base.clone()
    ops.gemm(x, w, a_mn_major=a_mn, b_mn_major=b_mn, out=f, accumulate=True, pair=True)
    wide = torch.full((M, N + 8), 7.0, device="cuda").bfloat16()
    ops.gemm(x, w, a_mn_major=a_mn, b_mn_major=b_mn, out=wide[:, :N], pair=True)
    _lib.check_status()
    slack = mags * K * 2.0 ** -24                      # fp32 sums of exact products, then one rounding
    assert ((c.double() - ref).abs() <= ref.abs() * 2.0 ** -8 * 1.01 + slack + 1e-6).all()
    assert ((f.double() - base.double() - ref).abs() <= slack + (base.double().abs() + ref.abs()) * 2.0 ** -23 + 1e-6).all()
    assert torch.equal(wide[:, :N], c) and (wide[:, N:] == 7).all(), "beside the result"
