"""GEMM with all rows in one tile: edges of row blocks and column tiles, remainders of K, gated and plain, and where it is taken."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu


def _check(c, x, w, glu):
    ref = x.double() @ w.double().t()
    # bf16 keeps 8 bits: rounding moves a value by at most 2^-8 of it; fp32 sums of K exact products by K * 2^-24 of the sum of magnitudes
    eps, slack = 2.0 ** -8, (x.double().abs() @ w.double().abs().t()) * x.shape[1] * 2.0 ** -24
    bound = ref.abs() * eps + slack
    if glu:
        F = w.shape[0] // 2
        g, u, dg, du = ref[:, :F], ref[:, F:], bound[:, :F], bound[:, F:]
        ref = torch.nn.functional.silu(g) * u
        # gate and up are rounded first: silu has a slope of at most 1.1 and is at most the gate; then the result is
        bound = 1.1 * dg * (u.abs() + du) + torch.nn.functional.silu(g).abs() * du + ref.abs() * eps
    assert ((c.double() - ref).abs() <= bound * 1.01 + 1e-6).all(), ((c.double() - ref).abs() - bound).max()


@pytest.mark.parametrize("M,N,K,glu,columns", [
    (17, 3552, 8, 1, 48), (24, 7104, 200, 0, 48), (127, 4664, 1032, 1, 64), (128, 16568, 64, 1, 224), (128, 14208, 72, 0, 96),
    (100, 47360, 136, 0, 160), (17, 70000, 264, 0, 160), (129, 3552, 136, 1, 48), (256, 11840, 520, 1, 160), (255, 7000, 72, 1, 96),
    (257, 10656, 64, 1, 144), (384, 11840, 520, 1, 160), (333, 9728, 320, 1, 144)])
def test_chosen_tile(M, N, K, glu, columns):
    torch.manual_seed(M)
    pitch = (K + 63) // 64 * 64
    x = torch.randn(M, pitch, device="cuda").bfloat16()[:, :K]
    w = (torch.randn((1 + glu) * N, pitch, device="cuda") * 0.1).bfloat16()[:, :K]
    assert _lib.gemm_tall_plan(M, N, K, glu, False) == columns
    with torch.no_grad():
        before = _lib.launch_count()
        c = ops.linear_swiglu(x, w) if glu else ops.gemm(x, w)
        assert _lib.launch_count() - before == 1
    _lib.check_status()
    _check(c, x, w, glu)
    wide = torch.full((M, N + 8), 7.0, device="cuda").bfloat16()
    _lib.call("ksa_gemm_tall_bf16", x, w, wide, M, N, K, pitch, pitch, N + 8, glu, columns)
    assert torch.equal(wide[:, :N], c) and (wide[:, N:] == 7).all(), "beside the result"


@pytest.mark.parametrize("M,N,K,glu", [
    (16, 9728, 2560, 1), (385, 9728, 2560, 1), (129, 12288, 2048, 0), (48, 2048, 2560, 0), (48, 9216, 4096, 0), (48, 14216, 2048, 0),
    (129, 14336, 4096, 1), (129, 1536, 2048, 1), (257, 6144, 2048, 1), (48, 35000, 1024, 0), (48, 12292, 2048, 0)])
def test_left_to_the_others(M, N, K, glu):
    assert _lib.gemm_tall_plan(M, N, K, glu, False) == 0 and _lib.gemm_tall_plan(48, 9728, 2560, 1, True) == 0


def test_rows_that_are_not_loaded_stay_out():
    """The rows behind the last that is loaded hold whatever the ring held, here infinities of the call before."""
    w = (torch.randn(12288, 512, device="cuda") * 0.1).bfloat16()
    ops.gemm(torch.full((128, 512), float("inf"), device="cuda").bfloat16(), torch.full_like(w, float("nan")))
    for M in (17, 33, 100, 130, 200):
        x = torch.randn(M, 512, device="cuda").bfloat16()
        with torch.no_grad():
            _check(ops.linear_swiglu(x, w), x, w, 1)
    _lib.check_status()


@pytest.mark.parametrize("columns,M,N,ldc,match", [(0, 48, 128, 128, "columns"), (24, 48, 128, 128, "columns"), (272, 48, 128, 128, "columns"),
                                                   (176, 300, 128, 128, "columns"), (48, 385, 128, 128, "rows"), (48, 48, 132, 136, "C"),
                                                   (48, 48, 128, 132, "C")])
def test_rejects(columns, M, N, ldc, match):
    x, w = [torch.zeros(400, 64, device="cuda").bfloat16() for _ in range(2)]
    c = torch.zeros(400 * 136, device="cuda").bfloat16()
    with pytest.raises(RuntimeError, match="gemm_tall.*" + match):
        _lib.call("ksa_gemm_tall_bf16", x, w, c, M, N, 64, 64, 64, ldc, 0, columns)
