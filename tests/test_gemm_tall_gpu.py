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


@pytest.mark.parametrize("M,N,K,glu,columns,split", [
    (17, 3552, 8, 1, 48, 1), (127, 4664, 1032, 1, 64, 1), (128, 16568, 64, 1, 224, 1), (129, 3552, 136, 1, 48, 1), (256, 11840, 520, 1, 160, 1),
    (255, 7000, 72, 1, 96, 1), (257, 10656, 64, 1, 144, 1), (384, 11840, 520, 1, 160, 1), (333, 9728, 320, 1, 144, 1),
    (24, 128, 64, 0, 16, 1), (100, 47360, 136, 0, 160, 1), (17, 70000, 264, 0, 160, 1), (128, 14208, 72, 0, 96, 1), (256, 11840, 520, 0, 80, 1),
    (17, 2576, 9736, 0, 80, 4), (48, 1528, 8960, 0, 112, 8), (130, 2560, 3080, 0, 80, 4), (255, 4096, 2056, 0, 64, 2), (129, 7104, 2560, 0, 96, 2),
    (256, 264, 4104, 0, 32, 8), (257, 1024, 3072, 0, 32, 4), (384, 3696, 6152, 0, 112, 4), (383, 136, 2568, 0, 16, 8)])
def test_chosen_tile(M, N, K, glu, columns, split):
    torch.manual_seed(M)
    pitch = (K + 63) // 64 * 64
    x = torch.randn(M, pitch, device="cuda").bfloat16()[:, :K]
    w = (torch.randn((1 + glu) * N, pitch, device="cuda") * 0.1).bfloat16()[:, :K]
    assert _lib.gemm_tall_plan(M, N, K, glu, False) == (columns, split)
    with torch.no_grad():
        before = _lib.launch_count()
        c = ops.linear_swiglu(x, w) if glu else ops.gemm(x, w)
        assert _lib.launch_count() - before == 1
    _lib.check_status()
    _check(c, x, w, glu)
    wide = torch.full((M, N + 8), 7.0, device="cuda").bfloat16()
    _lib.call("ksa_gemm_tall_bf16", x, w, wide, M, N, K, pitch, pitch, N + 8, glu, columns, split)
    assert torch.equal(wide[:, :N], c) and (wide[:, N:] == 7).all(), "beside the result, and the same each time"


@pytest.mark.parametrize("M,N,K,glu", [
    (16, 9728, 2560, 1), (385, 9728, 2560, 1), (129, 12288, 2048, 0), (48, 120, 2560, 0), (385, 1024, 2560, 0), (48, 14216, 2048, 0),
    (129, 14336, 4096, 1), (129, 1536, 2048, 1), (257, 6144, 2048, 1), (48, 35000, 1024, 0), (48, 12292, 2048, 0), (48, 4608, 4096, 1),
    (257, 2560, 4096, 0), (257, 4096, 12288, 0)])
def test_left_to_the_others(M, N, K, glu):
    assert _lib.gemm_tall_plan(M, N, K, glu, False) is None and _lib.gemm_tall_plan(48, 9728, 2560, 1, True) is None


def test_plans_are_valid():
    """Every plan is one that the kernel takes, and splits only what is long enough."""
    for M in range(17, 385, 11):
        for N in (128, 136, 1000, 2560, 4096, 6152, 11840, 14208, 151936):
            for K in (8, 72, 200, 1032, 4096, 20000):
                plan = _lib.gemm_tall_plan(M, N, K, 0, False)
                if plan is not None:
                    columns, split = plan
                    assert 16 <= columns <= (256 if M <= 256 else 160) and columns % 16 == 0
                    assert split in (1, 2, 4, 8) and split <= (K + 63) // 64
                    assert split * -(-(columns // 8) // split) * (M + 7) // 8 * 8 * 32 <= 222 * 1024 or split == 1


def test_parts_on_two_streams():
    """Clusters of two products at once: a block that waits for its cluster never holds what the other's blocks wait for."""
    x = torch.randn(48, 2560, device="cuda").bfloat16()
    w = (torch.randn(2560, 2560, device="cuda") * 0.1).bfloat16()
    want = ops.gemm(x, w)
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    got = []
    for _ in range(20):
        for s in streams:
            with torch.cuda.stream(s):
                got.append(ops.gemm(x, w))
    torch.cuda.synchronize()
    _lib.check_status()
    assert all(torch.equal(g, want) for g in got)


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
        _lib.call("ksa_gemm_tall_bf16", x, w, c, M, N, 64, 64, 64, ldc, 0, columns, 1)


@pytest.mark.parametrize("M,columns,split,glu", [(48, 48, 2, 1), (48, 48, 2, 0), (48, 48, 9, 0), (48, 48, 0, 0), (384, 160, 2, 0)])
def test_rejects_splits(M, columns, split, glu):
    """SwiGLU and K = 64 in parts, more than eight, more than shared memory holds."""
    K = 640 if glu or M > 48 else 64
    x, w, c = [torch.zeros(400, 640, device="cuda").bfloat16() for _ in range(3)]
    with pytest.raises(RuntimeError, match="gemm_tall.*parts"):
        _lib.call("ksa_gemm_tall_bf16", x, w, c, M, 128, K, 640, 640, 640, glu, columns, split)
