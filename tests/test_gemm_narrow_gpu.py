"""The split-K GEMM for few activation rows against fp64: edges of its tiles, every split, both weight layouts, the gated form."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu

# one rounding of the result to bf16 (2^-9 relative to each value, in the 2-norm at most 2^-9) and fp32 sums of K products,
# whose error is far below it
REL = 2.0 ** -9 + 1e-5


def _check(c, x, w, glu=False):
    assert torch.isfinite(c).all()
    r = x.double() @ w.double().t()
    rel = REL
    if glu:
        # gate and up are rounded before the activation; a rounding the other way moves the product by up to 2^-8 each
        g, u = r.bfloat16().double().chunk(2, -1)
        r, rel = torch.nn.functional.silu(g) * u, 3 * REL
    assert ((c.double() - r).norm() / r.norm()).item() < rel


@pytest.mark.parametrize("glu", [False, True])
@pytest.mark.parametrize("M,N,K,bt,split", [
    (17, 128, 64, 32, 1), (15, 16, 8, 16, 1), (100, 272, 200, 64, 2), (129, 1040, 1000, 48, 4), (333, 512, 4096, 176, 8),
    (257, 144, 520, 256, 8), (1, 2576, 136, 16, 2), (64, 4096, 2048, 64, 2)])
def test_given_plan(M, N, K, bt, split, glu):
    torch.manual_seed(M + N)
    x = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.1).bfloat16()
    n_out = N // 2 if glu else N
    buf = torch.full((M + 2, n_out + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    c = buf[1:M + 1, :n_out]
    for w_mn in ([0] if glu else [0, 1]):
        ws = w.t().contiguous() if w_mn else w
        buf.fill_(7.0)
        _lib.call("ksa_gemm_narrow_bf16", x, ws, c, M, N, K, K, ws.stride(0), c.stride(0), w_mn, int(glu), bt, split, 1.0)
        _lib.check_status()
        _check(c, x, w, glu)
        assert (buf[0] == 7).all() and (buf[-1] == 7).all() and (buf[:, n_out:] == 7).all(), "wrote outside C"


@pytest.mark.parametrize("M,N,K", [(17, 2560, 9728), (48, 6144, 2560), (128, 4096, 1032), (129, 2048, 2048), (700, 2560, 4096),
                                   (1793, 256, 2048), (1700, 1000, 6144)])
def test_chosen_plan(M, N, K):
    torch.manual_seed(M)
    x = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.1).bfloat16()
    assert _lib.gemm_narrow_plan(M, N, K, 0, ops.GEMM_PAIR_MIN_TILES) is not None
    _check(ops.gemm(x, w), x, w)
    _check(ops.gemm(x, w.t().contiguous(), b_mn_major=True, alpha=-0.5), -0.5 * x, w)
    if N % 16 == 0:
        with torch.no_grad():
            h = ops.linear_swiglu(x, w)
        _check(h, x, w, glu=True)
    assert torch.equal(ops.gemm(x, w), ops.gemm(x, w)), "the parts are added in a fixed order"
    _lib.check_status()


def test_plans_are_valid():
    """Every plan is one that the kernel takes, and tiny products stay with the tiled kernels."""
    n = 0
    for M in (1, 16, 17, 100, 129, 257, 333, 1000, 4097, 20000):
        for N in (8, 64, 264, 2560, 19456, 151936):
            for K in (8, 64, 200, 520, 2048, 9728):
                for glu in (0, 1):
                    plan = _lib.gemm_narrow_plan(M, N, K, glu, 32)
                    if plan is not None:
                        n += 1
                        assert plan[0] % 16 == 0 and 16 <= plan[0] <= 256
                        assert plan[1] in (1, 2, 4, 8) and plan[1] <= (K + 63) // 64
    assert n > 100 and _lib.gemm_narrow_plan(48, 64, 64, 0, 32) is None


def test_rejects_bad_plans():
    x = torch.zeros(32, 64, device="cuda", dtype=torch.bfloat16)
    w = torch.zeros(128, 64, device="cuda", dtype=torch.bfloat16)
    c = torch.empty(32, 128, device="cuda", dtype=torch.bfloat16)
    for bt, split in ((24, 1), (272, 1), (0, 1), (32, 3), (32, 2)):       # K = 64 cannot be split
        with pytest.raises(RuntimeError, match="gemm_narrow"):
            _lib.call("ksa_gemm_narrow_bf16", x, w, c, 32, 128, 64, 64, 64, 128, 0, 0, bt, split, 1.0)


@pytest.mark.parametrize("M,N,K,ragged,slow", [
    (779, 3552, 6008, 3, (160, 2)), (126, 14456, 7384, 3, (128, 2)), (151, 10896, 4760, 3, (160, 2)),
    (522, 15440, 7544, 3, (144, 1)), (1041, 7624, 7984, 3, (160, 1)), (193, 4256, 3352, 3, (208, 4)),
    (1397, 584, 4032, 0, (208, 4)), (1465, 720, 6200, 3, (256, 4))])
def test_plans_that_were_slower_than_tiles(M, N, K, ragged, slow):
    """Rows off the 128-byte lines, and clusters of four that do not fit all at once: measured 12 to 45 % slower than tiles."""
    assert _lib.gemm_narrow_plan(M, N, K, 0, 32, ragged) != slow
    if ragged == 3:
        x = torch.randn(M, K, device="cuda").bfloat16()
        w = (torch.randn(N, K, device="cuda") * 0.1).bfloat16()
        _check(ops.gemm(x, w), x, w)
        _lib.check_status()


@pytest.mark.parametrize("M,N,K,fused", [(48, 19456, 2560, True), (333, 1040, 1032, True), (129, 272, 2048, True),
                                         (48, 272, 64, False), (2047, 12288, 2048, False), (2049, 256, 2048, False)])
def test_linear_swiglu_takes_the_gated_kernel(M, N, K, fused):
    """One launch where there is a plan for the gated form, the projection and the activation where there is none (too little
    or too much work, too many rows)."""
    torch.manual_seed(M)
    x = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.1).bfloat16()
    plan = _lib.gemm_narrow_plan(M, N, K, 1, ops.GEMM_PAIR_MIN_TILES, 3 * (K % 64 != 0))
    assert (plan is not None) == fused
    with torch.no_grad():
        before = _lib.launch_count()
        h = ops.linear_swiglu(x, w)
        assert _lib.launch_count() - before == (1 if fused else 2)
    _lib.check_status()
    _check(h, x, w, glu=True)


@pytest.mark.parametrize("N,ldc,w_mn,glu,offset", [(132, 136, 0, 0, 0), (128, 132, 0, 0, 0), (136, 136, 0, 1, 0),
                                                   (128, 128, 1, 1, 0), (128, 128, 0, 0, 4)])
def test_rejects_bad_outputs_and_layouts(N, ldc, w_mn, glu, offset):
    """Rows of C off 16 bytes, feature counts the gated form does not pair, gated weights in the other layout."""
    x = torch.zeros(32, 64, device="cuda", dtype=torch.bfloat16)
    w = torch.zeros(144, 144, device="cuda", dtype=torch.bfloat16)
    c = torch.empty(32 * 144 + 8, device="cuda", dtype=torch.bfloat16)[offset:]
    with pytest.raises(RuntimeError, match="gemm_narrow"):
        _lib.call("ksa_gemm_narrow_bf16", x, w, c, 32, N, 64, 64, 144, ldc, w_mn, glu, 32, 1, 1.0)
