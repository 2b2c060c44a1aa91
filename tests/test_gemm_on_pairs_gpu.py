"""Products on CTA pairs or on single CTAs, by the waves that each would take: the same bits from both, in every form of the operands."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu
TILES = ops.GEMM_PAIR_MIN_TILES


def test_the_rule():
    def pairs(M, N):
        return _lib.gemm_on_pairs(M, N, 32)

    assert not pairs(333, 19456) and not pairs(600, 7168)                   # 3 waves against 2, 2 against 1
    assert pairs(256, 4096 * 2) and pairs(8192, 6144) and pairs(512, 9472)   # one wave each, many waves, a full wave of 74
    assert not pairs(256, 7936) and not _lib.gemm_on_pairs(8192, 6144, 0)      # 31 tiles; the switch


@pytest.mark.parametrize("a_mn, b_mn, fp32", [(0, 0, 0), (0, 1, 0), (1, 1, 0), (0, 0, 1), (1, 1, 1)])
@pytest.mark.parametrize("M, N, K", [(336, 19456, 136), (264, 12544, 64), (600, 7168, 1000), (384, 9736, 328)])
def test_same_bits_as_on_pairs(M, N, K, a_mn, b_mn, fp32):
    assert (M + 255) // 256 * ((N + 255) // 256) >= TILES and not _lib.gemm_on_pairs(M, N, TILES)
    a = torch.randn(*((K, M + 8) if a_mn else (M, K + 8)), device="cuda").bfloat16()[:, :-8]      # rows of a wider buffer
    b = torch.randn(*((K, N) if b_mn else (N, K)), device="cuda").bfloat16()
    kw = dict(a_mn_major=bool(a_mn), b_mn_major=bool(b_mn), accumulate=bool(fp32))
    outs = [torch.ones(M, N, device="cuda", dtype=torch.float32 if fp32 else torch.bfloat16) for _ in range(3)]
    for out, pair in zip(outs, (True, False, None)):
        ops.gemm(a, b, out=out, pair=pair, **kw)
    assert torch.equal(outs[0], outs[1])
    A, B = (a.t() if a_mn else a).double(), (b if b_mn else b.t()).double()
    want, size = A @ B + (1 if fp32 else 0), A.abs() @ B.abs() + 1
    # fp32 sums of K products (2^-22 of their sizes for sums in the tensor core, K / 16 of them) and one rounding of the result
    for got in outs[1:]:
        bound = size * (K / 16 + 2) * 2.0 ** -22 + (0 if fp32 else want.abs() * 2.0 ** -8)
        assert bool(((got.double() - want).abs() <= bound).all())
    _lib.check_status()
