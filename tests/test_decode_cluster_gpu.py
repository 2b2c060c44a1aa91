"""Decode attention on clusters: slices that leave splits, warps or whole groups without keys, and both sides of the rule."""
import pytest
import torch

from ksa_b200.inference.engine import _decode_attention
from ksa_b200.ops import _lib, reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [40, 1200, 2048, 2049])       # the last by the splits of a grid
@pytest.mark.parametrize("B,Tq,Hq,Hkv", [(1, 1, 1, 1), (4, 1, 32, 8), (5, 1, 32, 8), (3, 2, 8, 2), (2, 4, 8, 2), (2, 3, 10, 2)])
def test_slices(B, Tq, Hq, Hkv, cap):
    torch.manual_seed(cap + B)
    D = 128
    k, v = [torch.randn(B, Hkv, cap, D, device="cuda").bfloat16() for _ in range(2)]
    q = torch.randn(B, Tq, Hq, D, device="cuda").bfloat16()
    counters = torch.zeros(B * Hkv, dtype=torch.int32, device="cuda")
    for n in (0, 1, 15, 16, 17, 95, 96, 97, 128, 129, 769, cap):
        if n > cap:
            continue
        # other queries and sequences have other slices, up to none at all
        length = torch.clamp(n - torch.arange(B * Tq, device="cuda").view(B, Tq) * 5, min=0).int()
        start = torch.randint(0, cap - n + 1, (B, Tq), device="cuda").int()
        got = _decode_attention(q, k, v, start, length, D ** -0.5, counters)
        for b in range(B):
            for t in range(Tq):
                if length[b, t] == 0:
                    assert (got[b, t] == 0).all()
                    continue
                want = ref.decode_attention(q[b:b + 1, t:t + 1].float(), k[b:b + 1].float(), v[b:b + 1].float(),
                                            length[b:b + 1, t].long(), start[b:b + 1, t].long(), D ** -0.5)
                # fp32 sums, the result rounded to bf16
                assert ((got[b, t].float() - want[0, 0]).norm() / want.norm()).item() < 4e-3
        assert torch.equal(got, _decode_attention(q, k, v, start, length, D ** -0.5, counters))
    assert (counters == 0).all()
    _lib.check_status()


@pytest.mark.parametrize("cap", [40, 1200, 2049])
@pytest.mark.parametrize("D", [64, 128])
def test_slices_end_with_the_cache(D, cap):
    """A slice that a device value makes too long, or start too early, is cut: nothing outside the cache is read."""
    torch.manual_seed(cap)
    B, Hq, Hkv = 2, 8, 2
    k, v = [torch.randn(B, Hkv, cap, D, device="cuda").bfloat16() for _ in range(2)]
    q = torch.randn(B, 1, Hq, D, device="cuda").bfloat16()
    at = lambda *x: torch.tensor(x, device="cuda").view(B, 1).int()
    want = _decode_attention(q, k, v, at(0, cap - 10), at(cap, 10), D ** -0.5)
    for far in (17, 100000, 2 ** 31 - 1 - cap):
        assert torch.equal(want, _decode_attention(q, k, v, at(0, cap - 10), at(cap + far, 10 + far), D ** -0.5))
    assert torch.equal(want, _decode_attention(q, k, v, at(-50, cap - 10), at(cap + 50, 10), D ** -0.5))
    _lib.check_status()


@pytest.mark.parametrize("cap", [1536, 1537])                 # by clusters and by the splits of a grid
def test_more_blocks_than_multiprocessors(cap):
    test_slices(4, 1, 32, 8, cap)
    test_slices(3, 1, 64, 8, cap)                              # eight queries a group: clusters either way
