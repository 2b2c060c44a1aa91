"""The weight-streaming products of 1 to 16 rows: edges of their row groups, boxes of K, stages and batch blocks, against fp32."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu


def _check(got, want, k, what):
    # one rounding to bf16 of an fp32 sum (2^-9 of the value), plus the sum's own error: k products of 2^-24 each, relative to the rms
    err = (got.float() - want).abs()
    bound = want.abs() * 2.0 ** -8 + want.square().mean().sqrt() * (k ** 0.5 * 2.0 ** -20 + 1e-6)
    assert bool((err <= bound).all()), (what, float((err - bound).max()))


@pytest.fixture(params=[False, True], ids=["", "dependent"])
def dependent(request):
    before = _lib.set_dependent_launch(request.param)
    yield request.param
    _lib.set_dependent_launch(before)


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 7, 8, 9, 16])
@pytest.mark.parametrize("n, k", [(1, 8), (15, 64), (16, 72), (147, 512), (149, 520), (148 * 18 - 1, 1024), (148 * 32 + 1, 136),
                                  (4736, 640), (9000, 64), (40000, 16), (320, 9728)])
def test_product(rows, n, k, dependent):
    x, w = torch.randn(rows, k + 8, device="cuda").bfloat16()[:, :k], torch.randn(n, k + 16, device="cuda").bfloat16()[:, 8:k + 8]
    out = torch.full((rows, n + 3), 7.0, device="cuda").bfloat16()
    ops.gemm(x, w, out=out[:, :n])
    _check(out[:, :n], x.float() @ w.float().t(), k, (rows, n, k))
    assert bool((out[:, n:] == 7.0).all())
    _lib.check_status()


@pytest.mark.parametrize("rows", [1, 2, 4, 8, 13, 16])
@pytest.mark.parametrize("f, k", [(1, 8), (16, 64), (147, 200), (148 * 16, 512), (148 * 17 + 5, 128), (9728, 256)])
def test_product_with_swiglu(rows, f, k, dependent):
    x, w = torch.randn(rows, k, device="cuda").bfloat16(), (torch.randn(2 * f, k, device="cuda") * k ** -0.5).bfloat16()
    with torch.no_grad():
        got = ops.linear_swiglu(x, w).float()
    z = x.float() @ w.float().t()
    want = torch.nn.functional.silu(z[:, :f]) * z[:, f:]
    # gate and up are rounded to bf16 first: 2^-9 of each travels into the product, whose slopes are at most 1.1 |up| and |silu|
    bound = 2.0 ** -7 * (want.abs() + z[:, :f].abs() * z[:, f:].abs()) + 1e-4
    assert bool(((got - want).abs() <= bound).all()), float(((got - want).abs() - bound).max())
    _lib.check_status()


@pytest.mark.parametrize("rows", [1, 2, 3, 4])
@pytest.mark.parametrize("delta_rows", [None, 0, 1])
@pytest.mark.parametrize("n, k", [(6, 8), (296, 72), (148 * 21, 2560), (5000, 4096), (64, 12288)])
def test_norm_and_product(rows, delta_rows, n, k, dependent):
    x, w = torch.randn(rows, k, device="cuda").bfloat16(), (torch.randn(n, k, device="cuda") * k ** -0.5).bfloat16()
    nw = (1 + 0.1 * torch.randn(k, device="cuda")).bfloat16()
    d = None if delta_rows is None else torch.randn(rows - delta_rows, k, device="cuda").bfloat16()
    if d is not None and d.shape[0] == 0:
        pytest.skip("no rows")
    with torch.no_grad():
        res, got = ops.norm_linear(x, d, nw, 1e-6, w)
    want_res = x.clone()
    if d is not None:
        want_res[:d.shape[0]] += d
    assert torch.equal(res, want_res)
    h = want_res.float()
    h = (h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * nw.float()).bfloat16().float()
    want = h @ w.float().t()
    # a row's normalised values may round the other way (2^-8 of one of k terms each): their rms is k^-1/2 of the sum of squares
    err = (got.float() - want).abs()
    assert bool((err <= want.abs() * 2.0 ** -8 + 2.0 ** -7).all()), float(err.max())
    _lib.check_status()


def test_expanded_rows_and_large_norm_rows():
    w = torch.randn(300, 128, device="cuda").bfloat16()
    x = torch.randn(1, 128, device="cuda").bfloat16()
    assert torch.equal(ops.linear(x.expand(5, 128), w), ops.linear(x.repeat(5, 1), w))
    assert torch.equal(ops.linear(x.repeat(5, 1), w[:1].expand(40, 128)), ops.linear(x.repeat(5, 1), w[:1].repeat(40, 1)))


@pytest.mark.parametrize("rows, k", [(4, 20480), (4, 20488), (3, 40960), (1, 81920)])
def test_norm_and_product_of_long_rows(rows, k):
    """The most that a CTA keeps in shared memory, and more: then row by row."""
    x, d = torch.randn(rows, k, device="cuda").bfloat16(), torch.randn(rows - rows // 3, k, device="cuda").bfloat16()
    nw, w = torch.ones(k, device="cuda").bfloat16(), (torch.randn(64, k, device="cuda") * k ** -0.5).bfloat16()
    with torch.no_grad():
        res, y = ops.norm_linear(x, d, nw, 1e-6, w)
        one = [ops.norm_linear(x[i:i + 1], d[i:i + 1] if i < len(d) else None, nw, 1e-6, w) for i in range(rows)]
    assert torch.equal(res, torch.cat([r for r, _ in one])) and torch.equal(y, torch.cat([v for _, v in one]))
    want_res = x.clone()
    want_res[:len(d)] += d
    h = want_res.float()
    h = (h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6)).bfloat16().float()
    assert torch.equal(res, want_res) and float((y.float() - h @ w.float().t()).abs().max()) < 2.0 ** -5
    _lib.check_status()


@pytest.mark.parametrize("rows, delta_rows", [(1, None), (1, 1), (4, 3), (3, None)])
@pytest.mark.parametrize("glu", [False, True])
def test_rows_wider_than_any_norm_kernel(rows, delta_rows, glu):
    k = 81928
    x, nw = torch.randn(rows, k, device="cuda").bfloat16(), (1 + 0.1 * torch.randn(k, device="cuda")).bfloat16()
    d = None if delta_rows is None else torch.randn(delta_rows, k, device="cuda").bfloat16()
    w = (torch.randn(64, k, device="cuda") * k ** -0.5).bfloat16()
    with torch.no_grad():
        res, y = ops.norm_linear(x, d, nw, 1e-6, w, glu)
    want_res = x.clone()
    if d is not None:
        want_res[:delta_rows] += d
    h = want_res.float()
    want = (h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * nw.float()).bfloat16().float() @ w.float().t()
    if glu:
        gate, up = want.bfloat16().float().chunk(2, -1)
        want = torch.nn.functional.silu(gate) * up
    assert torch.equal(res, want_res)
    assert float((y.float() - want).norm()) <= 2.0 ** -6 * float(want.norm())      # a rounding of gate, up and result each, 2^-8
    _lib.check_status()


def test_norm_and_product_with_expanded_weights():
    """Long rows, so that no other way is open."""
    x, nw = torch.randn(2, 16384, device="cuda").bfloat16(), torch.ones(16384, device="cuda").bfloat16()
    w = torch.randn(1, 16384, device="cuda").bfloat16()
    with torch.no_grad():
        assert torch.equal(ops.norm_linear(x, None, nw, 1e-6, w.expand(40, -1))[1], ops.norm_linear(x, None, nw, 1e-6, w.repeat(40, 1))[1])
    _lib.check_status()


def test_operands_off_16_bytes_are_refused():
    w, x = torch.zeros(300 * 64 + 4, device="cuda").bfloat16(), torch.zeros(3, 64, device="cuda").bfloat16()
    with pytest.raises(RuntimeError, match="aligned"):
        ops.gemm(x, w[4:].view(300, 64))
