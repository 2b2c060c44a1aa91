"""Gate/up projection with the activation in the epilogue of the CTA-pair GEMM: the bits of the separate kernels, edges of its tiles."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M, F, K", [(1, 64, 8), (31, 64, 72), (255, 128, 64), (256, 192, 128), (257, 320, 200), (600, 1088, 320), (3000, 640, 64)])
def test_bits_of_the_separate_kernels(M, F, K):
    x, w = torch.randn(M, K + 8, device="cuda").bfloat16()[:, :K], (torch.randn(2 * F, K, device="cuda") * K ** -0.5).bfloat16()
    h, gu = torch.full((M + 1, F + 8), 7.0, device="cuda").bfloat16(), torch.full((M + 1, 2 * F + 8), 7.0, device="cuda").bfloat16()
    _lib.call("ksa_gemm2_swiglu_bf16", x, w, gu, h, M, F, K, x.stride(0), w.stride(0), gu.stride(0), h.stride(0))
    _lib.check_status()
    want_gu = ops.gemm(x, w, pair=True)
    want = ops.swiglu(want_gu)
    assert torch.equal(h[:M, :F], want) and bool((h[M] == 7).all()) and bool((h[:, F:] == 7).all())
    assert bool((gu[M] == 7).all()) and bool((gu[:, 2 * F:] == 7).all())
    assert torch.equal(gu[:M, :2 * F], want_gu)


def test_features_off_64_are_refused():
    x, w, h = (torch.zeros(*s, device="cuda").bfloat16() for s in ((64, 64), (192, 64), (64, 96)))
    with pytest.raises(RuntimeError, match="multiple of 64"):
        _lib.call("ksa_gemm2_swiglu_bf16", x, w, torch.zeros(64, 192, device="cuda").bfloat16(), h, 64, 96, 64, 64, 64, 192, 96)


@pytest.mark.parametrize("rows, fused", [(20, 2), (300, None), (2000, 1), (4100, 1)])
@pytest.mark.parametrize("main_grad", [False, True])
def test_the_operator(rows, fused, main_grad):
    """The same values and gradients as the projection followed by the activation; one launch where the pair kernel takes it."""
    F, K = 1024, 512
    x = torch.randn(rows, K, device="cuda").bfloat16().requires_grad_()
    w = torch.nn.Parameter((torch.randn(2 * F, K, device="cuda") * K ** -0.5).bfloat16())
    g = torch.randn(rows, F, device="cuda").bfloat16()
    results = []
    for call in (lambda: ops.linear_swiglu(x, w), lambda: ops.swiglu(ops.linear(x, w))):
        if main_grad:
            w.main_grad, w._grad_written = torch.zeros(w.shape, dtype=torch.float32, device="cuda"), False
        x.grad = w.grad = None
        before = _lib.launch_count()
        y = call()
        launches = _lib.launch_count() - before
        y.backward(g)
        results.append([y.detach(), x.grad, w.main_grad if main_grad else w.grad])
        if fused is not None and len(results) == 1:
            assert launches == fused
    assert all(torch.equal(a, b) for a, b in zip(*results))
    with torch.no_grad():
        assert (ops.linear_swiglu(x, w).float() - results[0][0].float()).abs().max() < 0.1
    _lib.check_status()


@pytest.mark.parametrize("rows, F, launches", [(333, 6144, 2), (640, 6144, 1), (336, 9728, 2)])
def test_the_fused_form_goes_by_the_rule_for_pairs(rows, F, launches):
    """Where single CTAs take fewer waves, they and a separate activation are faster than the activation on pairs."""
    x, w = torch.randn(rows, 512, device="cuda").bfloat16(), torch.randn(2 * F, 512, device="cuda").bfloat16().requires_grad_()
    assert _lib.count_launches(lambda: ops.linear_swiglu(x, w)) == launches
    assert _lib.gemm_on_pairs(rows, 2 * F, ops.GEMM_PAIR_MIN_TILES) == (launches == 1)
    _lib.check_status()
