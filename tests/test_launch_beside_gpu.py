"""Text rows and summary rows of one call run beside one another: in chains whose inputs come from the kernel before and whose results go to the
kernel after, everything is what ordinary launches give."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu


def _ordinary(fn):
    before = _lib.set_dependent_launch(_lib.ORDINARY)
    try:
        return fn()
    finally:
        _lib.set_dependent_launch(before)
        torch.cuda.synchronize()


def _same(a, b):
    return all(torch.equal(x, y) for x, y in zip(a, b))


# summary rows: one and two (a warp per weight row), up to sixteen (the ring), split K, tiles; text rows: the last that must not go beside, few, many
@pytest.mark.parametrize("n_b", [1, 2, 3, 16, 40, 300])
@pytest.mark.parametrize("n_a", [16, 17, 333, 2100])
def test_projections(n_a, n_b):
    torch.manual_seed(n_a + n_b)
    D, N, R = 512, 1024, n_a + n_b
    wa, wb = [(torch.randn(N, D, device="cuda") * 0.05).bfloat16().requires_grad_() for _ in range(2)]
    for w in (wa, wb):
        w.main_grad = torch.zeros(N, D, device="cuda")
    norm = torch.ones(D, device="cuda").bfloat16()
    inputs = [torch.randn(R, D, device="cuda").bfloat16() for _ in range(4)]
    dy = [torch.randn(R, N, device="cuda").bfloat16() for _ in range(4)]

    def chain():
        got = []
        for w in (wa, wb):
            w._grad_written = False
        for x, g in zip(inputs, dy):            # the second to fourth accumulate into the weights' gradients
            x = x.detach().requires_grad_()
            y = ops.dual_linear(ops.rms_norm(x, norm), wa, wb, n_a)
            (y * 1).backward(g)
            got += [ops.swiglu(y.detach()), x.grad]
        return got + [w.main_grad.clone() for w in (wa, wb)]
    want = _ordinary(chain)
    for _ in range(3):
        assert _same(chain(), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        held = chain()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert _same(held, want)


@pytest.mark.parametrize("B,L,Hq,Hkv", [(1, 130, 8, 2), (1, 333, 8, 2), (2, 700, 4, 2), (1, 5000, 8, 4)])
def test_attention(B, L, Hq, Hkv):
    torch.manual_seed(L)
    D, C, Ns = 128, 128, L // 128
    R = B * (L + Ns)
    width = (Hq + 2 * Hkv) * D
    x = [torch.randn(R, width, device="cuda").bfloat16() for _ in range(4)]
    w = (torch.randn(256, Hq * D, device="cuda") * 0.05).bfloat16()
    norm = torch.ones(width, device="cuda").bfloat16()

    def chain():
        got = []
        with torch.no_grad():
            for t in x:
                o = ops.attention_packed(ops.rms_norm(t, norm), B, L, Ns, Hq, Hkv, D, C, 1, 2)
                got += [ops.linear(o, w), o]
        return got
    want = _ordinary(chain)
    for _ in range(3):
        assert _same(chain(), want)
