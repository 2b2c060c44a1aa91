"""Row-wise kernels at the edges of what a thread, a warp or a CTA holds of a row."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib, reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def bf(*shape, scale=1.0):
    return (torch.randn(*shape, device=DEV) * scale).bfloat16()


@pytest.mark.parametrize("rows", [1, 2, 3, 443, 889, 2500])
@pytest.mark.parametrize("D", [8, 256, 2048, 2056, 4096, 4104, 8192])
@pytest.mark.parametrize("with_res", [False, True])
def test_rms_norm_backward(rows, D, with_res):
    x, w, dy, dr = bf(rows, D), (1 + 0.1 * torch.randn(D, device=DEV)).bfloat16(), bf(rows, D), bf(rows, D)
    xs, ws = x.clone().requires_grad_(), w.clone().requires_grad_()
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    yd = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * wd
    if with_res:
        delta = bf(rows, D)
        res, y = ops.add_rms_norm(xs, delta, ws, 1e-6)
        torch.autograd.backward([res, y], [dr, dy])
        s = (x.float() + delta.float()).bfloat16().double().requires_grad_()
        yd = s * torch.rsqrt(s.square().mean(-1, keepdim=True) + 1e-6) * wd
        torch.autograd.backward([s, yd], [dr.double(), dy.double()])
        want = s.grad
    else:
        ops.rms_norm(xs, ws, 1e-6).backward(dy)
        yd.backward(dy.double())
        want = xd.grad
    _lib.check_status()
    # one rounding to bf16: at most 2^-8 of every element
    assert (xs.grad.double() - want).norm() < 4e-3 * want.norm()
    assert (ws.grad.double() - wd.grad).norm() < 4e-3 * wd.grad.norm()


@pytest.mark.parametrize("Hq,Hkv", [(1, 1), (3, 1), (5, 5), (16, 8), (32, 8)])
@pytest.mark.parametrize("rows", [1, 9, 300])
@pytest.mark.parametrize("interleaved", [False, True])
def test_qk_norm_rope_head_counts(Hq, Hkv, rows, interleaved):
    """Head counts below, at and across the number of heads that one warp takes."""
    D, H = 128, Hq + 2 * Hkv
    qkv, pos = bf(rows, H * D), torch.randint(0, 5000, (rows,), device=DEV)
    wq, wk = [(1 + 0.1 * torch.randn(D, device=DEV)).bfloat16() for _ in range(2)]
    xs, qs, ks = qkv.clone().requires_grad_(), wq.clone().requires_grad_(), wk.clone().requires_grad_()
    out = ops.qk_norm_rope_packed(xs, qs, ks, pos, Hq, Hkv, D, 1e6, 1e-6, interleaved)
    g = bf(*out.shape)
    out.backward(g)
    xf, qf, kf = [t.float().requires_grad_() for t in (qkv, wq, wk)]
    q, k = ref.qk_norm_rope(xf[:, :Hq * D].reshape(1, rows, Hq, D), xf[:, Hq * D:(Hq + Hkv) * D].reshape(1, rows, Hkv, D),
                            qf, kf, pos, 1e6, 1e-6, interleaved)
    want = torch.cat([q.reshape(rows, -1), k.reshape(rows, -1), xf[:, (Hq + Hkv) * D:]], 1)
    want.backward(g.float())
    _lib.check_status()
    assert (out.float() - want).norm() < 5e-3 * want.norm()
    assert torch.equal(out[:, (Hq + Hkv) * D:], qkv[:, (Hq + Hkv) * D:])
    for got, exp in ((xs.grad, xf.grad), (qs.grad, qf.grad), (ks.grad, kf.grad)):
        assert (got.float() - exp).norm() < 1e-2 * exp.norm()


@pytest.mark.parametrize("Hq,Hkv", [(1, 1), (2, 1), (3, 1), (2, 2)])
@pytest.mark.parametrize("rows", [1, 9, 300])
@pytest.mark.parametrize("interleaved", [False, True])
def test_rope_of_few_heads(Hq, Hkv, rows, interleaved):
    """Rows of up to four heads have a kernel of their own: a head's result is that of the same head in a wide row."""
    D = 128
    wide, pos = bf(rows, 16 * D), torch.randint(0, 5000, (rows,), device=DEV)           # 8 q heads, 4 k heads, 4 v heads
    wq, wk = [(1 + 0.1 * torch.randn(D, device=DEV)).bfloat16() for _ in range(2)]

    def few(t):
        return torch.cat([t[:, :Hq * D], t[:, 8 * D:(8 + Hkv) * D], t[:, 12 * D:(12 + Hkv) * D]], 1)

    want = ops.qk_norm_rope_packed(wide, wq, wk, pos, 8, 4, D, 1e6, 1e-6, interleaved)
    got = ops.qk_norm_rope_packed(few(wide), wq, wk, pos, Hq, Hkv, D, 1e6, 1e-6, interleaved)
    _lib.check_status()
    assert torch.equal(got, few(want))


@pytest.mark.parametrize("rows", [148, 149, 295, 296, 297, 592, 593])
@pytest.mark.parametrize("D", [2048, 2560])
def test_rms_norm_backward_rounds(rows, D):
    """Row counts at which the number of CTAs and of their rounds changes."""
    test_rms_norm_backward(rows, D, True)
