"""Row-wise kernels at the edges of what a thread, a warp or a CTA holds of a row."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

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
