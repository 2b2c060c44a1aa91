"""RMSNorm forward: the line between a CTA and a warp per row, widths around the vectors of a lane, residuals of fewer rows."""
import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 1023, 1024, 1025, 5001])
@pytest.mark.parametrize("D", [8, 248, 1024, 1032, 2048, 2056, 2560, 2568])
def test_forward(rows, D):
    x, w = (torch.randn(rows, D, device="cuda") * 2).bfloat16(), (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16()
    for n in (None, rows, max(1, rows // 3)):
        d = None if n is None else torch.randn(n, D, device="cuda").bfloat16()
        res, y = ops.add_rms_norm(x, d, w)
        want = x.clone()
        if d is not None:
            want[:n] += d
        assert torch.equal(res, want)
        h = want.double()
        h = h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * w.double()
        # one rounding to bf16, half of 2^-7, of a value whose fp32 sum, rsqrt and products leave less than 2^-19
        assert bool(((y.double() - h).abs() <= h.abs() * (2.0 ** -8 + 2.0 ** -19) + 1e-30).all())
    _lib.check_status()
