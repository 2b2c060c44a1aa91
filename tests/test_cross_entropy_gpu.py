"""Cross entropy in place with a row in the shared memory of 1, 2, 4 or 8 CTAs (and above that on one CTA), against fp64."""
import pytest
import torch

from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grad", [0, 1])
@pytest.mark.parametrize("V", [8, 24, 4096, 40960, 40968, 81920, 81928, 151936, 163848, 327680, 327688])
def test_rows(V, grad):
    rows = 7
    x = (torch.randn(rows, V + 16, device="cuda") * 3).bfloat16()
    labels = torch.randint(0, V, (rows,), device="cuda")
    labels[1], labels[2], labels[3], labels[4] = -100, V - 1, V, 0
    x[4, 1:V] = float("-inf")                                     # all but the label masked: whole CTAs without a finite score
    x[5, :V // 2] = float("-inf")
    labels[5] = V - 1
    x[6, 0] = float("nan")
    y, loss, scale = x.clone(), torch.full((rows,), 7.0, device="cuda"), torch.tensor([0.25], device="cuda")
    _lib.call("ksa_cross_entropy", y, labels, loss, scale, rows, V, y.stride(0), -100, grad)
    _lib.check_status()
    assert torch.equal(y[:, V:], x[:, V:])
    z = x[:, :V].double()
    logp, ok = z.log_softmax(-1), (labels >= 0) & (labels < V)
    at = labels.clamp(0, V - 1)[:, None]
    want = torch.where(ok, -logp.gather(1, at)[:, 0], torch.zeros_like(logp[:, 0]))
    assert bool(loss[6].isnan()) and bool(want[6].isnan())
    # __expf and __logf: 2^-21 relative each, a sum of V terms of one sign
    assert float((loss[:6].double() - want[:6]).abs().max()) < 2e-5
    if not grad:
        assert torch.equal(y[:6], x[:6])
        return
    g = logp.exp()
    g.scatter_add_(1, at, -torch.ones_like(at, dtype=torch.float64))
    g = torch.where(ok[:, None], g * 0.25, torch.zeros_like(g))
    assert bool(y[6, :V].isnan().all())
    err = (y[:6, :V].double() - g[:6]).abs()
    # one rounding to bf16, half of 2^-7, of a p with less than 2^-17 (arguments of __expf down to -40), and (p - 1) / 4 with p's 2^-19
    assert bool((err <= (2.0 ** -8 + 2.0 ** -16) * g[:6].abs() + 2.0 ** -21).all()), float(err.max())


@pytest.mark.parametrize("V", [4096, 327688])
def test_logits_off_16_bytes_are_refused(V):
    """Both kernels read and write 16 bytes at a time."""
    x = torch.zeros(2 * V + 8, device="cuda").bfloat16()[4:4 + 2 * V].view(2, V)
    loss, labels = torch.zeros(2, device="cuda"), torch.zeros(2, dtype=torch.int64, device="cuda")
    with pytest.raises(RuntimeError, match="aligned"):
        _lib.call("ksa_cross_entropy", x, labels, loss, loss, 2, V, V, -100, 1)
    _lib.check_status()
