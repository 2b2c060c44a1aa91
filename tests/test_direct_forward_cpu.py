"""Calls without autograd skip the autograd function; whoever follows the calls still meets it."""
import pytest
import torch
import torch.autograd.forward_ad as fwd

from ksa_b200 import ops


class _Twice(torch.autograd.Function):
    seen = []

    @staticmethod
    def forward(ctx, x, k):
        _Twice.seen.append(type(ctx).__name__)
        ctx.save_for_backward(x)
        ctx.k = k
        return x * k

    @staticmethod
    def backward(ctx, g):
        return g * ctx.k, None


@pytest.mark.parametrize("grad_mode", [False, True])
@pytest.mark.parametrize("requires", [False, True])
def test_direct_exactly_without_autograd(grad_mode, requires):
    _Twice.seen.clear()
    x = torch.ones(3, requires_grad=requires)
    with torch.set_grad_enabled(grad_mode):
        y = ops._run(_Twice, x, 2)
    assert y.requires_grad == (grad_mode and requires) and torch.equal(y, torch.full((3,), 2.0))
    assert (_Twice.seen == ["_NoGrad"]) == (not y.requires_grad)
    if y.requires_grad:
        y.sum().backward()
        assert torch.equal(x.grad, torch.full((3,), 2.0))


def test_forward_mode_is_still_refused():
    with fwd.dual_level(), torch.no_grad():
        x = fwd.make_dual(torch.ones(3), torch.ones(3))
        with pytest.raises(RuntimeError):
            ops._run(_Twice, x, 2)


def test_a_trace_still_meets_the_function():
    with torch.no_grad():
        traced = torch.jit.trace(lambda x: ops._run(_Twice, x, 2), torch.ones(3), check_trace=False)
    assert torch.equal(traced(torch.full((3,), 5.0)), torch.full((3,), 10.0))
