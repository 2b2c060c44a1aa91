"""Calls without autograd skip the autograd function; whoever follows the calls still meets it."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch
import torch.autograd.forward_ad as fwd

from ksa_b200 import ops
from ksa_b200.ops import _lib

ROOT = Path(__file__).resolve().parents[1]


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


# ------------------------------------------------------------------------- the framework's own calls, kernels replaced by a recorder
def _bf(*shape):
    return torch.ones(*shape).bfloat16()


_W = {"w": _bf(64, 64), "n": _bf(64), "n16": _bf(16), "kv": _bf(1, 128, 1, 128)}
_CALLS = {
    "linear": (lambda x: ops.linear(x, _W["w"]), (32, 64)),
    "dual_linear": (lambda x: ops.dual_linear(x, _W["w"], _W["w"], 20), (32, 64)),
    "rms_norm": (lambda x: ops.rms_norm(x, _W["n"]), (32, 64)),
    "add_rms_norm": (lambda x: ops.add_rms_norm(x, x, _W["n"])[1], (32, 64)),
    "qk_norm_rope_packed": (lambda x: ops.qk_norm_rope_packed(x, _W["n16"], _W["n16"], torch.arange(32), 2, 1, 16, 1e4, 1e-6), (32, 64)),
    "swiglu": (lambda x: ops.swiglu(x), (32, 64)),
    "linear_swiglu": (lambda x: ops.linear_swiglu(x, _W["w"]), (32, 64)),
    "linear_swiglu of few rows": (lambda x: ops.linear_swiglu(x, _W["w"]), (8, 64)),
    "embedding": (lambda x: ops.embedding(torch.arange(3), x), (32, 64)),
    "causal_attention": (lambda x: ops.causal_attention(x, _W["kv"], _W["kv"]), (1, 128, 1, 128)),
    "ksa_attention": (lambda x: ops.ksa_attention(x, _W["kv"], _W["kv"], x[:, :1], _W["kv"][:, :1], _W["kv"][:, :1], 128, 1, 2)[0],
                      (1, 128, 1, 128)),
    "attention_packed": (lambda x: ops.attention_packed(x, 1, 32, 0, 2, 1, 16, 16, 1, 2), (32, 64)),
}
_TRANSFORMS = {
    "functionalize": lambda f, x: torch.func.functionalize(f)(x),
    "vmap": lambda f, x: torch.func.vmap(f)(x[None]),
    "vmap of something else": lambda f, x: torch.func.vmap(lambda other: f(x) + other)(torch.ones(2).bfloat16()),
    "grad": lambda f, x: torch.func.grad(lambda t: f(t).float().sum())(x),
    "jvp": lambda f, x: torch.func.jvp(f, (x,), (x,)),
}


@pytest.fixture
def recorder(monkeypatch):
    """What reaches the kernels' entry points: the addresses of the tensors."""
    calls = []
    monkeypatch.setattr(ops, "_cuda", lambda x: True)
    monkeypatch.setattr(_lib, "call", lambda name, *args: calls.append(
        [a.data_ptr() for a in args if isinstance(a, torch.Tensor) and a.numel() > 0]))
    monkeypatch.setattr(_lib, "gemm_narrow_plan", lambda *sizes: (32, 1))
    return calls


@pytest.mark.parametrize("name", list(_CALLS))
def test_an_op_reaches_its_kernel(name, recorder):
    f, shape = _CALLS[name]
    f(_bf(*shape))
    assert recorder and all(p != 0 for c in recorder for p in c)


@pytest.mark.parametrize("transform", list(_TRANSFORMS))
@pytest.mark.parametrize("name", [n for n in _CALLS if n != "linear_swiglu of few rows"])
def test_an_op_is_refused_under_a_transform(name, transform, recorder):
    """The autograd functions have no rule for transforms, and PyTorch says so; nothing of a wrapper reaches a kernel."""
    f, shape = _CALLS[name]
    with torch.no_grad(), pytest.raises(RuntimeError, match="functorch transforms"):
        _TRANSFORMS[transform](f, _bf(*shape))
    assert not recorder


def test_a_tensor_without_memory_is_refused():
    class OnGpu(torch.Tensor):
        is_cuda = True

    def make(t):
        return torch.Tensor._make_subclass(OnGpu, t)

    assert _lib._ptr(make(torch.ones(3))) != 0 and _lib._ptr(make(torch.empty(0))) == 0
    hollow = torch._to_functional_tensor(torch.ones(3))
    assert hollow.data_ptr() == 0
    hollow = make(torch.ones(3))
    hollow.data_ptr = lambda: 0
    with pytest.raises(RuntimeError, match="without memory"):
        _lib._ptr(hollow)


@pytest.mark.parametrize("transform", ["jvp", "grad"])
@pytest.mark.parametrize("call", [lambda t: ops.linear(_bf(32, 64), t), lambda t: ops.embedding(torch.arange(3), t),
                                  lambda t: ops.linear(t, _W["w"]), lambda t: ops.rms_norm(t, _W["n"])])
def test_a_tensor_that_outlived_its_transform(call, transform, monkeypatch):
    """What a finished transform left behind is an ordinary tensor again."""
    calls = []
    monkeypatch.setattr(ops, "_cuda", lambda x: True)

    def record(name, *args):
        for a in args:
            if isinstance(a, torch.Tensor):
                calls.append(_lib._address(a))
    monkeypatch.setattr(_lib, "call", record)
    kept = []
    _TRANSFORMS[transform](lambda t: (kept.append(t), t.float().sum())[1], _bf(64, 64))
    call(kept[0])
    assert calls and all(calls)


@pytest.mark.parametrize("rows", [8, 32])
@pytest.mark.parametrize("width", [56, 72])
def test_linear_swiglu_refuses_other_widths(rows, width, recorder):
    """The fused kernels take the reduction length from the activations alone."""
    with torch.no_grad(), pytest.raises(AssertionError, match="reduction mismatch"):
        ops.linear_swiglu(_bf(rows, width), _W["w"])
    with torch.no_grad(), pytest.raises(AssertionError):
        ops.linear_swiglu(_bf(rows, 64), _W["w"][None])
    assert not recorder


@pytest.mark.parametrize("width", [56, 72])
@pytest.mark.parametrize("glu", [False, True])
def test_norm_linear_refuses_other_widths(width, glu, recorder):
    with torch.no_grad(), pytest.raises(AssertionError, match="reduction mismatch"):
        ops.norm_linear(_bf(2, width), None, _bf(width), 1e-6, _W["w"], glu)
    assert len(recorder) == 1, "the norm alone, as a call of its own"


@pytest.mark.parametrize("requires", [False, True])
def test_linear_swiglu_asks_for_its_plan_once(requires, recorder, monkeypatch):
    """Once where it can use the answer, not at all where the call is differentiated (the projection asks for its own)."""
    asked = []
    monkeypatch.setattr(_lib, "gemm_narrow_plan", lambda M, N, K, glu, *rest: asked.append(glu) or (32, 1))
    ops.linear_swiglu(_bf(32, 64).requires_grad_(requires), _W["w"])
    assert asked == ([0] if requires else [1])


def test_private_names_of_pytorch_are_there():
    """The bypass works without them, but then every call takes the long way; a newer PyTorch should not do that unseen."""
    assert hasattr(torch._C, "_are_functorch_transforms_active") and hasattr(fwd, "_current_level")
    assert torch._C._functorch.unwrap_if_dead(torch.ones(1)) is not None
    assert not ops._observed()


def test_without_private_names_every_call_is_observed():
    code = ("import torch\nimport torch.autograd.forward_ad as fwd\ndel fwd._current_level\n"
            "from ksa_b200 import ops\nassert ops._observed()\n")
    assert subprocess.run([sys.executable, "-c", code], cwd=ROOT).returncode == 0
