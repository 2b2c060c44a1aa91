"""The ordinary operator calls in native code against the general Python way: same bits, same refusals, same prototypes."""
import re
from pathlib import Path

import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib

CSRC = Path(__file__).resolve().parents[1] / "ksa_b200" / "csrc"


def _kinds(args):
    return ["P" if "*" in a else "L" if "long long" in a else "F" if "float" in a else "I" for a in args.split(",")]


def test_declarations_match_the_prototypes():
    prototypes = {}
    for f in CSRC.glob("*.cu"):
        prototypes.update(re.findall(r"KSA_API int (ksa_\w+)\(([^)]*)\)\s*\{", f.read_text()))
    declared = re.findall(r"^int (ksa_\w+)\(([^)]*)\);", (CSRC / "native.cpp").read_text(), flags=re.M)
    assert len(declared) >= 15
    for name, args in declared:
        assert _kinds(args) == _kinds(prototypes[name]), name


def test_what_is_not_plain_is_left_to_python():
    """CPU tensors, subclasses, wrappers, other numbers of arguments: None, before anything is read or launched."""
    if isinstance(_lib.native, _lib.NotBuilt):
        pytest.skip("the native calls are not built")
    w = torch.ones(64, 64).bfloat16()

    class Sub(torch.Tensor):
        pass
    for x in (w, w.as_subclass(Sub), torch._to_functional_tensor(w), None, 3):
        assert _lib.native.linear(x, w, 32) is None and _lib.native.gemm(x, w, None, False, False, False, False, 32) is None
        assert _lib.native.swiglu(x) is None and _lib.native.rms_norm(x, None, w[0], 1e-6) is None
    assert _lib.native.linear(w, w) is None and _lib.native.linear() is None and _lib.native.linear(w, w, "32") is None
    assert _lib.native.launches() == 0 or torch.cuda.is_available()


def _n(*shape, std=1.0):
    return (torch.randn(*shape, device="cuda") * std).bfloat16()


def _weight(n, k, main_grad):
    w = torch.nn.Parameter(_n(n, k, std=0.05) if k else 1 + _n(n, std=0.1))
    if main_grad:
        w.main_grad = torch.zeros(w.shape, dtype=torch.float32, device="cuda")
    return w


def _case(name, rows, main_grad):
    """A call and the tensors that it differentiates."""
    x, w, pos = _n(rows, 256), _weight(512, 256, main_grad), torch.arange(rows, device="cuda")
    if name == "linear":
        return lambda: ops.linear(x, w), [x, w]
    if name == "linear of rows with a pitch":
        wide = _n(rows, 320)
        return lambda: ops.linear(wide[:, :256], w), [wide, w]
    if name == "linear of three dimensions":
        y = _n(2, rows, 256)
        return lambda: ops.linear(y, w), [y, w]
    if name == "linear of columns":
        y = _n(256, rows)
        return lambda: ops.linear(y.t(), w), [y, w]
    if name == "dual_linear":
        w2 = _weight(512, 256, main_grad)
        return lambda: ops.dual_linear(x, w, w2, rows // 3), [x, w, w2]
    if name == "add_rms_norm":
        s, d = _weight(256, 0, main_grad), _n(rows - rows // 4, 256)
        return lambda: torch.cat(ops.add_rms_norm(x, d, s)), [x, d, s]
    if name == "rms_norm of three dimensions":
        s, y = _weight(256, 0, main_grad), _n(2, rows, 256)
        return lambda: ops.rms_norm(y, s), [y, s]
    if name == "swiglu":
        return lambda: ops.swiglu(x), [x]
    if name == "qk_norm_rope":
        q, k, y = _weight(128, 0, main_grad), _weight(128, 0, main_grad), _n(rows, 4 * 128)
        return lambda: ops.qk_norm_rope_packed(y, q, k, pos, 2, 1, 128, 1e4), [y, q, k]
    if name == "qk_norm_rope of rows with a pitch, without norms":
        y = _n(rows, 640)
        return lambda: ops.qk_norm_rope_packed(y[:, :512], None, None, pos, 2, 1, 128, 1e4), [y]
    if name == "attention":
        y = _n(rows, 4 * 128)
        return lambda: ops.attention_packed(y, 1, rows, 0, 2, 1, 128), [y]
    y = _n(2 * (rows + rows // 16 * 2), 4 * 128)
    return lambda: ops.attention_packed(y, 2, rows, rows // 16 * 2, 2, 1, 128, 16, 2, 3), [y]


_NAMES = ["linear", "linear of rows with a pitch", "linear of three dimensions", "linear of columns", "dual_linear", "add_rms_norm",
          "rms_norm of three dimensions", "swiglu", "qk_norm_rope", "qk_norm_rope of rows with a pitch, without norms", "attention",
          "summary attention"]


def _run(name, rows, main_grad, monkeypatch, native):
    with monkeypatch.context() as m:
        if not native:
            m.setattr(ops, "_native", _lib.NotBuilt())
        torch.manual_seed(7)
        f, leaves = _case(name, rows, main_grad)
        with torch.no_grad():
            plain = f()
        for t in leaves:
            t.requires_grad_()
        y = f()
        y.backward(torch.randn(y.shape, device="cuda").bfloat16())
        y2 = f()                                            # a second use of the weights adds to their gradients
        y2.backward(torch.ones_like(y2))
        return [plain, y, y2] + [t.grad if t.grad is not None else t.main_grad for t in leaves]


@pytest.mark.gpu
@pytest.mark.parametrize("main_grad", [False, True])
@pytest.mark.parametrize("rows", [3, 16, 17, 130])
@pytest.mark.parametrize("name", _NAMES)
def test_same_bits_as_the_general_way(name, rows, main_grad, monkeypatch):
    assert not isinstance(_lib.native, _lib.NotBuilt)
    if name == "summary attention" and rows < 16:
        rows = 16
    before, python = _lib.native.launches(), _lib._launch_count
    a = _run(name, rows, main_grad, monkeypatch, True)
    assert _lib.native.launches() > before or name.startswith("rms_norm")
    if main_grad and not any(w in name for w in ("dimensions", "columns", "pitch")):
        assert _lib._launch_count == python, "an ordinary call went the long way"
    b = _run(name, rows, main_grad, monkeypatch, False)
    for i, (x, y) in enumerate(zip(a, b)):
        if i >= 3 and ("attention" in name or "rope" in name):      # sums with atomics: their order varies
            assert (x.float() - y.float()).norm() <= 1e-2 * y.float().norm() + 1e-6, (name, i)
        else:
            assert torch.equal(x, y), (name, i)
    _lib.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("call, error", [
    (lambda: ops.linear(_n(4, 64).float(), _n(8, 64)), TypeError),
    (lambda: ops.linear(_n(4, 64), _n(8, 72)), AssertionError),
    (lambda: ops.linear(_n(4, 64), _n(8, 64).cpu()), TypeError),
    (lambda: ops.linear(_n(40, 60), _n(64, 60)), RuntimeError),
    (lambda: ops.dual_linear(_n(4, 64), _n(8, 64), _n(16, 64), 2), AssertionError),
    (lambda: ops.gemm(_n(32, 64), _n(64, 64), out=_n(32, 32)), AssertionError),
    (lambda: ops.attention_packed(_n(100, 512), 1, 64, 0, 2, 1, 128), AssertionError),
    (lambda: ops.qk_norm_rope_packed(_n(4, 288), None, None, torch.arange(4, device="cuda"), 1, 1, 96, 1e4), RuntimeError),
])
@pytest.mark.parametrize("native", [False, True])
def test_same_refusals(call, error, native, monkeypatch):
    if not native:
        monkeypatch.setattr(ops, "_native", _lib.NotBuilt())
    with pytest.raises(error):
        call()


@pytest.mark.gpu
def test_saved_tensor_hooks_and_a_capture():
    x, w = _n(40, 256).requires_grad_(), _weight(512, 256, False)
    ref = torch.autograd.grad(ops.swiglu(ops.linear(x, w)).float().sum(), [x, w])
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.cuda()):
        y = ops.swiglu(ops.linear(x, w)).float().sum()
    got = torch.autograd.grad(y, [x, w])
    assert all(torch.equal(a, b) for a, b in zip(ref, got))
    with torch.no_grad():
        want, g = ops.linear_swiglu(x, w), torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out = ops.linear_swiglu(x, w)
        out.zero_()
        g.replay()
        assert torch.equal(out, want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side), torch.no_grad():
        z = ops.linear_swiglu(x, w)
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(z, want)
