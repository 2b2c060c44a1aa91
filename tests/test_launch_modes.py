"""Launch modes of a thread: what ``KSA_DEPENDENT_LAUNCH=0`` and ``set_dependent_launch`` switch."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch

from ksa_b200 import ops
from ksa_b200.ops import _lib


@pytest.mark.parametrize("value,mode", [("0", "ORDINARY"), ("1", "DEPENDENT"), (None, "DEPENDENT")])
def test_the_environment_gives_every_thread_its_first_mode(value, mode):
    env = {k: v for k, v in os.environ.items() if k != "KSA_DEPENDENT_LAUNCH"}
    if value is not None:
        env["KSA_DEPENDENT_LAUNCH"] = value
    code = ("import threading\nfrom ksa_b200.ops import _lib\n"
            f"def look(): assert _lib.set_dependent_launch(_lib.EARLY_WEIGHTS) == _lib.{mode}; seen.append(1)\n"
            "seen = []\nt = threading.Thread(target=look); t.start(); t.join(); look(); assert len(seen) == 2")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], env=env, cwd=root, check=True, timeout=300)


def _edges(mode, work):
    """Types of the edges between the kernels of ``work``, captured in a launch mode: 0 full, 1 programmatic."""
    work()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    before = _lib.set_dependent_launch(mode)
    try:
        with torch.cuda.graph(graph):
            work()
    finally:
        _lib.set_dependent_launch(before)
    rt = ctypes.CDLL("libcudart.so.12")               # PyTorch's
    raw, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert rt.cudaGraphGetEdges_v2(raw, None, None, None, ctypes.byref(n)) == 0
    start, end, data = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)(), (ctypes.c_ubyte * (8 * n.value))()
    assert rt.cudaGraphGetEdges_v2(raw, start, end, data, ctypes.byref(n)) == 0
    return list(data[2::8])                           # 8 bytes an edge: from port, to port, type


@pytest.mark.gpu
def test_ordinary_launches_have_full_edges():
    x, w = torch.randn(64, 512, device="cuda").bfloat16(), torch.randn(512, 512, device="cuda").bfloat16()
    norm, ws = torch.ones(512, device="cuda").bfloat16(), torch.randn(1024, 512, device="cuda").bfloat16()
    labels, scale = torch.zeros(4, dtype=torch.int64, device="cuda"), torch.ones(1, device="cuda")
    loss = torch.empty(4, device="cuda")

    def work():                                       # a norm, the split-K product, a tiled one, the ring, a cluster kernel
        h = ops.linear(ops.rms_norm(x, norm), w)
        h = ops.gemm(h, w, out_dtype=torch.float32)
        h = ops.linear_swiglu(x[:4], ws)
        _lib.call("ksa_cross_entropy", h, labels, loss, scale, 4, 512, 512, -100, 1)
    with torch.no_grad():
        assert set(_edges(_lib.DEPENDENT, work)) == {1}
        assert set(_edges(_lib.EARLY_WEIGHTS, work)) == {1}
        ordinary = _edges(_lib.ORDINARY, work)
        assert len(ordinary) == 4 and set(ordinary) == {0}
