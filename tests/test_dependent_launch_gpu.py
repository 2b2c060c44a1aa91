"""Kernels start while their predecessor on the stream still runs: whatever one writes, the next one reads, weights included."""
import threading

import pytest
import torch

from ksa_b200 import ops
from ksa_b200.config import get_preset
from ksa_b200.inference.engine import KsaInferenceEngine
from ksa_b200.models import get_model_class
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu


def _n(*shape, std=1.0):
    return (torch.randn(*shape, device="cuda") * std).bfloat16()


def _chain(x, a, b, norm, sync):
    """Products whose weights and activations come from the kernel just before, through buffers that are used again."""
    outs = []
    w, y = torch.empty(512, 512, device="cuda").bfloat16(), torch.empty(x.shape[0], 512, device="cuda").bfloat16()
    for i in range(8):
        ops.gemm(a[i], b, out=w)                       # weights of the next product
        sync()
        ops.gemm(x if i == 0 else y.clone(), w, out=y)
        sync()
        res, h = ops.add_rms_norm(y, x, norm)
        sync()
        h = ops.swiglu(ops.linear(h, w))
        sync()
        ops.gemm(torch.cat([h, h], 1), w, out=y)
        sync()
        outs += [y.clone(), res]
    return outs


@pytest.mark.parametrize("rows", [1, 3, 16, 40, 700, 6000])
def test_a_chain_of_products(rows):
    with torch.no_grad():
        x, a, b, norm = _n(rows, 512), _n(8, 512, 512, std=0.05), _n(512, 512, std=0.05), _n(512)
        want = _chain(x, a, b, norm, torch.cuda.synchronize)
        for _ in range(5):
            got = _chain(x, a, b, norm, lambda: None)
            assert all(torch.equal(g, w) for g, w in zip(got, want))
    _lib.check_status()


@pytest.mark.parametrize("writer", ["adamw", "gemm", "copy"])
def test_a_decode_step_sees_the_weights_of_the_kernel_before(writer):
    cfg = get_preset("qwen3-ksa-tiny").merge({"head_dim": 128, "num_heads": 4, "num_kv_heads": 2, "embed_dim": 512})
    torch.manual_seed(0)
    model = get_model_class(cfg.model_class)(cfg)
    model.init_weights(seed=0)
    model = model.to("cuda").to(torch.bfloat16)
    w = model.layers[0].attn.wqkv.weight
    prompt = torch.randint(0, cfg.vocab_size, (2, 40), device="cuda")
    tokens = torch.randint(0, cfg.vocab_size, (12, 2), device="cuda")
    master = [w.detach().float() * (1 + 0.2 * i) for i in range(12)]
    start = w.detach().clone()

    def steps(sync):
        w.detach().copy_(start)
        engine = KsaInferenceEngine(model, max_len=128, batch=2)
        engine.prefill(prompt)
        out = []
        for i, t in enumerate(tokens):
            flat = master[i].reshape(-1).clone()
            if writer == "adamw":
                zero = torch.zeros_like(flat)
                ops.adamw_step(flat, zero, zero.clone(), zero.clone(), w.detach().view(-1),
                               torch.tensor([0.0, 1, 1, 1], device="cuda"), 0.9, 0.9, 1e-8, 0.0)
            elif writer == "gemm":
                ops.gemm(master[i].bfloat16(), torch.eye(w.shape[1], device="cuda").bfloat16(), out=w.detach())
            else:
                w.detach().copy_(master[i])
            sync()
            out.append(engine.decode_step(t))
            sync()
        return torch.stack(out)
    with torch.no_grad():
        want = steps(torch.cuda.synchronize)
        for _ in range(3):
            assert torch.equal(steps(lambda: None), want)
    _lib.check_status()


def test_products_beside_a_decode_step_wait_for_their_weights():
    """Early weights belong to the thread that runs a decode step: products of other threads, of up to 16 rows as well, wait."""
    with torch.no_grad():
        x, a, b, norm = _n(3, 512), _n(8, 512, 512, std=0.05), _n(512, 512, std=0.05), _n(512)
        want = _chain(x, a, b, norm, torch.cuda.synchronize)
        got = []

        def other():
            with torch.no_grad():
                got.extend(_chain(x, a, b, norm, lambda: None) for _ in range(5))
        before = _lib.set_dependent_launch(_lib.EARLY_WEIGHTS)
        try:
            t = threading.Thread(target=other)
            t.start()
            t.join()
        finally:
            _lib.set_dependent_launch(before)
        torch.cuda.synchronize()
        assert len(got) == 5 and all(torch.equal(g, w) for run in got for g, w in zip(run, want))
    _lib.check_status()
