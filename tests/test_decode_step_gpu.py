"""The small parts of a decode step: slices in one launch, queries at their pitch, the merge of splits, the last norm inside the head."""
import pytest
import torch

from ksa_b200.config import get_preset
from ksa_b200.inference import KsaInferenceEngine
from ksa_b200.inference.cache import CacheSpec, CacheState, text_step_slices
from ksa_b200.inference.engine import _decode_attention, _step_slices
from ksa_b200.models import get_model_class
from ksa_b200.ops import _lib, reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk,n_sum,window", [(128, 1, 8), (64, 4, 2), (16, 2, 0), (128, 1, 1)])
def test_slices_of_a_step(chunk, n_sum, window):
    """Every chunk phase, with fewer chunks done than the window holds, as many, and more; more sequences than a block has threads."""
    spec = CacheSpec(chunk=chunk, n_sum=n_sum, window=window, max_chunks=3 * window + 4)
    done = torch.arange(3 * window + 4, dtype=torch.int32).repeat_interleave(chunk)
    state = CacheState(done.numel(), "cuda")
    state.chunks.copy_(done)
    state.cbl.copy_(torch.arange(chunk, dtype=torch.int32).repeat(3 * window + 4))
    for got, want in zip(_step_slices(spec, state), text_step_slices(spec, state)):
        assert torch.equal(got, want)
    _lib.check_status()


def _cache(B, Hkv, cap, D):
    return tuple(torch.randn(B, Hkv, cap, D, device="cuda").bfloat16() for _ in range(2))


@pytest.mark.parametrize("B,Tq,Hq,Hkv,D,pitch,offset", [
    (3, 1, 8, 2, 128, 1536, 0),       # the query columns of packed projection rows
    (3, 1, 8, 2, 128, 1032, 8),       # any multiple of 16 bytes
    (3, 1, 8, 2, 128, 1028, 0),       # rows off the 16-byte lines: copied first
    (3, 1, 8, 2, 128, 1536, 4),       # a start off them
    (1, 1, 8, 2, 128, 1536, 0), (2, 3, 8, 2, 128, 1536, 0), (1, 2, 4, 2, 64, 520, 8), (4, 1, 4, 2, 64, 512, 16)])
def test_queries_at_a_pitch(B, Tq, Hq, Hkv, D, pitch, offset):
    k, v = _cache(B, Hkv, 300, D)
    start = torch.randint(0, 50, (B, Tq), device="cuda", dtype=torch.int32)
    length = torch.randint(1, 250, (B, Tq), device="cuda", dtype=torch.int32)
    rows = torch.randn(offset + B * Tq * pitch, device="cuda").bfloat16()[offset:].view(B * Tq, pitch)
    q = rows[:, :Hq * D].unflatten(0, (B, Tq)).unflatten(2, (Hq, D))
    want = _decode_attention(q.contiguous().clone(), k, v, start, length, D ** -0.5)
    assert torch.equal(_decode_attention(q, k, v, start, length, D ** -0.5), want)
    heads_first = q.transpose(1, 2).contiguous().transpose(1, 2)
    assert torch.equal(_decode_attention(heads_first, k, v, start, length, D ** -0.5), want)
    _lib.check_status()


@pytest.mark.parametrize("cap", [100, 128, 129, 640, 1000, 8064, 8192, 20000])     # 1, 1, 2, 5, 8, 63, 64 and 64 wider splits
@pytest.mark.parametrize("Tq,Hq,Hkv", [(1, 2, 2), (1, 6, 2), (3, 2, 2), (1, 10, 2), (2, 6, 2), (1, 14, 2)])   # 1, 3, 3, 5, 6, 7 queries
def test_merge_of_splits(cap, Tq, Hq, Hkv):
    D = 128
    k, v = _cache(2, Hkv, cap, D)
    q = torch.randn(2, Tq, Hq, D, device="cuda").bfloat16()
    start = torch.randint(0, 3, (2, Tq), device="cuda", dtype=torch.int32)
    length = torch.randint(cap - 10, cap - 2, (2, Tq), device="cuda", dtype=torch.int32)
    out = _decode_attention(q, k, v, start, length, D ** -0.5)
    for t in range(Tq):
        want = ref.decode_attention(q[:, t:t + 1].float(), k.float(), v.float(), length[:, t].long(), start[:, t].long(), D ** -0.5)
        # probabilities and result in bf16: 2^-9 each, some more for the scores' products
        assert (out[:, t:t + 1].float() - want).norm() <= 2 ** -7 * want.norm()
    _lib.check_status()


@pytest.mark.parametrize("batch", [1, 3, 4])
def test_the_last_norm_inside_the_head(batch):
    cfg = get_preset("qwen3-ksa-tiny").merge({"head_dim": 128, "num_heads": 4, "num_kv_heads": 2, "embed_dim": 512})
    model = get_model_class(cfg.model_class)(cfg)
    model.init_weights(seed=0)
    model = model.to("cuda").to(torch.bfloat16)
    prompt = torch.randint(0, cfg.vocab_size, (batch, 50), device="cuda")
    token = torch.randint(0, cfg.vocab_size, (batch,), device="cuda")
    logits = []
    with torch.no_grad():
        for with_head in (True, False):
            engine = KsaInferenceEngine(model, max_len=128, batch=batch)
            engine.prefill(prompt)
            out = engine._decode_impl(token, False, with_head)
            logits.append((out if with_head else engine._logits(out)).float())
            assert engine.state.text_len.tolist() == [51] * batch
    # the order of the norm's sum turns some roundings of the norm and of the logits, 2^-8 at most each
    assert (logits[0] - logits[1]).norm() <= 2 ** -7 * logits[1].norm()
    _lib.check_status()
