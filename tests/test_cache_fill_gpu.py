"""A prompt's keys and values in the caches: one launch a layer against the copies of every part."""
import pytest
import torch

from ksa_b200.config import get_preset
from ksa_b200.inference import KsaInferenceEngine
from ksa_b200.inference import engine as module
from ksa_b200.models import get_model_class
from ksa_b200.ops import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window,n_sum", [(2, 1), (4, 2), (0, 1)])
@pytest.mark.parametrize("lengths", [[1, 1], [15, 15], [16, 16], [31, 31], [32, 32], [64, 64], [100, 100], [100, 33], [7, 100]])
def test_one_launch_fills_what_the_copies_fill(monkeypatch, lengths, window, n_sum):
    cfg = get_preset("qwen3-ksa-tiny").merge({"summary_chunk_size": 16, "summary_sliding_chunk_num": window, "summary_token_num": n_sum})
    torch.manual_seed(0)
    model = get_model_class(cfg.model_class)(cfg)
    model.init_weights(seed=0)
    model = model.cuda().bfloat16()
    tokens = torch.randint(0, cfg.vocab_size, (2, max(lengths)), device="cuda")
    fill, used = module._cache_fill, []

    def run(one_launch):
        monkeypatch.setattr(module, "_cache_fill", lambda *a: used.append(fill(*a)) or used[-1] if one_launch else False)
        engine = KsaInferenceEngine(model, max_len=160, batch=2)
        logits = engine.prefill(tokens, lengths)
        return [logits] + [t for c in engine.layer_caches for t in (c.k, c.v)]
    got, want = run(True), run(False)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert used and all(used)
    _lib.check_status()


def test_a_cache_that_is_too_small_is_refused():
    k = torch.zeros(1, 2, 16, 64, device="cuda").bfloat16()
    qkv = torch.zeros(17, 8 * 64, device="cuda").bfloat16()
    with pytest.raises(RuntimeError, match="17 rows"):
        module._cache_fill(qkv, k, k.clone(), 1, 17, 0, 4, 2, 64, None)
