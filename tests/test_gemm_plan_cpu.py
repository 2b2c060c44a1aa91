"""Which plan the split-K kernel gets: near the measured best of a shape, and none where the tiled kernels are as fast."""
import pytest

from ksa_b200.ops import _lib


@pytest.mark.parametrize("M,N,K,glu,plan", [
    (333, 2560, 4096, 0, (48, 2)), (576, 2560, 9728, 0, (192, 2)), (700, 2048, 12288, 0, (176, 2)), (448, 2048, 6144, 0, (224, 4)),
    (900, 4096, 2048, 0, None), (2048, 9728, 2560, 0, None), (2049, 256, 2048, 0, None),
    (64, 512, 56, 0, None),                                                    # less than 64 KB of weights
    (140, 12288, 2048, 0, (48, 1)), (140, 12288, 2048, 2, None),               # 2: a separate activation counts on this side
    (576, 4096, 9728, 2, (144, 2))])
def test_plan(M, N, K, glu, plan):
    assert _lib.gemm_narrow_plan(M, N, K, glu, 32) == plan


@pytest.mark.parametrize("plan,args", [(_lib.gemm_narrow_plan, (333, 2560, 4096, 0, 32)), (_lib.gemm_tall_plan, (48, 2560, 4096, 0, False))])
def test_a_plan_is_searched_once(plan, args):
    plan.cache_clear()
    assert plan(*args) == plan(*args) and plan.cache_info()[:2] == (1, 1)         # hits, misses
