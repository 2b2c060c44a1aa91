"""Which kernel and plan a product of some rows gets: near the measured best of its shape, wherever the models' figures stand."""
import pytest

from ksa_b200.ops import _lib

# (rows, columns, K, ragged), us of the tiled kernel that serves it otherwise, and of the split-K plans (tile, split) that come within a fifth
# of the best; with ragged: bit 0 activations, bit 1 weights off the 128-byte lines.  Row-major and K-major weights take the same plan.
MEASURED = [
    ((333, 2560, 4096, 0), 28.7, {(48, 2): 14.2, (64, 2): 15.7, (80, 2): 16.7, (176, 2): 16.9}),
    ((576, 2560, 9728, 0), 59.8, {(192, 2): 29.5}),
    ((700, 2048, 12288, 0), 73.0, {(80, 2): 39.9, (176, 2): 34.2}),
    ((448, 2048, 6144, 0), 39.1, {(64, 2): 20.1, (80, 2): 21.9, (112, 2): 22.6, (112, 4): 21.4, (224, 2): 22.4, (224, 4): 19.4}),
    ((900, 4096, 2048, 0), 15.7, {}),
    ((2048, 9728, 2560, 0), 70.4, {}),
    ((140, 12288, 2048, 0), 16.1, {(48, 1): 15.3, (80, 1): 16.7}),
    ((8, 2560, 9728, 0), 55.8, {(16, 4): 12.6, (16, 8): 12.7}),
    ((12, 9728, 2560, 0), 21.8, {(16, 1): 12.2, (16, 2): 12.6}),
    ((17, 6144, 2560, 0), 18.1, {(32, 2): 9.7, (32, 4): 9.7}),
    ((40, 2048, 6144, 0), 36.3, {(48, 4): 11.0, (48, 8): 11.3}),
    ((64, 12288, 2048, 0), 15.4, {(64, 1): 14.9, (64, 2): 13.7}),
    ((128, 2560, 4096, 1), 29.9, {(48, 2): 12.0, (48, 4): 13.0, (64, 2): 14.0, (64, 4): 13.8, (128, 4): 14.0}),
    ((256, 4096, 2560, 0), 18.8, {(48, 1): 14.9, (64, 2): 12.7, (128, 2): 14.5}),
    ((40, 2560, 4096, 3), 34.2, {(48, 4): 9.9}),
    ((64, 9728, 2560, 2), 18.1, {(64, 1): 18.0, (64, 2): 15.2}),
    ((200, 3328, 1280, 3), 16.9, {(48, 1): 10.0, (48, 2): 10.8, (64, 1): 10.7, (64, 2): 11.2, (80, 1): 11.4, (112, 2): 10.3}),
    ((62, 1704, 416, 3), 4.3, {}),
    ((1151, 1184, 8472, 3), 54.6, {(176, 2): 39.1, (192, 2): 40.6, (240, 2): 46.1}),
    ((310, 3840, 4096, 0), 29.1, {(48, 1): 20.9, (80, 2): 17.6, (112, 2): 20.7, (160, 2): 19.5}),
    ((924, 408, 512, 0), 4.7, {}),
    ((32, 15856, 9728, 0), 57.7, {(32, 1): 52.9, (32, 2): 48.7, (32, 4): 54.2}),
    ((5, 18408, 6144, 2), 55.4, {(16, 1): 35.3, (16, 2): 38.5}),
]

GATED = [
    ((471, 7776, 2048), 18.5, {(128, 1): 20.6, (240, 1): 20.6}),
    ((675, 6144, 1024), 13.9, {(128, 1): 14.1, (144, 1): 14.6, (240, 1): 15.1}),
    ((1193, 3504, 2048), 18.4, {(128, 1): 20.1, (144, 1): 21.2, (240, 1): 20.2}),
    ((471, 9728, 2048), 24.8, {(160, 1): 23.1}),
    ((48, 19456, 2560), 22.5, {(48, 1): 20.2}),
    ((333, 1040, 1024), 8.1, {(48, 1): 7.6, (48, 2): 6.4, (64, 2): 7.4, (80, 2): 7.6}),
    ((129, 272, 2048), 6.7, {(48, 2): 7.3, (48, 4): 6.5, (48, 8): 7.1, (80, 4): 7.6}),
    ((200, 7680, 6144), 27.2, {(112, 2): 29.5, (208, 2): 25.8}),
    ((132, 6144, 4096), 17.3, {(48, 2): 15.9, (80, 2): 18.3}),
    ((280, 6144, 2560), 17.3, {(48, 1): 15.7, (64, 1): 17.2, (80, 1): 18.8, (96, 2): 16.0}),
    ((700, 3072, 4096), 21.0, {(64, 1): 24.0, (128, 2): 22.4, (144, 2): 23.6, (176, 1): 24.5, (240, 2): 21.3}),
    ((1024, 12288, 2048), 44.0, {}),
    ((1306, 3072, 1024), 13.8, {(112, 1): 13.1, (128, 1): 13.8, (144, 1): 14.4, (160, 1): 15.1, (224, 1): 14.3}),
    ((64, 2048, 1024), 6.7, {(64, 2): 7.5, (64, 4): 7.1}),
    ((381, 12288, 256), 11.7, {(128, 1): 9.6}),
]


@pytest.mark.parametrize("shape,tiled,plans", MEASURED, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "")
def test_the_choice_is_near_the_best(shape, tiled, plans):
    """Within a tenth, about the standard deviation of the modelled times."""
    M, N, K, ragged = shape
    plan = _lib.gemm_narrow_plan(M, N, K, 0, 32, ragged)
    time = tiled if plan is None else plans.get(plan, float("inf"))
    assert time <= 1.1 * min([tiled, *plans.values()]), (plan, time)


# (rows, gate and up rows, K), us of CTA pairs that apply the activation, and of the split-K kernel with the activation in a launch of its own
@pytest.mark.parametrize("shape,fused,split", [((429, 9728, 4096), 45.7, 39.4), ((571, 3072, 2048), 16.3, 14.8), ((77, 9728, 2048), 16.8, 15.2),
                                               ((1325, 6144, 2048), 28.4, 41.0), ((670, 12288, 2560), 36.7, 47.7), ((234, 12288, 2048), 17.7, 19.4)])
def test_a_separate_activation_counts_against_the_split(shape, fused, split):
    M, N, K = shape
    assert (_lib.gemm_narrow_plan(M, N, K, 2, 32) is not None) == (split < fused)


# (rows, gate and up rows, K), us of the product and the activation in two launches, and of the gated plans that come within a fifth of the best
@pytest.mark.parametrize("shape,two,gated", GATED, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "")
def test_the_gated_choice_is_near_the_best(shape, two, gated):
    M, N, K = shape
    plan = _lib.gemm_narrow_plan(M, N, K, 1, 32)
    time = two if plan is None else gated.get(plan, float("inf"))
    assert time <= 1.1 * min([two, *gated.values()]), (plan, time)


# (rows, columns, K, gated), us of the kernels that serve it otherwise, and with all rows in one tile
@pytest.mark.parametrize("shape,others,tall", [((357, 152, 512, 0), 4.5, 5.8), ((346, 1024, 1024, 0), 6.2, 6.8), 
                                               ((333, 2560, 9728, 0), 28.8, 24.5), ((328, 2048, 6144, 0), 16.9, 16.0), ((333, 2560, 4096, 0), 14.2, 15.7),
                                               ((290, 640, 4096, 0), 10.0, 9.2), ((334, 152, 12288, 0), 11.2, 13.5),
                                               ((132, 3072, 4096, 1), 16.1, 19.7), ((200, 3840, 6144, 1), 25.8, 30.1), ((100, 3072, 4096, 1), 16.1, 14.7),
                                               ((200, 3072, 2048, 1), 13.4, 11.9), ((132, 5920, 4096, 1), 25.3, 24.1)])
def test_all_rows_in_one_tile_where_that_is_faster(shape, others, tall):
    M, N, K, glu = shape
    assert (_lib.gemm_tall_plan(M, N, K, glu, False) is not None) == (tall < others)


@pytest.mark.parametrize("M,N,K", [(2049, 256, 2048), (64, 512, 56), (0, 512, 512)])
def test_no_plan(M, N, K):
    """More rows than the model holds for, less than 64 KB of weights, nothing."""
    assert _lib.gemm_narrow_plan(M, N, K, 0, 32) is None


@pytest.mark.parametrize("plan,args", [(_lib.gemm_narrow_plan, (333, 2560, 4096, 0, 32)), (_lib.gemm_tall_plan, (48, 2560, 4096, 0, False))])
def test_a_plan_is_searched_once(plan, args):
    plan.cache_clear()
    assert plan(*args) == plan(*args) and plan.cache_info()[:2] == (1, 1)         # hits, misses
