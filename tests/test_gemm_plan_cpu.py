"""How bf16 tensor-core projections are cut (l3_debug_gemm_plan; needs no GPU): where the slices of a residual projection may be added in
the order they arrive, so that last bits differ from run to run, and where they may not."""
import numpy as np
import pytest

from llama3_np_b200 import _cabi

STORE, RESID, GATED = 0, 1, 2


def plan(rows, n, k, epi=STORE, fp32=0):
    p = np.zeros(5, np.int32)
    _cabi.check(_cabi.lib().l3_debug_gemm_plan(rows, n, k, epi, fp32, _cabi.i32p(p)))
    return dict(zip(("swapped", "ctas", "width", "slices", "any_order"), p.tolist()))


@pytest.mark.parametrize("rows", [1, 9, 16, 17, 32, 36, 64, 100, 128])
@pytest.mark.parametrize("n", [128, 256, 288, 512, 1024, 2048, 4096, 8192, 9472, 9473, 12288, 14336])
def test_sums_that_always_came_in_order_still_do(rows, n):
    for k in (72, 256, 384, 385, 392, 448, 512, 520, 704, 768, 896, 960, 1024, 2048, 4096, 14336):
        if k % 8:
            continue
        p = plan(rows, n, k, RESID)
        assert p["swapped"] == 1
        if k <= 960 or n > 9472:   # fewer than 16 blocks of 64, or row blocks on more than half of 148 SMs
            assert p["any_order"] == 0, (rows, n, k, p)
        assert not p["any_order"] or p["slices"] > 1


@pytest.mark.parametrize("epi", [STORE, GATED])
def test_other_epilogues_sum_in_slice_order(epi):
    for rows in (9, 36, 128, 129, 700, 4096):
        for n in (96, 256, 2048, 28672):
            for k in (72, 512, 2048, 14336):
                assert plan(rows, n, k, epi)["any_order"] == 0


def test_more_than_128_rows_add_to_the_residual_in_slice_order():
    for rows in (129, 300, 2000):
        for k in (448, 2048, 8192):
            p = plan(rows, 1024, k, RESID)
            assert p["swapped"] == 0 and p["any_order"] == 0


# us whole, in the best number of published slices and as these clusters: 74 x 288 x 768 26.8, 24.7, 14.5; 100 x 288 x 768 28.8, 28.8, 14.6;
# 128 x 4096 x 768 31.0, 32.9, 18.3; 12 x 8192 x 1536 25.0, 21.8, 20.8; 128 x 8192 x 1536 50.6, 46.8, 34.6; 9 x 288 x 288 7.3, 7.2, 6.7
@pytest.mark.parametrize("rows,n,k,slices", [(74, 288, 768, 6), (100, 288, 768, 6), (128, 4096, 768, 4), (74, 1024, 768, 6), (12, 8192, 1536, 2), (48, 8192, 1536, 2),
                                             (74, 8192, 1536, 2), (128, 8192, 1536, 2), (74, 8192, 768, 2), (128, 288, 288, 2), (9, 288, 288, 2)])
def test_fp32_products_are_cut_where_that_was_measured_faster(rows, n, k, slices):
    p = plan(rows, n, k, STORE, 1)
    assert p["slices"] == slices and p["ctas"] == slices and p["any_order"] == 0
    assert plan(rows, n, k, RESID, 1)["any_order"] == 0   # fp32 sums always come in slice order


@pytest.mark.parametrize("rows,n,k,epi,fp32,slices,ctas", [
    (9, 6144, 4096, STORE, 0, 3, 1), (16, 6144, 4096, STORE, 0, 3, 1),   # 48 clusters of three are more than fit at once
    (32, 6144, 4096, STORE, 0, 2, 2), (20, 3072, 2048, STORE, 0, 5, 5),
    (28, 7680, 760, STORE, 0, 1, 1), (32, 28672, 4096, GATED, 0, 1, 1),
    (32, 4096, 4096, RESID, 0, 4, 1)])                                   # added in place, in any order
def test_slices_are_a_cluster_where_all_of_them_are_resident(rows, n, k, epi, fp32, slices, ctas):
    p = plan(rows, n, k, epi, fp32)
    assert (p["slices"], p["ctas"]) == (slices, ctas)


def test_refused_arguments():
    p = np.zeros(5, np.int32)
    for bad in ((0, 256, 256, 0, 0), (9, 0, 256, 0, 0), (9, 256, 0, 0, 0), (9, 256, 12, 0, 0), (9, 256, 256, 3, 0), (9, 256, 256, -1, 0), (129, 256, 256, 0, 1)):
        assert _cabi.lib().l3_debug_gemm_plan(*bad, _cabi.i32p(p)) == _cabi.L3_EINVAL


def test_shapes_of_the_gpu_test_reach_every_cut():
    from test_gemm_pairs_gpu import SHAPES
    seen = set()
    for rows, n, k in SHAPES:
        p = plan(rows, n, k)
        assert p["swapped"] == 0
        tiles = -(-rows // (128 * p["ctas"])) * -(-n // p["width"]) * p["slices"]
        rounds = -(-tiles // (148 // p["ctas"]))
        seen |= {("width", p["ctas"], p["width"]), ("rounds", p["ctas"], rounds > 1), ("slices", p["ctas"], p["slices"] > 1, rounds > 1)}
    assert {w for kind, c, w, *_ in seen if kind == "width" and c == 1} == set(range(32, 257, 32))
    assert {w for kind, c, w, *_ in seen if kind == "width" and c == 2} >= set(range(96, 257, 32))
    for c in (1, 2):
        assert {("rounds", c, False), ("rounds", c, True), ("slices", c, True, False), ("slices", c, True, True), ("slices", c, False, True)} <= seen
