"""bf16 tensor-core projections whose tiles are cut along K (gemm_tc.cu): widths of 32 to 256 columns with remainders, two to eight
slices, more tiles than the machine holds at once.  Bound: the operands are bf16 numbers, products are exact, and the accumulator
loses at most 2^-23 of its value per instruction of 16 terms, half of that on average: K / 16 * 2^-24 of the result, 3.1e-5 at
K = 8192 - a slice that is missing, doubled or misplaced changes it by a share of order 1 / 8."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bf16(a):
    u = np.ascontiguousarray(a, np.float32).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32)


@pytest.mark.parametrize("rows,n,k", [(129, 256, 4096), (300, 250, 8192), (768, 2048, 6144), (200, 4096, 4096), (2048, 256, 2048),
                                      (1462, 2048, 1024), (140, 72, 2056), (640, 3000, 512), (257, 1000, 8192)])
def test_k_splits_add_up(rows, n, k):
    from llama3_np_b200 import _cabi
    rng = np.random.default_rng(rows + n + k)
    x, w = _bf16(rng.standard_normal((rows, k))), _bf16(rng.standard_normal((n, k)) / np.sqrt(k))
    out = np.empty((rows, n), np.float32)
    _cabi.check(_cabi.lib().l3_op_linear(0, _cabi.f32p(x), _cabi.f32p(w), rows, n, k, 3, 1, _cabi.f32p(out)))
    want = x.astype(np.float64) @ w.astype(np.float64).T
    assert np.linalg.norm(out - want) < k / 16 * 2.0 ** -24 * np.linalg.norm(want)
    again = np.empty_like(out)
    _cabi.check(_cabi.lib().l3_op_linear(0, _cabi.f32p(x), _cabi.f32p(w), rows, n, k, 3, 1, _cabi.f32p(again)))
    assert np.array_equal(out, again)   # slices are added in their order, whoever arrives last


@pytest.mark.parametrize("rows,n,k", [(129, 7001, 3000), (385, 4096, 2056), (384, 14000, 600), (513, 8190, 520), (700, 1024, 4096), (1000, 3000, 1000),
                                      (1462, 2048, 2048), (2050, 1999, 2056), (130, 160, 520), (1000, 992, 72)])
def test_widths_and_pairs(rows, n, k):
    """Widths in steps of 32, one CTA or two on a tile (all of them: test_gemm_pairs_gpu.py): a last pair whose second CTA has no row or one, columns and k-blocks
    that end inside a tile, odd widths of the result (element stores)."""
    from llama3_np_b200 import _cabi
    rng = np.random.default_rng(rows + n + k)
    x, w = _bf16(rng.standard_normal((rows, k))), _bf16(rng.standard_normal((n, k)) / np.sqrt(k))
    out = np.empty((rows, n), np.float32)
    _cabi.check(_cabi.lib().l3_op_linear(0, _cabi.f32p(x), _cabi.f32p(w), rows, n, k, 3, 1, _cabi.f32p(out)))
    want = x.astype(np.float64) @ w.astype(np.float64).T
    # every entry: the bound above, its terms' size (1 / sqrt(k) each, of x in N(0, 1)) and the largest of rows * n entries at 6 sigma
    assert np.abs(out - want).max() < 6 * k / 16 * 2.0 ** -24
    assert np.linalg.norm(out - want) < k / 16 * 2.0 ** -24 * np.linalg.norm(want) + 1e-6 * np.linalg.norm(want)
