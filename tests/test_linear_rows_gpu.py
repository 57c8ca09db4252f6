"""Row-streaming products of 3 - 8 rows with bf16 weights (linear.cu) on both sides of the lines between the two orders of the staged
activations, with remainders of the 256-value blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [2, 3, 4, 5, 8])
@pytest.mark.parametrize("n,k", [(2046, 768), (2047, 768), (2048, 768), (2048, 760), (2049, 1032), (1024, 4096), (4099, 2056), (16384, 264)])
def test_both_orders(rows, n, k):
    """fp32 sums of exact products in 32 lanes and 5 steps of a tree: at most (k / 32 + 6) 2^-24 of the sum of the terms' sizes."""
    from llama3_np_b200 import _cabi
    rng = np.random.default_rng(rows + n + k)
    x = rng.standard_normal((rows, k)).astype(np.float32)
    w = ((rng.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32).view(np.uint32) & 0xFFFF0000).view(np.float32)
    out = np.empty((rows, n), np.float32)
    _cabi.check(_cabi.lib().l3_op_linear(0, _cabi.f32p(x), _cabi.f32p(w), rows, n, k, 1, 1, _cabi.f32p(out)))
    want = x.astype(np.float64) @ w.astype(np.float64).T
    size = np.abs(x).astype(np.float64) @ np.abs(w).astype(np.float64).T
    assert (np.abs(out - want) <= (k / 32 + 6) * 2.0 ** -24 * size).all()
