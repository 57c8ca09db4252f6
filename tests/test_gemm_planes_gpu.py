"""fp32 products whose operands were cut into bf16 parts beforehand (gemm_f32.cu, OP_PLANES): sizes at the edges of the 128 x 128 tiles, of
the blocks of 64 and the accumulators' turns of 128 values of K, with and without a K split - bit for bit what the kernel that cuts its
operands itself gives, since parts, products and the order of the sums are the same."""
import numpy as np
import pytest

from llama3_np_b200 import _cabi

pytestmark = pytest.mark.gpu


def _product(x, w, path):
    out = np.empty((len(x), len(w)), np.float32)
    _cabi.check(_cabi.lib().l3_op_linear(0, _cabi.f32p(x), _cabi.f32p(w), len(x), len(w), x.shape[1], path, 0, _cabi.f32p(out)))
    return out


@pytest.mark.parametrize("rows,n,k", [(9, 64, 64), (127, 128, 72), (128, 129, 128), (129, 97, 136), (300, 257, 192), (600, 1024, 4096), (1500, 2304, 200)])
def test_same_bits_as_cut_in_the_kernel(rows, n, k):
    rng = np.random.default_rng(rows + k)
    x, w = rng.standard_normal((rows, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    x[0, :8] = [0.0, -0.0, 2.0 ** -100, -3e-38, 1.5e38, 1.0 + 2.0 ** -23, 2.0 ** -60, 65504.0]
    got = _product(x, w, 6)
    assert np.array_equal(got, _product(x, w, 5))
    assert np.linalg.norm(got[1:] - x[1:].astype(np.float64) @ w.astype(np.float64).T) < 6e-7 * np.linalg.norm(got[1:])


def test_infinities_and_nan():
    rng = np.random.default_rng(0)
    x, w = rng.standard_normal((140, 256)).astype(np.float32), rng.standard_normal((200, 256)).astype(np.float32)
    x[3, 17], x[130, 255], w[199, 0] = np.inf, np.nan, -np.inf
    got = _product(x, w, 6)
    assert np.array_equal(got, _product(x, w, 5), equal_nan=True)
    assert np.isnan(got[130]).all() and np.isinf(got[3, :199]).all()
