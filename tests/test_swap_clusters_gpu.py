"""Products of 9 - 128 rows whose K slices are a cluster (gemm_swap.cu): shapes for which the plan chooses one, rows that do not divide
over the slices, tiles' edges and a ragged K, in both operand kinds; against float64, and bit for bit the same from run to run.
Bounds: bf16 operands are exact, sums of K terms in fp32 accumulators that truncate, K / 16 * 2^-24 of the accumulated size at the worst,
4096 / 16 * 2^-24 = 1.5e-5; three TF32 products leave 2^-22 of each term and truncate likewise."""
import numpy as np
import pytest

from llama3_np_b200 import _cabi

pytestmark = pytest.mark.gpu


def _product(x, w, bf16):
    out = np.empty((len(x), len(w)), np.float32)
    _cabi.check(_cabi.lib().l3_op_linear(0, _cabi.f32p(x), _cabi.f32p(w), len(x), len(w), x.shape[1], 4, int(bf16), _cabi.f32p(out)))
    return out


@pytest.mark.parametrize("bf16", [True, False])
@pytest.mark.parametrize("n,k", [(128, 2048), (389, 4096), (3072, 2056), (6144, 4096), (9336, 2048)])
@pytest.mark.parametrize("rows", [9, 16, 19, 33, 64, 127])
def test_slices_in_a_cluster(rows, n, k, bf16):
    import torch
    rng = np.random.default_rng(rows + n)
    x, w = (torch.from_numpy(rng.standard_normal(s).astype(np.float32)) for s in ((rows, k), (n, k)))
    if bf16:
        x, w = x.bfloat16().float(), w.bfloat16().float()
    x, w = x.numpy(), w.numpy()
    got = _product(x, w, bf16)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    assert np.linalg.norm(got - want) < 1.5e-5 * np.linalg.norm(want)
    assert np.array_equal(got, _product(x, w, bf16))
