"""Gated units whose activation runs in a product's epilogue without routing weights: GELU (Risalix) and the clamped unit (Vupitar), at the
row counts where the product changes its kernel (8 | 9, 128 | 129) and with rows and hidden values that do not fill a tile; against the
oracles, at the families' bars.  In fp32 mode the gate's weights are eight times as large, so that both of GELU's tails and both clamps
are reached."""
import numpy as np
import pytest

import test_risalix_gpu as risalix
import test_vupitar_gpu as vupitar
from llama3_np_b200 import _cabi

pytestmark = pytest.mark.gpu

ROWS = [1, 8, 9, 31, 128, 129, 300]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("ff", [72, 296])
@pytest.mark.parametrize("family", ["gelu", "clamp"])
def test_gated_units_over_rows(family, ff, dtype):
    f = risalix if family == "gelu" else vupitar
    cfg = f.config([f.attn(ff=ff)]) if family == "gelu" else f.config([f.layer(mlp={"kind": "dense", "ff": ff, "limit": 0.6})])
    t = f.random_model(cfg, 3)
    if dtype == "float32":
        for k in t:
            if k.endswith("mlp.gate"):
                t[k] = t[k] * 8
    m, o = f.build(cfg, dtype=dtype, max_seq_len=max(ROWS), tensors=t)
    ids = f.toks(max(ROWS), cfg["vocab"])
    want = o.run(ids)
    for n in ROWS:
        got = m.forward_rows(ids[None, :n], 0, list(range(n)))
        assert f.err(got, want[:n]) < (f.FP32_BAR if dtype == "float32" else f.BF16_BAR), n
    m.close()


def _gelu(z):
    z, one, out = np.ascontiguousarray(z, np.float32), np.ones(len(z), np.float32), np.empty(len(z), np.float32)
    _cabi.check(_cabi.lib().l3_op_geglu(0, _cabi.f32p(z), _cabi.f32p(one), len(z), _cabi.f32p(out)))
    return out


@pytest.mark.parametrize("sigma", [0.3, 1.0, 4.0])
def test_gelu_is_as_exact_as_with_tanh(sigma):
    """The 2-norm of the error of gates as they come is no larger than that of the form with tanhf (measured: 4.5e-8, 3.8e-8, 2.2e-8), and no
    negative value loses its bits to the difference of nearly equal numbers.  The argument 2 |y| has two rounded constants, a square, a fused
    sum and a product, four roundings of 2^-24 of it at the worst; the exponential's own error is two units of 2^-23, sum, quotient and last
    step have 2^-24 each: 2^-22 |2 y| + 2^-22 + 3 x 2^-24, below 2^-21 + 2^-22 |2 y|."""
    z = np.random.default_rng(0).normal(0, sigma, 1 << 20).astype(np.float32).astype(np.float64)
    y = np.sqrt(2 / np.pi) * (z + 0.044715 * z ** 3)
    want = z / (1 + np.exp(-2 * y))
    got = _gelu(z).astype(np.float64)
    assert np.linalg.norm(got - want) < {0.3: 4.5e-8, 1.0: 3.8e-8, 4.0: 2.2e-8}[sigma] * np.linalg.norm(want)
    seen = np.abs(want) > 1e-30
    assert (np.abs(got - want)[seen] <= (2.0 ** -21 + 2.0 ** -22 * np.abs(2 * y[seen])) * np.abs(want[seen])).all()


def test_gelu_at_the_ends():
    got = _gelu([np.inf, 3e38, 1e30, 1e13, 20.0, -0.0, 0.0, -20.0, -1e13, -3e38, np.nan])
    assert np.array_equal(got[:5], np.float32([np.inf, 3e38, 1e30, 1e13, 20.0])) and np.array_equal(got[5:10], np.zeros(5, np.float32)) and np.isnan(got[10])
