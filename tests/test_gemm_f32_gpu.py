"""fp32 projections of many rows on the tensor cores at fp32 precision (gemm_f32.cu).

A Risalix layer whose output matrices are zero leaves the stream as it is, so the logits are one product of the normed embedding
rows and the output projection: K = width, N = vocabulary.  Sizes at the edges of the 128 x 128 tiles, of the 64-wide blocks and
128-wide accumulator turns of K, with and without a K split, odd N (rows that are no multiple of 16 bytes).  Bound: 8 truncations
of at most 2^-23 of an accumulator's value, half of that on average, and the norm's few roundings: 8 * 2^-24 + 2^-23 = 6e-7 of the
result in the 2-norm; a missing correction product would show as 2^-16 or 2^-9."""
import numpy as np
import pytest

import test_risalix_gpu as ris

pytestmark = pytest.mark.gpu


def _stream_only(width, vocab):
    cfg = ris.config([ris.lightning(1, 16, 16, (0.9,))], width=width, vocab=vocab, side=0)
    t = ris.random_model(cfg, width + vocab, bf16_grid=False)
    t["l0.mix.o"] = np.zeros_like(t["l0.mix.o"])
    return cfg, t


@pytest.mark.parametrize("width,vocab", [(64, 64), (72, 97), (128, 128), (136, 130), (320, 300), (1032, 513), (4096, 256)])
def test_products_of_every_tile_edge(width, vocab):
    cfg, t = _stream_only(width, vocab)
    x, w = t["embed"].astype(np.float32).astype(np.float64), t["head"].astype(np.float32).astype(np.float64)
    fin = 1.0 + t["final.norm"].astype(np.float32).astype(np.float64)
    m, _ = ris.build(cfg, tensors=t, max_seq_len=310)
    for rows in (9, 127, 128, 129, 300):
        ids = np.random.default_rng(rows).integers(0, vocab, rows)
        e = x[ids]
        want = (e / np.sqrt((e * e).mean(-1, keepdims=True) + cfg["norm"]["eps"]) * fin) @ w.T
        got = m.forward_rows(ids[None], 0, list(range(rows)))
        assert np.linalg.norm(got - want) < 6e-7 * np.linalg.norm(want), rows
    m.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_gated_units_and_strided_second_projections(dtype):
    """The gate's and the residual-free store epilogues, and the two-matrix projections of the delta rule: slices of a wider row as
    the left operand, with a bf16 matrix in bf16 mode.  A portion of up to 8 tokens runs the row-streaming kernels instead."""
    cfg = ris.config([ris.delta(4, 2, 64, 64, 4, ff=328)], width=512, vocab=150, side=72)
    m, o = ris.build(cfg, 3, dtype, max_seq_len=150)
    ids = np.random.default_rng(1).integers(0, 150, 140)
    want = o.run(ids)
    whole = m.forward_rows(ids[None], 0, list(range(140)))
    parts = np.concatenate([m.forward_rows(ids[None, p:p + 8], p, list(range(len(ids[p:p + 8])))) for p in range(0, 140, 8)])
    m.close()
    assert ris.err(whole, want) < (2e-5 if dtype == "float32" else 6e-2)
    assert ris.err(whole, parts) < (2e-5 if dtype == "float32" else 1e-2)


def _product(x, w, bf16):
    from llama3_np_b200 import _cabi
    out = np.empty((len(x), len(w)), np.float32)
    _cabi.check(_cabi.lib().l3_op_linear(0, _cabi.f32p(x), _cabi.f32p(w), len(x), len(w), x.shape[1], 5, int(bf16), _cabi.f32p(out)))
    return out


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("rows,n,k", [(9, 64, 64), (130, 260, 320), (128, 128, 4096)])
def test_infinities_and_nan(rows, n, k, bf16):
    """Infinities and NaN in the rows and in the matrix give what they give in a plain sum (an infinity of the sign of the products, NaN
    for a sum of both signs or for a zero); results without them are as exact as ever.  With and without a K split."""
    rng = np.random.default_rng(k)
    x, w = rng.standard_normal((rows, k)).astype(np.float32), (rng.integers(-64, 65, (n, k)) / 64).astype(np.float32)  # bf16 numbers, some 0
    x[1, 5], x[2, k - 1], x[3, [0, 7]], x[4, 9], x[rows - 1, 31] = np.inf, -np.inf, [np.inf, -np.inf], np.nan, 3e38
    w[3, 2], w[n - 1, 33], w[7, 1] = np.inf, -np.inf, np.nan
    got = _product(x, w, bf16)
    with np.errstate(all="ignore"):
        want = np.stack([(x[i].astype(np.float64) * w).sum(-1) for i in range(rows)])
    want32 = want.astype(np.float32)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(got[np.isinf(want32)], want32[np.isinf(want32)])
    fine = np.isfinite(want32)
    fine[-1] = False
    assert np.abs(got[fine] - want[fine]).max() < 6e-7 * np.sqrt(k) * 4


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("rows,n,k", [(9, 64, 64), (128, 97, 72), (129, 130, 64), (300, 64, 136), (127, 384, 96), (640, 256, 4096)])
def test_products_alone(rows, n, k, bf16):
    """The kernel by itself at sizes whose products the decoders leave to the FFMA tiles as well (K below 128): same bound."""
    rng = np.random.default_rng(rows + n)
    x, w = rng.standard_normal((rows, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    if bf16:
        w = (np.ascontiguousarray(w).view(np.uint32) & 0xFFFF0000).view(np.float32)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    assert np.linalg.norm(_product(x, w, bf16) - want) < 6e-7 * np.linalg.norm(want)
